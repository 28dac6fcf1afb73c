// Launch shapes of the persistent Euler loop (euler_loop.cu): one cell per
// thread, two blocks per SM, in one of three forms.  Plain C++.
#pragma once

#include <cstdint>

namespace gb {

// WIDE: up to kLoopWide threads per block a thread may use 128 registers; it
// gathers all its neighbours at once and keeps its face states, ghosts and two
// derived values per face in shared memory.
// NARROW: up to kLoopFull threads, 72 to 96 registers: one face at a time, all of
// a cell's geometry in shared memory.
// LEAN: up to kLoopMax threads, 64 registers: as NARROW, the face normals and
// areas read from L2.
enum class LoopForm { kNone, kWide, kNarrow, kLean };

constexpr int kLoopWide = 256;
constexpr int kLoopFull = 416;
constexpr int kLoopMax = 512;
// Dynamic shared memory of a block, at most: two blocks, with up to 3 KB of
// static and 1 KB of reserved shared memory each, share an SM's 228 KB.
constexpr int kLoopSmem = 110 * 1024;

// shared memory of a block (bytes)
constexpr int loop_smem(LoopForm form, int max_faces, int threads) {
    return threads * (form == LoopForm::kWide     ? 72 * max_faces + 92
                      : form == LoopForm::kNarrow ? 44 * max_faces + 28
                                                  : 28 * max_faces + 28);
}

// The first form that fits.  Where WIDE's memory does not (5 faces at 256
// threads, 6 at 224 and 256) NARROW's does, which is why it must not be passed
// over for LEAN.
constexpr LoopForm loop_form(int max_faces, int threads) {
    return threads <= kLoopWide && loop_smem(LoopForm::kWide, max_faces, threads) <= kLoopSmem     ? LoopForm::kWide
           : threads <= kLoopFull && loop_smem(LoopForm::kNarrow, max_faces, threads) <= kLoopSmem ? LoopForm::kNarrow
           : threads <= kLoopMax && loop_smem(LoopForm::kLean, max_faces, threads) <= kLoopSmem    ? LoopForm::kLean
                                                                                                   : LoopForm::kNone;
}

// Where the loop beats the kernels it replaces depends on how well the lanes of
// a warp share the 32-byte sectors of their neighbours' records: `sectors`,
// counted over a warp's face slots (neighbour_sectors).  One-layer meshes have
// 50 to 67, prisms stacked in layers 75 to 92, 3-D hexes 97 to 99, prisms under
// tets, tets, pyramids and mixes of elements 102 to 120.  The narrow forms wait
// for these loads one face after another; WIDE has them all in flight.
constexpr float kLoopLayer = 72.f, kLoopStacked = 94.f, kLoopScattered = 105.f;
constexpr int64_t kLoopNever = int64_t(1) << 62;

// Iterations from which a launch of the Euler loop (of a run of n_iter) is taken
// over the kernels.  Loop / kernels, us per iteration in developed flow (B200,
// 148 SMs), 64,000 to 146,000 cells unless stated:
//   WIDE    12,000 to 66,000: layers 11..20 / 19..23, stacked 13..18 / 19..22,
//           tets 10..14 / 19..21, pyramids 13..18 / 19..21, hexes 18..22 / 23, mixes
//           18 / 21 at 12,000, 22.6 / 23.0 at 46,000, 24.2 / 23.1 at 54,000.  A launch
//           of 4 breaks even for tets, up to 19,000 cells with 5 faces and up to
//           57,000 (us per call of 5: 132 / 154 at 50,000) in one layer of prisms,
//           of 6 on larger layers and stacked prisms, of 8 on the largest of these,
//           one-layer hexes and small hexes and mixes, of 16 on other hexes.  In a
//           batch, whose kernels take a launch more, a little earlier (of 6, 12,000
//           hexes: 169 / 184).
//   NARROW  layers 14..32 / 22..33, stacked 19..27 / 21..27 (a launch of 8 breaks even
//           on a layer of prisms, of 16 of hexes and below 94,000 stacked cells, of
//           32 above), tets 90,000 21.3 / 23.1 (in a batch 24.2 / 23.0), 105,000
//           26.0 / 24.0, hexes 25..37 / 23..31, pyramids 24..34 / 21..27, mixes 29..41 /
//           23..27.  3-D hexes from a uniform start, its limiter still idle, take
//           22..27 / 25..29 for their first hundred iterations.
//   LEAN    layers 22..37 / 29..46 from launches of 32 on, stacked 27..34 / 27..32, tets
//           30..35 / 25..27, mixes 42..48 / 27..31.
constexpr int64_t loop_shortest(LoopForm form, int max_faces, int threads, float sectors, bool batch, int64_t n_iter) {
    if (form == LoopForm::kWide) {
        const bool small = threads <= 64, medium = threads <= 192;
        if (max_faces <= 4 || (max_faces == 5 && small)) return 4;
        if (max_faces == 5) {
            if (sectors <= kLoopLayer) return medium ? 4 : 6;
            if (sectors <= kLoopStacked) return medium ? 6 : 8;
            return medium ? 8 : 16;
        }
        if (sectors <= kLoopLayer) return 8;
        if (batch) return sectors <= kLoopScattered ? (small ? 4 : 8) : (small ? 6 : 16);
        if (small) return 8;
        return sectors <= kLoopScattered ? 16 : threads <= 160 ? 32 : kLoopNever;
    }
    if (form == LoopForm::kNarrow) {
        if (sectors <= kLoopLayer) return max_faces <= 5 ? 8 : 16;
        if (sectors <= kLoopStacked) return threads <= 320 ? 16 : 32;
        if (batch) return kLoopNever;
        if (max_faces <= 4) return threads <= 352 ? 8 : kLoopNever;
        return max_faces == 6 && sectors <= kLoopScattered && n_iter <= 96 ? 32 : kLoopNever;
    }
    return form == LoopForm::kLean && !batch && sectors <= kLoopLayer ? 32 : kLoopNever;
}

// The same for the incompressible loop (nsi_loop.cu).  Loop / kernels:
//   up to 256 threads (75,000 cells): 7..13 / 17..32 without, 12..21 / 23..39 with the
//           limiter.
//   up to 448: without the limiter 12..31 / 23..38; with it layers 19..33 / 28..36,
//           stacked 31..37 / 39..43 (27..36 / 28..33 where the kernels apply the
//           conditions inside the gradient pass and are faster for it), tets 36..42 /
//           37..43, hexes 39..50 / 30..44, pyramids 41..46 / 41..45, mixes 46..52 / 42..46.
//   above: layers 24 / 29 without, 29 / 33 with the limiter, stacked 29..34 / 27..37 and
//           46..48 / 34..44, tets 36..37 / 36..37 and 50..53 / 42..44.
// Runs of up to 64 iterations take the last shape of tets with the limiter too:
// it is compared with the kernels there.
constexpr int64_t nsi_loop_shortest(int max_faces, int threads, float sectors, bool limited, bool inline_bcs,
                                    int64_t n_iter) {
    if (threads <= 256) return 4;
    if (threads <= 448) {
        if (!limited) return 8;
        if (sectors <= kLoopLayer) return max_faces <= 5 ? 8 : 24;
        return !inline_bcs && (max_faces <= 4 || sectors <= kLoopStacked) ? 8 : kLoopNever;
    }
    if (sectors <= kLoopLayer) return limited ? 32 : 16;
    return max_faces <= 4 && (!limited || n_iter <= 64) ? 16 : kLoopNever;
}

}  // namespace gb
