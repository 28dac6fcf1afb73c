// The Euler loop of a mesh that fits on the GPU one cell per thread, as one
// persistent launch for many iterations.
//
// A cell's geometry stays in its thread's shared-memory column and its state
// in registers; what its neighbours need -- the state for their gradients,
// the reconstructed face states for their fluxes -- is handed over through L2
// in 16-byte records that carry the iteration they belong to, so a reader
// polls the data itself: no barrier, no fence and no flag is on the way from
// one cell to the next, and every warp runs as far ahead as its own
// neighbours allow.  Records are single 128-bit accesses (atomic as a whole).
// A buffer is free when it is written again: a cell writes its new state only
// after reading its neighbours' face states, which they form after reading
// its old one, and its new face states only after reading its neighbours' new
// states, which they form after reading its old face states.
//
// The residual is summed by one more block, in the order of k_flux and
// k_reduce_final, from per-warp sums handed over the same way; its verdict
// (go on, converged, not finite) is waited for by the update of the next
// iteration, behind that iteration's gradient pass.
//
// What bounds it is latency: a cell's chain in an iteration is two hand-overs
// through L2 of about 1 us each and the dependent arithmetic of a gradient and
// a flux, and one cell per thread leaves few warps to hide it.  Counters (B200):
// 28,800 tets, 6 warps per SM, issue slots 21 % busy, L2 at 10 % of its
// throughput, 3.2 warps waiting for memory per instruction issued; 120,000
// prisms, 25 warps, 47 %, 36 %, 8.3.  So the wide form gathers all of a cell's
// neighbours at once and keeps what it can on chip; the narrow ones have one
// face in flight in few registers and live off their warps.  Per iteration in
// launches of 100 against the replayed graph of three or four kernels: 12,060
// prisms in one layer 11.3 / 19.1 us, 28,350 tets 10.5 / 19.1, 45,240 prisms 13.0 /
// 21.1, 74,148 prisms 13.2 / 23.1, 120,416 prisms 18.8 / 27.2, 148,208 prisms
// (normals read from L2) 21.8 / 33.4; where it loses and is not taken:
// loop_shape.h.  With a state's two records side by side instead of in planes
// 120,000 prisms took 19.5 where they took 16.8.
// Flags per block instead of tagged data took 12 to 21 us for these: a fence
// on each side and a block barrier per hand-over, and the slowest warp of
// every block in everyone's way.
#include "euler_loop.cuh"

#include <algorithm>
#include <type_traits>

namespace gb {
namespace {

// A state is two records, `plane` apart: the lanes of a warp read and write
// whole sectors of each plane (side by side, every 16-byte access would move a
// 32-byte sector and use half of it).
__device__ __forceinline__ void st_state(TagRec* p, size_t plane, float r, float3 u, float e, unsigned int tag) {
    st_rec(p, __float_as_uint(r), __float_as_uint(u.x), __float_as_uint(u.y), tag);
    st_rec(p + plane, __float_as_uint(u.z), __float_as_uint(e), tag, tag);
}
// whether both records of a state carry `tag`; their values if so
__device__ __forceinline__ bool ld_state(const TagRec* p, size_t plane, unsigned int tag, float& r, float4& ue) {
    const TagRec a = ld_rec(p), b = ld_rec(p + plane);
    r = __uint_as_float(a.x);
    ue = make_float4(__uint_as_float(a.y), __uint_as_float(a.z), __uint_as_float(b.x), __uint_as_float(b.y));
    return fresh<3>(a, tag) && fresh<2>(b, tag);
}

// One cell's face entries in shared memory, [slot][component][cell of the
// block]: the neighbour word, the offsets of the neighbour and of the face
// centre, the outward normal and area / volume; then the cell's least-squares
// inverse and volume; and with WIDE, for its first kGhostSlots ghosts the
// offset of the face centre from the ghost and the ghost's state (after the
// gradient pass its face state), its own face states, and 1 / |dn|^2 and
// |df|^3 (formed anew in every iteration otherwise, by the same operations).
constexpr int kGhostSlots = 2;
template <int MAXF, bool LEAN>
struct TileGeo {
    static constexpr int kLsq = (LEAN ? 7 : 11) * MAXF;   // first word after the entries
    float* base;      // this thread's column
    int T;
    const float4* cf_geo;   // LEAN: this cell's first entry in the mesh's array, N entries to the next slot
    uint32_t N;
    __device__ __forceinline__ uint32_t& nb(int t) const { return reinterpret_cast<uint32_t*>(base)[t * T]; }
    __device__ __forceinline__ float& dn(int t, int k) const { return base[(MAXF + 3 * t + k) * T]; }
    __device__ __forceinline__ float& df(int t, int k) const { return base[(4 * MAXF + 3 * t + k) * T]; }
    __device__ __forceinline__ float& cf(int t, int k) const { return base[(7 * MAXF + 4 * t + k) * T]; }
    __device__ __forceinline__ float& lsq(int k) const { return base[(kLsq + k) * T]; }
    __device__ __forceinline__ float& vol() const { return base[(kLsq + 6) * T]; }
    __device__ __forceinline__ float& ghost(int g, int k) const { return base[(kLsq + 7 + 8 * g + k) * T]; }
    __device__ __forceinline__ float& own(int t, int k) const {
        return base[(kLsq + 7 + 8 * kGhostSlots + 5 * t + k) * T];
    }
    __device__ __forceinline__ float& w2(int t) const { return base[(kLsq + 7 + 8 * kGhostSlots + 5 * MAXF + t) * T]; }
    __device__ __forceinline__ float& k3(int t) const { return base[(kLsq + 7 + 8 * kGhostSlots + 6 * MAXF + t) * T]; }
    __device__ __forceinline__ float3 dn3(int t) const { return make_float3(dn(t, 0), dn(t, 1), dn(t, 2)); }
    __device__ __forceinline__ float3 df3(int t) const { return make_float3(df(t, 0), df(t, 1), df(t, 2)); }
    __device__ __forceinline__ float4 cf4(int t) const {
        if (LEAN) return __ldg(cf_geo + (size_t)t * N);
        return make_float4(cf(t, 0), cf(t, 1), cf(t, 2), cf(t, 3));
    }
    __device__ __forceinline__ float3 cf3(int t) const { return f3(cf4(t)); }
};

// In the top four bits of the neighbour word (kNbMask): the slot of the same
// face among the neighbour's entries, or a ghost's region.

template <int MAXF, bool WIDE, bool LEAN>
__device__ __forceinline__ void load_geo(const EulerLoopArgs& a, uint32_t i, int nf, const TileGeo<MAXF, LEAN>& g) {
    const MeshDev& m = a.m;
    const float4 l0 = __ldg(&m.lsq[2 * i]), l1 = __ldg(&m.lsq[2 * i + 1]);
    g.lsq(0) = l0.x; g.lsq(1) = l0.y; g.lsq(2) = l0.z; g.lsq(3) = l0.w; g.lsq(4) = l1.x; g.lsq(5) = l1.y;
    g.vol() = __ldg(&m.cell_geo[i]).w;
    int ng = 0;
#pragma unroll 1
    for (int t = 0; t < nf; ++t) {
        const uint32_t k = i + t * m.N, j = __ldg(&m.nbc[k]);
        uint32_t top = 0;
        if (j < m.N) {
            top = __ldg(&m.twin[k]) / m.N;
        } else {
            while ((int)top < a.ghosts.n - 1 && j >= a.ghosts.start[top + 1]) ++top;
            if (WIDE && ng < kGhostSlots) {
                const float4 o = __ldg(&a.ghost_off[j - m.N]);
                g.ghost(ng, 0) = o.x; g.ghost(ng, 1) = o.y; g.ghost(ng, 2) = o.z;
                ++ng;
            }
        }
        g.nb(t) = j | (top << 28);
        const float4 n = __ldg(&m.dn[k]), b = __ldg(&m.df[k]);
        if (WIDE) { g.w2(t) = n.w; g.k3(t) = b.w; }
        g.dn(t, 0) = n.x; g.dn(t, 1) = n.y; g.dn(t, 2) = n.z;
        g.df(t, 0) = b.x; g.df(t, 1) = b.y; g.df(t, 2) = b.z;
        if (!LEAN) {
            const float4 c = __ldg(&m.cf_geo[k]);
            g.cf(t, 0) = c.x; g.cf(t, 1) = c.y; g.cf(t, 2) = c.z; g.cf(t, 3) = c.w;
        }
    }
}

struct CellState {
    float r, e;
    float3 u;
};

// grad_lim_cell with the cell's own state in registers, its entries in shared
// memory and GATHER neighbours polled for at once.  False: a wait gave up.
template <bool TRANSPOSED, int MAXF, bool WIDE, bool LEAN>
__device__ __forceinline__ bool grad_loop_cell(const EulerLoopArgs& a, int buf, unsigned int tag,
                                               const TileGeo<MAXF, LEAN>& g, uint32_t i, int nf, const CellState& own) {
    const MeshDev& m = a.m;
    const TagRec* nbs = a.state[buf];
    const float v[5] = {own.r, own.u.x, own.u.y, own.u.z, own.e};
    float3 gs[5];
    float vmin[5], vmax[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) { gs[c] = make_float3(0.f, 0.f, 0.f); vmin[c] = v[c]; vmax[c] = v[c]; }
    int ng = 0;
    Patience wait(a);
    auto add = [&](int t, float r, float4 ue) {
        const float3 d = g.dn3(t);
        const float w = WIDE ? g.w2(t) : 1.f / ydot(d, d);
        const float vj[5] = {r, ue.x, ue.y, ue.z, ue.w};
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            gs[c] = gs[c] + (d * (vj[c] - v[c])) * w;
            vmin[c] = fminf(vmin[c], vj[c]);
            vmax[c] = fmaxf(vmax[c], vj[c]);
        }
    };
    if constexpr (WIDE) {
        // few warps: all neighbours in flight at once
        float nr[MAXF];
        float4 nu[MAXF];
        unsigned int pending = 0;
#pragma unroll
        for (int t = 0; t < MAXF; ++t) {
            if (t >= nf) continue;
            const uint32_t j = g.nb(t) & kNbMask;
            if (j < m.N) {
                pending |= 1u << t;
            } else if (ng < kGhostSlots) {
                nr[t] = g.ghost(ng, 3);
                nu[t] = make_float4(g.ghost(ng, 4), g.ghost(ng, 5), g.ghost(ng, 6), g.ghost(ng, 7));
                ++ng;
            } else {
                const float4 u = __ldcg(&a.rhou[buf][j]);
                nr[t] = __ldcg(&a.rho[buf][j]);
                nu[t] = make_float4(u.x, u.y, u.z, __ldcg(&a.rhoe[buf][j]));
            }
        }
        for (;;) {
            unsigned int left = 0;
#pragma unroll
            for (int t = 0; t < MAXF; ++t)
                if (pending & (1u << t))
                    if (!ld_state(&nbs[g.nb(t) & kNbMask], m.N, tag, nr[t], nu[t])) left |= 1u << t;
            pending = left;
            if (pending == 0) break;
            if (!wait.more()) return false;
        }
#pragma unroll
        for (int t = 0; t < MAXF; ++t)
            if (t < nf) add(t, nr[t], nu[t]);
    } else {
        // many warps: one neighbour at a time, in few registers
#pragma unroll 1
        for (int t = 0; t < nf; ++t) {
            const uint32_t j = g.nb(t) & kNbMask;
            float r;
            float4 ue;
            if (j < m.N) {
                while (!ld_state(&nbs[j], m.N, tag, r, ue))
                    if (!wait.more()) return false;
            } else {
                ue = __ldcg(&a.rhou[buf][j]);
                r = __ldcg(&a.rho[buf][j]);
                ue.w = __ldcg(&a.rhoe[buf][j]);
            }
            add(t, r, ue);
        }
    }
    const float4 l0 = make_float4(g.lsq(0), g.lsq(1), g.lsq(2), g.lsq(3)), l1 = make_float4(g.lsq(4), g.lsq(5), 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < 5; ++c) gs[c] = sym_mul(l0, l1, gs[c]);
    float lim[5] = {2.f, 2.f, 2.f, 2.f, 2.f};
    float du[5], dd[5], dmm2[5];
    limiter_range(v, vmin, vmax, du, dd, dmm2);
#pragma unroll 1
    for (int t = 0; t < nf; ++t) {
        const float3 d = g.df3(t);
        float k3;
        if (WIDE) {
            k3 = g.k3(t);
        } else {
            const float dl = sqrtf(ydot(d, d));
            k3 = __fmul_rn(__fmul_rn(dl, dl), dl);
        }
        limit_face(lim, du, dd, dmm2, gs, d, k3);
    }
    const float4 u0 = make_float4(own.u.x, own.u.y, own.u.z, 0.f);
    const float4 gr = make_float4(gs[0].x, gs[0].y, gs[0].z, lim[0]);
    const float4 gu[3] = {make_float4(gs[1].x, gs[1].y, gs[1].z, lim[1]),
                          make_float4(gs[2].x, gs[2].y, gs[2].z, lim[2]),
                          make_float4(gs[3].x, gs[3].y, gs[3].z, lim[3])};
    const float4 ge = make_float4(gs[4].x, gs[4].y, gs[4].z, lim[4]);
    ng = 0;
#pragma unroll 1
    for (int t = 0; t < nf; ++t) {
        float rr, re;
        float3 ru;
        reconstruct<TRANSPOSED>(v[0], u0, v[4], gr, gu, ge, g.df3(t), rr, ru, re);
        const uint32_t j = g.nb(t) & kNbMask;
        if (j < m.N || !WIDE) st_state(&a.rec[i + t * m.N], m.S, rr, ru, re, tag);
        if (WIDE) {
            g.own(t, 0) = rr; g.own(t, 1) = ru.x; g.own(t, 2) = ru.y; g.own(t, 3) = ru.z; g.own(t, 4) = re;
        }
        if (j < m.N) continue;
        // the ghost's face state is read by this thread alone
        if (WIDE && ng < kGhostSlots) {
            const float4 uj = make_float4(g.ghost(ng, 4), g.ghost(ng, 5), g.ghost(ng, 6), 0.f);
            reconstruct<TRANSPOSED>(g.ghost(ng, 3), uj, g.ghost(ng, 7), gr, gu, ge,
                                    make_float3(g.ghost(ng, 0), g.ghost(ng, 1), g.ghost(ng, 2)), rr, ru, re);
            g.ghost(ng, 3) = rr; g.ghost(ng, 4) = ru.x; g.ghost(ng, 5) = ru.y; g.ghost(ng, 6) = ru.z; g.ghost(ng, 7) = re;
            ++ng;
        } else {
            reconstruct<TRANSPOSED>(__ldcg(&a.rho[buf][j]), __ldcg(&a.rhou[buf][j]), __ldcg(&a.rhoe[buf][j]), gr, gu,
                                    ge, f3(__ldg(&a.ghost_off[j - m.N])), rr, ru, re);
            a.rec_rho[m.S + (j - m.N)] = rr;
            a.rec_rhou[m.S + (j - m.N)] = make_float4(ru.x, ru.y, ru.z, re);
        }
    }
    return true;
}

// The states of the cell's ghosts for its state `own`, for the next gradient
// pass: in its ghost slots, or in the buffer `buf` that the pass reads.  Nobody
// else reads them, so they are formed before the neighbours are waited for.
template <int MAXF, bool WIDE, bool LEAN>
__device__ __forceinline__ void ghost_states(const EulerLoopArgs& a, const GhostBcTable& bc, const TileGeo<MAXF, LEAN>& g,
                                             int nf, int buf, const CellState& own) {
    int ng = 0;
#pragma unroll 1
    for (int t = 0; t < nf; ++t) {
        const uint32_t word = g.nb(t), j = word & kNbMask;
        if (j < a.m.N) continue;
        const int k = WIDE ? ng++ : kGhostSlots;
        float r, e;
        float4 u;
        if (!region_state(bc, word >> 28, g.cf3(t), own.r, own.u, own.e, r, u, e)) {
            if (k >= kGhostSlots) continue;
            r = __ldcg(&a.rho[buf][j]);
            u = __ldcg(&a.rhou[buf][j]);
            e = __ldcg(&a.rhoe[buf][j]);
        }
        if (k < kGhostSlots) {
            g.ghost(k, 3) = r; g.ghost(k, 4) = u.x; g.ghost(k, 5) = u.y; g.ghost(k, 6) = u.z; g.ghost(k, 7) = e;
        } else {
            a.rho[buf][j] = r;
            a.rhou[buf][j] = u;
            a.rhoe[buf][j] = e;
        }
    }
}

// flux_cell's sum over the faces.  False: a wait gave up.
template <int MAXF, bool WIDE, bool FULL, bool LEAN>
__device__ __forceinline__ bool flux_loop_cell(const EulerLoopArgs& a, unsigned int tag, const TileGeo<MAXF, LEAN>& g,
                                               uint32_t i, int nf, FluxSum& s) {
    const MeshDev& m = a.m;
    Patience wait(a);
    auto twin = [&](uint32_t word) { return &a.rec[(word >> 28) * m.N + (word & kNbMask)]; };
    if constexpr (WIDE) {
        float rb[MAXF];
        float4 ub[MAXF];
        unsigned int pending = 0;
        int ng = 0;
#pragma unroll
        for (int t = 0; t < MAXF; ++t) {
            if (!FULL && t >= nf) continue;
            const uint32_t j = g.nb(t) & kNbMask;
            if (j < m.N) {
                pending |= 1u << t;
            } else if (ng < kGhostSlots) {
                rb[t] = g.ghost(ng, 3);
                ub[t] = make_float4(g.ghost(ng, 4), g.ghost(ng, 5), g.ghost(ng, 6), g.ghost(ng, 7));
                ++ng;
            } else {
                rb[t] = __ldcg(&a.rec_rho[m.S + (j - m.N)]);
                ub[t] = __ldcg(&a.rec_rhou[m.S + (j - m.N)]);
            }
        }
        float ra[MAXF];
        float4 ua[MAXF];
#pragma unroll
        for (int t = 0; t < MAXF; ++t) { ra[t] = g.own(t, 0); ua[t] = make_float4(g.own(t, 1), g.own(t, 2), g.own(t, 3), g.own(t, 4)); }
        for (;;) {
            unsigned int left = 0;
#pragma unroll
            for (int t = 0; t < MAXF; ++t)
                if (pending & (1u << t))
                    if (!ld_state(twin(g.nb(t)), m.S, tag, rb[t], ub[t])) left |= 1u << t;
            pending = left;
            if (pending == 0) break;
            if (!wait.more()) return false;
        }
#pragma unroll
        for (int t = 0; t < MAXF; ++t) {
            if (!FULL && t >= nf) continue;
            s.face(g.cf3(t), g.cf(t, 3), ra[t], rb[t], ua[t], ub[t]);
        }
    } else {
#pragma unroll 1
        for (int t = 0; t < nf; ++t) {
            const uint32_t word = g.nb(t), j = word & kNbMask;
            float ra, rb;
            float4 ua, ub;
            ld_state(&a.rec[i + t * m.N], m.S, tag, ra, ua);   // this thread's own stores
            if (j < m.N) {
                while (!ld_state(twin(word), m.S, tag, rb, ub))
                    if (!wait.more()) return false;
            } else {
                rb = __ldcg(&a.rec_rho[m.S + (j - m.N)]);
                ub = __ldcg(&a.rec_rhou[m.S + (j - m.N)]);
            }
            const float4 c = g.cf4(t);
            s.face(f3(c), c.w, ra, rb, ua, ub);
        }
    }
    return true;
}

// Thread t of warp w of worker block b owns cell 32 (w n_blocks + b) + t: the
// warps of a block are spread over the mesh, so that the regions where the
// limiter works are shared by all SMs.
// LEAN: the face normals and areas stay in global memory.
template <bool TRANSPOSED, int MAXF, bool WIDE, bool LEAN>
__device__ __forceinline__ void euler_loop_worker(const EulerLoopArgs& a, const GhostBcTable& s_bc, uint32_t block,
                                                  float* s_geo) {
    const MeshDev& m = a.m;
    const uint32_t chunk = (threadIdx.x >> 5) * (uint32_t)a.n_blocks + block;
    const uint32_t i = 32u * chunk + (threadIdx.x & 31);
    if (32u * chunk >= m.N) return;
    const bool have = i < m.N;
    const TileGeo<MAXF, LEAN> geo{s_geo + threadIdx.x, (int)blockDim.x, m.cf_geo + i, m.N};
    const int nf = have ? __ldg(&m.nfc[i]) : 0;
    // a warp whose cells all have the most faces runs the flux's face loop without bounds
    const bool full = __all_sync(0xffffffffu, nf == MAXF);
    CellState own{};
    if (have) {
        load_geo<MAXF, WIDE, LEAN>(a, i, nf, geo);
        const int c = a.cur0 & 1;
        own.r = a.rho[c][i];
        own.u = f3(a.rhou[c][i]);
        own.e = a.rhoe[c][i];
        st_state(&a.state[c][i], m.N, own.r, own.u, own.e, a.tag0);
        ghost_states<MAXF, WIDE, LEAN>(a, s_bc, geo, nf, c, own);
    }
    for (int it = 0; it < a.iters; ++it) {
        const int cur = (a.cur0 + it) & 1, nxt = 1 - cur;
        const unsigned int tag = a.tag0 + it;
        bool ok = true;
        if (have) ok = grad_loop_cell<TRANSPOSED, MAXF, WIDE, LEAN>(a, cur, tag, geo, i, nf, own);
        FluxSum s{};
        if (ok) {
            if (WIDE && full) ok = flux_loop_cell<MAXF, WIDE, true, LEAN>(a, tag, geo, i, nf, s);
            else if (have) ok = flux_loop_cell<MAXF, WIDE, false, LEAN>(a, tag, geo, i, nf, s);
        }
        // the update waits for the verdict on the iteration before it
        if (ok && it > 0) ok = await_verdict(a, tag);
        if (!__all_sync(0xffffffffu, ok)) return;
        float e = 0.f, rsq = 0.f;
        if (have) {
            const float dt = a.cfl / s.dts;
            own.r = own.r - s.fr * dt;
            own.u = make_float3(own.u.x - s.fu.x * dt, own.u.y - s.fu.y * dt, own.u.z - s.fu.z * dt);
            own.e = own.e - s.fe * dt;
            st_state(&a.state[nxt][i], m.N, own.r, own.u, own.e, tag + 1u);
            const float vol = geo.vol();
            // flux_cell's multiply-adds, written out: the density part below must not change them
            e = __fmul_rn(__fmaf_rn(s.fe, s.fe, __fmaf_rn(s.fr, s.fr, ydot(s.fu, s.fu))), vol);
            rsq = __fmul_rn(__fmul_rn(s.fr, s.fr), vol);
        }
        st_warp_sum(&a.wsum[chunk], (double)e, tag);
        if (a.hist_rho) st_warp_sum(&a.wsum_rho[chunk], (double)rsq, tag);
        if (have) {
            a.rho[nxt][i] = own.r;
            a.rhou[nxt][i] = make_float4(own.u.x, own.u.y, own.u.z, 0.f);
            a.rhoe[nxt][i] = own.e;
            if (a.err) a.err[i] = e;
            if (it + 1 < a.iters) ghost_states<MAXF, WIDE, LEAN>(a, s_bc, geo, nf, nxt, own);
        }
    }
}

template <bool TRANSPOSED, int MAXF, int THREADS, LoopForm FORM>
__global__ void __launch_bounds__(THREADS, kLoopBlocksPerSM) k_euler_loop(const __grid_constant__ EulerLoopArgs a) {
    extern __shared__ float s_geo[];
    __shared__ GhostBcTable s_bc;
    if (blockIdx.x == gridDim.x - 1) {
        loop_reducer(a);
        return;
    }
    for (unsigned int k = threadIdx.x; k < sizeof(GhostBcTable) / 4; k += blockDim.x)
        reinterpret_cast<uint32_t*>(&s_bc)[k] = reinterpret_cast<const uint32_t*>(&a.ghosts)[k];
    __syncthreads();
    euler_loop_worker<TRANSPOSED, MAXF, FORM == LoopForm::kWide, FORM == LoopForm::kLean>(a, s_bc, blockIdx.x, s_geo);
}

// k_batch_reduce for one instance of the batched loop.
__device__ void batch_reducer(const BatchLoopInst& a) {
    bool ok = true;
    int n = *a.n_iters;
    double res0 = *a.res0;
    for (int it = 0; it < a.iters; ++it) {
        const unsigned int tag = a.tag0 + it;
        const double bs = reduce_groups(a, a.wsum, tag, nullptr, ok);
        if (!ok) return;
        if (n == 0) res0 = a.res0_fixed > 0.0 ? a.res0_fixed : bs;
        const double ratio = res0 > 0.0 ? bs / res0 : 0.0;
        const int at = n++;
        int status = 0;
        if (!(bs == bs) || bs > 1e300) status = 3;
        else if (a.tol > 0.0 && ratio < a.tol) status = 1;
        else if (n >= a.max_iter) status = 2;
        const bool last = status || it + 1 == a.iters;
        if (threadIdx.x == 0) {
            st_relaxed64(a.verdict, (unsigned long long)status << 32 | tag);
            if (a.history) a.history[at] = bs;
            if (last) {
                *a.n_iters = n;
                *a.cur = (a.cur0 + it + 1) & 1;
                *a.res0 = res0;
                *a.ratio = ratio;
                *a.status = status;
            }
        }
        if (last) return;
        __syncthreads();
    }
}

// The loop for the instances of a batch that fit on the GPU together, one
// cell per thread: each instance has worker blocks and a reducer of its own,
// and nothing waits across instances.  Per iteration against the replayed
// graph of three kernels (B200): 2 instances of 4,608 prisms 11.4 / 21.0 us, 10
// of 57,168 together 15.7 / 23.1, 40 of 92,160 together 20.0 / 33.2.
template <bool TRANSPOSED, int MAXF, int THREADS, LoopForm FORM>
__global__ void __launch_bounds__(THREADS, kLoopBlocksPerSM)
    k_euler_loop_batch(const BatchLoopInst* __restrict__ insts, const int* __restrict__ inst_of_block) {
    extern __shared__ float s_geo[];
    __shared__ BatchLoopInst a;
    const BatchLoopInst* src = insts + inst_of_block[blockIdx.x];
    for (unsigned int k = threadIdx.x; k < sizeof(BatchLoopInst) / 4; k += blockDim.x)
        reinterpret_cast<uint32_t*>(&a)[k] = reinterpret_cast<const uint32_t*>(src)[k];
    __syncthreads();
    if (a.iters == 0) return;                     // stopped before
    const uint32_t block = blockIdx.x - (uint32_t)a.first_block;
    if (block == (uint32_t)a.n_blocks) batch_reducer(a);
    else euler_loop_worker<TRANSPOSED, MAXF, FORM == LoopForm::kWide, false>(a, a.ghosts, block, s_geo);
}

// off[g]: ghost g's face centre - its centroid
__global__ void k_ghost_off(MeshDev m, uint32_t G, const uint2* __restrict__ ghost, float4* off) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const float3 d = f3(m.face_geo[2 * ghost[g].y + 1]) - f3(m.cell_geo[m.N + g]);
    off[g] = make_float4(d.x, d.y, d.z, 0.f);
}

// Two blocks per SM leave a thread 96 registers up to 320 threads per block and
// 72 up to 416: with 72 for all, 78,000 prisms took 16.5 us per iteration (14.9
// with 96) and 90,000 15.9 (14.6).
template <bool TRANSPOSED, int MAXF>
cudaError_t launch(EulerLoopArgs& a, LoopForm form, int threads, cudaStream_t s) {
    const void* fn = form == LoopForm::kWide   ? (const void*)k_euler_loop<TRANSPOSED, MAXF, kLoopWide, LoopForm::kWide>
                     : form == LoopForm::kLean ? (const void*)k_euler_loop<TRANSPOSED, MAXF, kLoopMax, LoopForm::kLean>
                     : threads <= 320          ? (const void*)k_euler_loop<TRANSPOSED, MAXF, 320, LoopForm::kNarrow>
                                      : (const void*)k_euler_loop<TRANSPOSED, MAXF, kLoopFull, LoopForm::kNarrow>;
    const int smem = loop_smem(form, MAXF, threads);
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    void* args[] = {(void*)&a};
    const cudaError_t r = cudaLaunchCooperativeKernel(fn, dim3(a.n_blocks + 1), dim3(threads), args, smem, s);
    if (r == cudaSuccess) count_launch();
    return r;
}

template <bool TRANSPOSED, int MAXF>
cudaError_t launch_batch(const BatchLoopInst* insts, const int* inst_of_block, int blocks, LoopForm form, int threads,
                         cudaStream_t s) {
    const void* fn = form == LoopForm::kWide
                         ? (const void*)k_euler_loop_batch<TRANSPOSED, MAXF, kLoopWide, LoopForm::kWide>
                         : (const void*)k_euler_loop_batch<TRANSPOSED, MAXF, kLoopFull, LoopForm::kNarrow>;
    const int smem = loop_smem(form, MAXF, threads);
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    void* args[] = {(void*)&insts, (void*)&inst_of_block};
    const cudaError_t r = cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(threads), args, smem, s);
    if (r == cudaSuccess) count_launch();
    return r;
}

}  // namespace

cudaError_t launch_batch_loop(const BatchLoopInst* insts, const int* inst_of_block, int blocks, LoopForm form,
                              int max_faces, int threads, bool transposed, cudaStream_t s) {
    auto go = [&](auto tr) {
        constexpr bool T = decltype(tr)::value;
        if (max_faces <= 4) return launch_batch<T, 4>(insts, inst_of_block, blocks, form, threads, s);
        if (max_faces == 5) return launch_batch<T, 5>(insts, inst_of_block, blocks, form, threads, s);
        return launch_batch<T, 6>(insts, inst_of_block, blocks, form, threads, s);
    };
    return transposed ? go(std::true_type{}) : go(std::false_type{});
}

void launch_ghost_off(const DevMesh& d, float4* ghost_off, cudaStream_t s) {
    if (d.G == 0) return;
    k_ghost_off<<<(unsigned)((d.G + kBlock - 1) / kBlock), kBlock, 0, s>>>(mesh_dev(d), (uint32_t)d.G, d.ghost, ghost_off);
    count_launch();
}

cudaError_t launch_euler_loop(EulerLoopArgs& a, LoopForm form, int max_faces, int threads, bool transposed,
                              cudaStream_t s) {
    if (max_faces <= 4) return transposed ? launch<true, 4>(a, form, threads, s) : launch<false, 4>(a, form, threads, s);
    if (max_faces == 5) return transposed ? launch<true, 5>(a, form, threads, s) : launch<false, 5>(a, form, threads, s);
    return transposed ? launch<true, 6>(a, form, threads, s) : launch<false, 6>(a, form, threads, s);
}

}  // namespace gb
