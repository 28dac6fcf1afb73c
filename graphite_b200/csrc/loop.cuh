// What the persistent loops (euler_loop.cu, nsi_loop.cu) share: records that
// are handed over through L2 with the iteration they belong to, waits that
// give up, and the block that sums the residual and judges each iteration.
#pragma once

#include "euler_ops.cuh"
#include "loop_shape.h"

namespace gb {

// 16 bytes that are written and read as one: three words and the tag that
// says which iteration they belong to.
struct alignas(16) TagRec {
    uint32_t x, y, z, tag;
};

// One cell per thread, two blocks per SM.
constexpr int kLoopBlocksPerSM = 2;
// Polls of a wait before it gives up (a poll takes about half a microsecond).
constexpr unsigned int kLoopSpinLimit = 1u << 23;

// Where a wait of at most `polls` polls (0: the default) starts counting.
constexpr unsigned int loop_spin_start(unsigned int polls) {
    return polls == 0 || polls > kLoopSpinLimit ? 0u : kLoopSpinLimit - polls;
}

// A cell's neighbour word: the neighbour's index below its top four bits.
constexpr uint32_t kNbMask = (1u << 28) - 1u;

struct LoopArgs {
    uint32_t N;
    int iters, cur0;                      // iterations of the launch, value buffer it starts from
    double tol;
    RunCtl* ctl;
    double *hist, *hist_rho;              // hist_rho null: the density part is not summed
    unsigned long long hist_cap;
    double *out, *partials;               // the residual, and its sums by 256-cell group
    int n_groups, n_blocks;
    unsigned int tag0;                    // tags of this launch: tag0 + iteration
    unsigned int spin0;                   // loop_spin_start of the launch's limit
    TagRec *wsum, *wsum_rho;              // per warp: a double
    unsigned long long* verdict;          // tag of the last iteration judged (low word), halt (high word)
};

namespace {

// A record is one 16-byte access only while all four of its words are used: a
// load with dead words may be narrowed to several, which can then see two
// records.  So words without a payload carry the tag, and fresh() compares
// them all: PAYLOAD words of r are data.
template <int PAYLOAD>
__device__ __forceinline__ bool fresh(const TagRec& r, unsigned int tag) {
    return ((r.tag ^ tag) | (PAYLOAD > 2 ? 0u : r.z ^ tag) | (PAYLOAD > 1 ? 0u : r.y ^ tag)) == 0u;
}
__device__ __forceinline__ TagRec ld_rec(const TagRec* p) {
    unsigned long long lo, hi;
    asm volatile(
        "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}\n"
        : "=l"(lo), "=l"(hi)
        : "l"(p)
        : "memory");
    return TagRec{(uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32)};
}
__device__ __forceinline__ void st_rec(TagRec* p, uint32_t x, uint32_t y, uint32_t z, uint32_t tag) {
    const unsigned long long lo = (unsigned long long)y << 32 | x, hi = (unsigned long long)tag << 32 | z;
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%0, %1};\n\tst.relaxed.gpu.global.b128 [%2], t;\n\t}\n" ::"l"(lo),
                 "l"(hi), "l"(p)
                 : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(v) : "memory");
}

// Counts the polls of one wait up to kLoopSpinLimit; false once it, or another
// one, has given up.  A shorter limit is a later start, so that the test of
// every 256th poll is all there is either way.
struct Patience {
    unsigned int n;
    int* error;
    __device__ __forceinline__ explicit Patience(const LoopArgs& a) : n(a.spin0), error(&a.ctl->error) {}
    __device__ __forceinline__ bool more() {
        if ((++n & 255u) == 0u && (n >= kLoopSpinLimit || *(volatile int*)error)) {
            atomicExch(error, 1);
            return false;
        }
        return true;
    }
};

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    return x;
}

// The residual of one iteration from the per-warp sums tagged `tag`, in the
// order of k_flux's block sums and k_reduce_final: 8 warps to a 256-cell group
// (into `groups`), the groups strided over 256 (virtual) threads, then the
// block tree.  Every thread of the block calls it and gets the sum; ok turns
// false when a wait gave up.
__device__ double reduce_groups(const LoopArgs& a, const TagRec* wsum, unsigned int tag, double* groups, bool& ok) {
    __shared__ double sv[kBlock];
    __shared__ double sw[kBlock / 32];
    const uint32_t n_warps = (a.N + 31) / 32;
    const int n_groups = a.n_groups;
    Patience wait(a);
    for (int v = threadIdx.x; v < kBlock; v += blockDim.x) {
        double s = 0.0;
        for (int i = v; i < n_groups; i += kBlock) {
            double w[8];
            unsigned int pending = 0xffu;
            while (pending && ok) {
                unsigned int left = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (!(pending & (1u << k))) continue;
                    w[k] = 0.0;
                    if (8u * i + k >= n_warps) continue;
                    const TagRec r = ld_rec(&wsum[8 * i + k]);
                    w[k] = __hiloint2double((int)r.y, (int)r.x);
                    if (!fresh<2>(r, tag)) left |= 1u << k;
                }
                pending = left;
                if (pending) ok = wait.more();
            }
            const double g = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
            if (groups) groups[i] = g;
            s += g;
        }
        sv[v] = s;
    }
    ok = !__syncthreads_or(!ok);
    const int lane = threadIdx.x & 31;
    for (int w = threadIdx.x >> 5; w < kBlock / 32; w += blockDim.x >> 5) {
        const double x = warp_sum(sv[32 * w + lane]);
        if (lane == 0) sw[w] = x;
    }
    __syncthreads();
    return ((sw[0] + sw[4]) + (sw[2] + sw[6])) + ((sw[1] + sw[5]) + (sw[3] + sw[7]));
}

// The block after the workers: residual, history and stop test of each
// iteration (k_reduce_final's).
__device__ void loop_reducer(const LoopArgs& a) {
    RunCtl* ctl = a.ctl;
    const unsigned long long run0 = ctl->it_run;
    double res0 = ctl->res0;
    bool ok = true;
    for (int it = 0; it < a.iters; ++it) {
        const unsigned int tag = a.tag0 + it;
        const double bs = reduce_groups(a, a.wsum, tag, nullptr, ok);
        double rs = 0.0;
        if (a.hist_rho) {
            __syncthreads();
            rs = reduce_groups(a, a.wsum_rho, tag, nullptr, ok);
        }
        if (!ok) return;
        if (run0 + it == 0) res0 = bs;
        unsigned int halt = 0;
        if (!(bs == bs) || bs > 1e300) halt = 2;
        else if (a.tol > 0.0 && res0 > 0.0 && bs / res0 < a.tol) halt = 1;
        const bool last = halt || it + 1 == a.iters;
        if (last) {
            __syncthreads();
            reduce_groups(a, a.wsum, tag, a.partials, ok);
        }
        if (threadIdx.x == 0) {
            st_relaxed64(a.verdict, (unsigned long long)halt << 32 | tag);
            if ((unsigned long long)it < a.hist_cap) {
                a.hist[it] = bs;
                if (a.hist_rho) a.hist_rho[it] = rs;
            }
            if (last) {
                a.out[0] = bs;
                ctl->it_chunk = it + 1;
                ctl->it_run = run0 + it + 1;
                ctl->res0 = res0;
                ctl->halt = halt;
            }
        }
        if (last) return;
        __syncthreads();
    }
}

// Whether the update of iteration `tag` may happen: false when the iteration
// before it has stopped the loop, or the wait for its verdict gave up.
__device__ __forceinline__ bool await_verdict(const LoopArgs& a, unsigned int tag) {
    Patience wait(a);
    for (;;) {
        const unsigned long long v = ld_relaxed64(a.verdict);
        if ((unsigned int)v >= tag - 1u) return (v >> 32) == 0;
        if (!wait.more()) return false;
    }
}

// Hands a warp's sum of x (a double per lane, valid lanes or zero) to the reducer.
__device__ __forceinline__ void st_warp_sum(TagRec* p, double x, unsigned int tag) {
    const double s = warp_sum(x);
    if ((threadIdx.x & 31) == 0) st_rec(p, (uint32_t)__double2loint(s), (uint32_t)__double2hiint(s), tag, tag);
}

}  // namespace
}  // namespace gb
