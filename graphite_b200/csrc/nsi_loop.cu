// The incompressible loop of a mesh that fits on the GPU one cell per thread,
// as one persistent launch for many iterations: the scheme of euler_loop.cu
// (geometry and state on chip, tagged records through L2, no barrier between
// cells) with what this model hands over -- a cell's state for its
// neighbours' gradients, and its gradients (with its limiters where it has
// any) for their fluxes, one set per cell instead of one per face, because
// the viscous flux needs the whole velocity gradient.  A new state is written
// after reading the neighbours' gradients, which they form after reading the
// old one; new gradients after reading the neighbours' new states, which they
// form after reading the old gradients.  Bound like euler_loop.cu by the latency
// of a cell's chain: 100,000 hexes in one layer, 21 warps per SM, issue slots
// 39 % busy, L2 at 16 % of its throughput, 7.9 warps waiting for memory per
// instruction issued.  Per iteration in launches of 100 against the replayed
// graph (B200): 27,984 hexes in one layer 7.9 / 19.9 us, 28,350 tets 7.5 / 27.2,
// 54,096 hexes 8.9 / 22.9, 89,823 hexes 20.3 / 27.4, 104,960 hexes 22.4 / 29.1; with
// the limiter 14.4 / 24.2, 16.2 / 33.3, 15.4 / 26.3, 27.6 / 30.7 and 29.1 / 31.3; where
// it loses and is not taken: loop_shape.h.
#include "nsi_loop.cuh"

#include <algorithm>

namespace gb {
namespace {

// One cell's entries in shared memory, [slot][component][cell of the block]:
// the neighbour word (index, and a ghost's region in the top four bits), the
// offsets of the neighbour, of the face centre and of the face centre from the
// neighbour, with WIDE the outward normal and area / volume; then the
// least-squares inverse and the volume.
template <int MAXF, bool WIDE>
struct NsiGeo {
    static constexpr int kLsq = (WIDE ? 14 : 10) * MAXF;
    float* base;
    int T;
    const float4* cf_geo;   // !WIDE: this cell's first entry in the mesh's array, N entries to the next slot
    uint32_t N;
    __device__ __forceinline__ uint32_t& nb(int t) const { return reinterpret_cast<uint32_t*>(base)[t * T]; }
    __device__ __forceinline__ float& v(int t, int k) const { return base[(MAXF + 9 * t + k) * T]; }
    __device__ __forceinline__ float& cf(int t, int k) const { return base[(10 * MAXF + 4 * t + k) * T]; }
    __device__ __forceinline__ float& lsq(int k) const { return base[(kLsq + k) * T]; }
    __device__ __forceinline__ float& vol() const { return base[(kLsq + 6) * T]; }
    __device__ __forceinline__ float3 v3(int t, int k) const { return make_float3(v(t, k), v(t, k + 1), v(t, k + 2)); }
    __device__ __forceinline__ float3 dn3(int t) const { return v3(t, 0); }
    __device__ __forceinline__ float3 df3(int t) const { return v3(t, 3); }
    __device__ __forceinline__ float3 dg3(int t) const { return v3(t, 6); }
    __device__ __forceinline__ float4 cf4(int t) const {
        if (!WIDE) return __ldg(cf_geo + (size_t)t * N);
        return make_float4(cf(t, 0), cf(t, 1), cf(t, 2), cf(t, 3));
    }
    // 1 / |dn|^2 and |df|^3 as entry_geo_cell forms them
    __device__ __forceinline__ float w2(float3 d) const { return fast_rcp(ydot(d, d)); }
    __device__ __forceinline__ float k3(float3 d) const {
        float l;
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(ydot(d, d)));
        return __fmul_rn(__fmul_rn(l, l), l);
    }
};

struct NsiState {
    float p;
    float3 u;
};

// The records of a state, and of a set of gradients, lie `plane` apart: the
// lanes of a warp read and write whole sectors of each plane.
__device__ __forceinline__ void st_nsi(TagRec* r, size_t plane, const NsiState& q, unsigned int tag) {
    st_rec(r, __float_as_uint(q.p), __float_as_uint(q.u.x), __float_as_uint(q.u.y), tag);
    st_rec(r + plane, __float_as_uint(q.u.z), tag, tag, tag);
}
__device__ __forceinline__ bool ld_nsi(const TagRec* r, size_t plane, unsigned int tag, NsiState& q) {
    const TagRec a = ld_rec(r), b = ld_rec(r + plane);
    q.p = __uint_as_float(a.x);
    q.u = make_float3(__uint_as_float(a.y), __uint_as_float(a.z), __uint_as_float(b.x));
    return fresh<3>(a, tag) && fresh<1>(b, tag);
}

// g[0] the pressure's gradient and limiter, g[1..3] the velocity components'
__device__ __forceinline__ void st_grads(TagRec* r, size_t plane, const float4 g[4], int limited, unsigned int tag) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
        st_rec(r + c * plane, __float_as_uint(g[c].x), __float_as_uint(g[c].y), __float_as_uint(g[c].z), tag);
    if (!limited) return;
    st_rec(r + 4 * plane, __float_as_uint(g[0].w), __float_as_uint(g[1].w), __float_as_uint(g[2].w), tag);
    st_rec(r + 5 * plane, __float_as_uint(g[3].w), tag, tag, tag);
}
__device__ __forceinline__ bool ld_grads(const TagRec* r, size_t plane, int limited, unsigned int tag, float4 g[4]) {
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const TagRec a = ld_rec(r + c * plane);
        g[c] = make_float4(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), 1.f);
        ok = ok && fresh<3>(a, tag);
    }
    if (limited) {
        const TagRec a = ld_rec(r + 4 * plane), b = ld_rec(r + 5 * plane);
        g[0].w = __uint_as_float(a.x);
        g[1].w = __uint_as_float(a.y);
        g[2].w = __uint_as_float(a.z);
        g[3].w = __uint_as_float(b.x);
        ok = ok && fresh<3>(a, tag) && fresh<1>(b, tag);
    }
    return ok;
}

// The ghost across entry t: its region's condition on the cell's own state, or
// its stored state.
template <class Geo>
__device__ __forceinline__ NsiState ghost_of(const NsiLoopArgs& a, const NsiGhostTable& bc, const Geo& g, int t,
                                             uint32_t word, int buf, const NsiState& own) {
    NsiState q;
    const int k = word >> 28;
    if (bc.type[k] >= 0) {
        nsi_ghost_state(bc.type[k], f3(g.cf4(t)), own.p, own.u, bc.vinf[k], bc.pinf[k], q.p, q.u);
    } else {
        const uint32_t j = word & kNbMask;
        q.p = __ldcg(&a.p[buf][j]);
        q.u = f3(__ldcg(&a.u[buf][j]));
    }
    return q;
}

// k_nsi_grad for one cell.  False: a wait gave up.
template <int MAXF, bool WIDE>
__device__ __forceinline__ bool nsi_grad_cell(const NsiLoopArgs& a, const NsiGhostTable& bc,
                                              const NsiGeo<MAXF, WIDE>& g, int buf, unsigned int tag, int nf,
                                              const NsiState& own, float4 out[4]) {
    const uint32_t N = a.N;
    const TagRec* nbs = a.state[buf];
    const float v[4] = {own.p, own.u.x, own.u.y, own.u.z};
    float3 gs[4];
    float vmin[4], vmax[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) { gs[c] = make_float3(0.f, 0.f, 0.f); vmin[c] = v[c]; vmax[c] = v[c]; }
    Patience wait(a);
    auto add = [&](int t, const NsiState& q) {
        const float3 d = g.dn3(t);
        const float w = g.w2(d);
        const float vj[4] = {q.p, q.u.x, q.u.y, q.u.z};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            gs[c] = gs[c] + (d * (vj[c] - v[c])) * w;
            vmin[c] = fminf(vmin[c], vj[c]);
            vmax[c] = fmaxf(vmax[c], vj[c]);
        }
    };
    if constexpr (WIDE) {
        NsiState q[MAXF];
        unsigned int pending = 0;
#pragma unroll
        for (int t = 0; t < MAXF; ++t)
            if (t < nf && (g.nb(t) & kNbMask) < N) pending |= 1u << t;
        for (;;) {
            unsigned int left = 0;
#pragma unroll
            for (int t = 0; t < MAXF; ++t)
                if (pending & (1u << t))
                    if (!ld_nsi(&nbs[g.nb(t) & kNbMask], N, tag, q[t])) left |= 1u << t;
            pending = left;
            if (pending == 0) break;
            if (!wait.more()) return false;
        }
#pragma unroll
        for (int t = 0; t < MAXF; ++t) {
            if (t >= nf) continue;
            const uint32_t word = g.nb(t);
            add(t, (word & kNbMask) < N ? q[t] : ghost_of(a, bc, g, t, word, buf, own));
        }
    } else {
#pragma unroll 1
        for (int t = 0; t < nf; ++t) {
            const uint32_t word = g.nb(t), j = word & kNbMask;
            NsiState q;
            if (j < N) {
                while (!ld_nsi(&nbs[j], N, tag, q))
                    if (!wait.more()) return false;
            } else {
                q = ghost_of(a, bc, g, t, word, buf, own);
            }
            add(t, q);
        }
    }
    const float4 l0 = make_float4(g.lsq(0), g.lsq(1), g.lsq(2), g.lsq(3)), l1 = make_float4(g.lsq(4), g.lsq(5), 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < 4; ++c) gs[c] = sym_mul(l0, l1, gs[c]);
    float lim[4] = {1.f, 1.f, 1.f, 1.f};
    if (a.limited) {
        lim[0] = lim[1] = lim[2] = lim[3] = 2.f;
#pragma unroll 1
        for (int t = 0; t < nf; ++t) {
            const float3 d = g.df3(t);
            const float k3 = g.k3(d);
#pragma unroll
            for (int c = 0; c < 4; ++c) lim[c] = fminf(lim[c], limiter(v[c], gs[c], vmin[c], vmax[c], d, k3));
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) out[c] = make_float4(gs[c].x, gs[c].y, gs[c].z, lim[c]);
    return true;
}

// k_nsi_flux's sum over the faces of one cell.  False: a wait gave up.
template <int MAXF, bool WIDE>
__device__ __forceinline__ bool nsi_flux_cell(const NsiLoopArgs& a, const NsiGhostTable& bc,
                                              const NsiGeo<MAXF, WIDE>& g, int buf, unsigned int tag, int nf,
                                              const NsiState& own, const float4 go[4], NsiSum& s) {
    const uint32_t N = a.N;
    Patience wait(a);
#pragma unroll 1
    for (int t = 0; t < nf; ++t) {
        const uint32_t word = g.nb(t), j = word & kNbMask;
        NsiState q;
        float4 gn[4];
        if (j < N) {
            ld_nsi(&a.state[buf][j], N, tag, q);       // read before, by the gradient pass
            while (!ld_grads(&a.grad[j], N, a.limited, tag, gn))
                if (!wait.more()) return false;
        } else {
            // a ghost carries its interior cell's gradient and limiter
            q = ghost_of(a, bc, g, t, word, buf, own);
#pragma unroll
            for (int c = 0; c < 4; ++c) gn[c] = go[c];
        }
        const float4 c = g.cf4(t);
        const float3 d = g.dn3(t);
        s.face(a.par, own.p, own.u, go[0], go + 1, q.p, q.u, gn[0], gn + 1, f3(c), c.w, g.df3(t), g.dg3(t),
               make_float4(d.x, d.y, d.z, g.w2(d)));
    }
    return true;
}

template <int MAXF, int THREADS>
__global__ void __launch_bounds__(THREADS, kLoopBlocksPerSM) k_nsi_loop(const __grid_constant__ NsiLoopArgs a) {
    constexpr bool WIDE = THREADS <= kNsiWide;
    extern __shared__ float s_geo[];
    __shared__ NsiGhostTable s_bc;
    if (blockIdx.x == gridDim.x - 1) {
        loop_reducer(a);
        return;
    }
    const MeshDev& m = a.m;
    for (unsigned int k = threadIdx.x; k < sizeof(NsiGhostTable) / 4; k += blockDim.x)
        reinterpret_cast<uint32_t*>(&s_bc)[k] = reinterpret_cast<const uint32_t*>(&a.ghosts)[k];
    __syncthreads();
    const uint32_t chunk = (threadIdx.x >> 5) * (uint32_t)a.n_blocks + blockIdx.x;
    const uint32_t i = 32u * chunk + (threadIdx.x & 31);
    if (32u * chunk >= m.N) return;
    const bool have = i < m.N;
    const NsiGeo<MAXF, WIDE> g{s_geo + threadIdx.x, (int)blockDim.x, m.cf_geo + i, m.N};
    const int nf = have ? __ldg(&m.nfc[i]) : 0;
    NsiState own{};
    if (have) {
        const float4 l0 = __ldg(&m.lsq[2 * i]), l1 = __ldg(&m.lsq[2 * i + 1]);
        g.lsq(0) = l0.x; g.lsq(1) = l0.y; g.lsq(2) = l0.z; g.lsq(3) = l0.w; g.lsq(4) = l1.x; g.lsq(5) = l1.y;
        g.vol() = __ldg(&m.cell_geo[i]).w;
#pragma unroll 1
        for (int t = 0; t < nf; ++t) {
            const uint32_t k = i + t * m.N, j = __ldg(&m.nbc[k]);
            uint32_t top = 0;
            float4 o;
            if (j < m.N) {
                o = __ldg(&m.df[__ldg(&m.twin[k])]);
            } else {
                while ((int)top < a.ghosts.n - 1 && j >= a.ghosts.start[top + 1]) ++top;
                o = __ldg(&a.ghost_off[j - m.N]);
            }
            g.nb(t) = j | (top << 28);
            const float4 n = __ldg(&m.dn[k]), b = __ldg(&m.df[k]);
            g.v(t, 0) = n.x; g.v(t, 1) = n.y; g.v(t, 2) = n.z;
            g.v(t, 3) = b.x; g.v(t, 4) = b.y; g.v(t, 5) = b.z;
            g.v(t, 6) = o.x; g.v(t, 7) = o.y; g.v(t, 8) = o.z;
            if (WIDE) {
                const float4 c = __ldg(&m.cf_geo[k]);
                g.cf(t, 0) = c.x; g.cf(t, 1) = c.y; g.cf(t, 2) = c.z; g.cf(t, 3) = c.w;
            }
        }
        const int c = a.cur0 & 1;
        own.p = a.p[c][i];
        own.u = f3(a.u[c][i]);
        st_nsi(&a.state[c][i], m.N, own, a.tag0);
    }
    for (int it = 0; it < a.iters; ++it) {
        const int cur = (a.cur0 + it) & 1, nxt = 1 - cur;
        const unsigned int tag = a.tag0 + it;
        bool ok = true;
        float4 go[4] = {};
        NsiSum s{};
        if (have) {
            ok = nsi_grad_cell<MAXF, WIDE>(a, s_bc, g, cur, tag, nf, own, go);
            if (ok) {
                st_grads(&a.grad[i], m.N, go, a.limited, tag);
                ok = nsi_flux_cell<MAXF, WIDE>(a, s_bc, g, cur, tag, nf, own, go, s);
            }
        }
        // the update waits for the verdict on the iteration before it
        if (ok && it > 0) ok = await_verdict(a, tag);
        if (!__all_sync(0xffffffffu, ok)) return;
        float e = 0.f;
        if (have) {
            const float dt = a.par.cfl / s.sr;
            own.p = own.p - s.rp * dt;
            own.u = make_float3(own.u.x - s.ru.x * dt, own.u.y - s.ru.y * dt, own.u.z - s.ru.z * dt);
            st_nsi(&a.state[nxt][i], m.N, own, tag + 1u);
            e = __fmul_rn(__fmaf_rn(s.rp, s.rp, ydot(s.ru, s.ru)), g.vol());
        }
        st_warp_sum(&a.wsum[chunk], (double)e, tag);
        if (have) {
            a.p[nxt][i] = own.p;
            a.u[nxt][i] = make_float4(own.u.x, own.u.y, own.u.z, 0.f);
            a.err[i] = e;
        }
    }
}

// Registers a thread: 128, 80 up to 352 threads per block, 72 up to 448, 64.  With
// 64 for all above 256 threads 90,000 hexes took 24.6 us per iteration (18.4), 112,000
// 30.0 (20.7), 126,000 tets 31.8 (21.6), with the limiter 31.9 (26.7), 36.6 (29.9) and
// 45.7 (39.3).
template <int MAXF>
cudaError_t launch(NsiLoopArgs& a, int threads, cudaStream_t s) {
    const void* fn = threads <= kNsiWide ? (const void*)k_nsi_loop<MAXF, kNsiWide>
                     : threads <= 352    ? (const void*)k_nsi_loop<MAXF, 352>
                     : threads <= 448    ? (const void*)k_nsi_loop<MAXF, 448>
                                         : (const void*)k_nsi_loop<MAXF, kNsiMax>;
    const int smem = nsi_loop_smem(MAXF, threads);
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    void* args[] = {(void*)&a};
    const cudaError_t r = cudaLaunchCooperativeKernel(fn, dim3(a.n_blocks + 1), dim3(threads), args, smem, s);
    if (r == cudaSuccess) count_launch();
    return r;
}

}  // namespace

cudaError_t launch_nsi_loop(NsiLoopArgs& a, int max_faces, int threads, cudaStream_t s) {
    if (max_faces <= 4) return launch<4>(a, threads, s);
    if (max_faces == 5) return launch<5>(a, threads, s);
    return launch<6>(a, threads, s);
}

}  // namespace gb
