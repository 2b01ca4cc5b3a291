// 3D radius-1 FP32 steps, k per pass over the state, with the tile in
// registers: vvsl_field_rescaled (src/standard/s_integrate.cpp:305-348).
//
// A pass of k steps reads psi_n and pih_{n-1} once and writes psi_{n+k} and
// pih_{n+k-1}: 32 B per site for k site-updates. The two-step kernel
// (k_zmarch_2step_lean) is at 0.89 of the HBM copy rate, so more steps per pass is what
// is left; through shared-memory rings a third step made the pass issue-bound
// (80 instructions per site-update, most of them shared-memory traffic). Here it takes
// 43 (three steps per pass on 12 warps of four rows), 32 per computed one:
//  * a block takes a tile of tx x TY sites with a k-site halo (columns rounded
//    up to pairs) through a z-chunk; lane i of warp w holds two neighbouring
//    sites of V rows, the warps lie above one another. The x neighbours come by
//    shuffles, the y neighbours from the thread's own rows, the z neighbours from
//    its own registers; both components go through packed FP32 operations;
//  * iteration j of the march does step 1 on plane m, step 2 on plane m - 1, ...
//    step k on plane m - k + 1. Step s needs psi_{n+s-1} of three planes: the
//    last arrives from step s - 1 in this iteration, in the same thread, and the
//    other two wait in registers, with the momentum of the plane between them.
//    What crosses threads, the first and last row of each warp, belongs to the
//    middle plane, which is one iteration old: one barrier per plane for all k
//    steps;
//  * psi_n and pih_{n-1} arrive by cp.async in a ring of own-thread slots (the
//    warps above and below read their edge rows from it too), AHEAD planes before
//    they are used, so that 40 KB per plane are in flight and hold no registers.
// Columns and rows past the shrinking region carry values that nobody reads. One
// site's operations are those of the other kernels (lap7, site_update), so any
// grouping of steps into passes gives the same bits. psi and pih are written
// out of place.
//
// Measured (GB300, us per step; two steps per pass through shared memory in
// brackets): 1024^3 2287 (2840), 512^3 313 (378), 256^3 47 (68), 128^3 9.9 (12.4).
// (The 1024^3 figure is that of intervals of whole three-step passes; a pass of two steps
// costs as much, so the tuner gives it to the two-step kernel: 20 steps 2340 per step.) At 512^3 with z-chunks of 128 planes (more
// planes than the tuner's choice there) a three-step pass issues 47 % of the time with three
// warps per scheduler, DRAM 54 %: the bound is the latency
// between issues, and the halo (1.35 sites computed per site kept). Tried and slower at 1024^3:
// rows chained through all steps with the planes in rotation (no register moves,
// less parallelism), 2420; barriers between neighbouring warps only, 2470; 16 warps
// of three rows (128 registers, spills), over 2490.
#include <algorithm>

#include "axs_internal.h"
#include "axs_tma.cuh"

namespace axs {

template <int K, int NW, int VR>
struct ZKCfg {
    static constexpr int V = VR, NT = 32 * NW, RY = V * NW;
    static constexpr int PLANE = V * NT * 16;                     // one field's plane in the ring, bytes
    static constexpr int EDGE = (K > 1 ? K - 1 : 0) * NW * 2 * 512;   // edge rows of steps 2 .. K, one buffer
    static constexpr int LIMIT = 232448 - 1024;
    static constexpr int AHEAD = (5 + 4) * PLANE + 2 * EDGE <= LIMIT ? 2 : 1;   // planes in flight
    static_assert((4 + 3) * PLANE + 2 * EDGE <= LIMIT, "the ring fits shared memory");
    static constexpr int DP = 3 + AHEAD, DQ = 2 + AHEAD;          // slots of psi and of pih
    static constexpr int SMEM = (DP + DQ) * PLANE + 2 * EDGE + 256;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// One step of two neighbouring sites (c[0], c[1]); same operations as update_vec2.
__device__ __forceinline__ void update_pair(const float2 (&c)[2], float2 left, float2 right, const float2 (&ym)[2],
                                            const float2 (&yp)[2], const float2 (&zm)[2], const float2 (&zp)[2],
                                            float2 (&p)[2], float2 (&o)[2], const StepCoefs<float> &cf) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float2 S = vnsum(i == 0 ? left : c[0], i == 0 ? c[1] : right, ym[i], yp[i], zm[i], zp[i]);
        const float2 L = vfma(-6.f, c[i], S);
        const float r = fmaf(c[i].x, c[i].x, fmaf(c[i].y, c[i].y, cf.c0)), g = cf.kdt_coef * r;
        p[i] = vfma(cf.kdt_idx2, L, vfma(g, c[i], p[i]));
        o[i] = vfma(cf.dt, p[i], c[i]);
    }
}
__device__ __forceinline__ void lds_pair(float2 (&d)[2], const unsigned char *p) {
    const float4 q = *reinterpret_cast<const float4 *>(p);
    d[0] = make_float2(q.x, q.y);
    d[1] = make_float2(q.z, q.w);
}
__device__ __forceinline__ void st_pair(void *p, const float2 (&d)[2]) {
    *reinterpret_cast<float4 *>(p) = make_float4(d[0].x, d[0].y, d[1].x, d[1].y);
}

template <int K, int NW, int VR>
__global__ void __launch_bounds__(32 * NW, 1) k_zmarch_k(const ZLat *__restrict__ lats, int nlat, int64_t total_items,
                                                         int *counters, int parity) {
    typedef ZKCfg<K, NW, VR> G;
    constexpr int V = G::V, NT = G::NT, A = G::AHEAD, DP = G::DP, DQ = G::DQ;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *ring = smem, *qring = smem + DP * G::PLANE, *edges = qring + DQ * G::PLANE;
    StepCoefs<float> *scoef = reinterpret_cast<StepCoefs<float> *>(edges + 2 * G::EDGE);
    volatile int64_t *next_item = reinterpret_cast<volatile int64_t *>(scoef + K);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int wu = w > 0 ? w - 1 : 0, wd = w < NW - 1 ? w + 1 : w;
    constexpr int HX = (K + 1) & ~1;
    const int own = tid * 16;                                        // the thread's slot of row 0 in a plane
    const int above = ((V - 1) * NT + wu * 32 + lane) * 16;          // the row before the warp's first ...
    const int below = (wd * 32 + lane) * 16;                         // ... and the one after its last, in the ring
    if (tid == 0) *next_item = (int64_t)atomicAdd(&counters[0], 1);
    for (;;) {
        __syncthreads();   // the item is there; the previous item's coefficients are no longer read
        const int64_t item = *next_item;
        if (item >= total_items) break;
        const ZLat &Lt = lats[find_lat(lats, nlat, item)];
        const int N = Lt.N, tx = Lt.tx, TY = Lt.ty, ntx = Lt.ntx, nty = Lt.nty, nzc = Lt.nzc;
        const int64_t local = item - Lt.item_base;
        const int ncols = ntx * nty, zq = (int)(local / ncols), col = (int)(local % ncols);
        const int x0 = (col % ntx) * tx, y0 = (col / ntx) * TY;
        const int za = (int)((int64_t)zq * N / nzc), zb = (int)((int64_t)(zq + 1) * N / nzc);
        const int bin = Lt.a_index ^ parity;
        if (tid < K) {   // step tid: tau advanced as single steps advance it
            double tau = Lt.clock[bin];
            for (int s = 0; s < tid; ++s) tau = tau + Lt.dt;
            scoef[tid] = make_coefs<float>(tau, Lt.dt, Lt.dt, Lt.inv_dx2, Lt.lambda, Lt.T0sq3, Lt.prs, Lt.form);
            if (tid == K - 1 && local == 0) Lt.clock[bin ^ 1] = tau + Lt.dt;
        }
        const size_t NN8 = (size_t)N * N * 8;
        const char *psi = reinterpret_cast<const char *>(Lt.psi[bin]), *pih = reinterpret_cast<const char *>(Lt.pih[bin]);
        char *psi_out = reinterpret_cast<char *>(Lt.psi[bin ^ 1]), *pih_out = reinterpret_cast<char *>(Lt.pih[bin ^ 1]);
        unsigned off[V];       // byte offsets of the thread's rows within a plane (below 2^31: N <= 4096)
        unsigned stores = 0;   // bit v: row v holds sites of the tile that are in the lattice
        {
            int gx = (x0 - HX + 2 * lane) % N, gy = (y0 - K + w * V) % N;
            if (gx < 0) gx += N;
            if (gy < 0) gy += N;
            const int lx = 2 * lane - HX;
            const bool okx = lx >= 0 && lx < tx && x0 + lx < N;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                off[v] = (unsigned)(gy * N + gx) * 8u;
                gy = gy + 1 == N ? 0 : gy + 1;
                const int ly = w * V + v - K;
                if (okx && ly >= 0 && ly < TY && y0 + ly < N) stores |= 1u << v;
            }
        }
        // loads q = 0 .. nload - 1 are the planes za - K + q; iteration j uses psi's
        // j .. j + 2 and pih's j + 1
        const int J = zb - za + 2 * (K - 1), nload = J + 2;
        int lz = (za - K) % N;
        if (lz < 0) lz += N;
        int lp = 0, lq = 0;   // the ring slots of the next load
        int issued = 0;
        auto issue = [&]() {
            if (issued < nload) {
                const char *sp = psi + (size_t)lz * NN8, *sq = pih + (size_t)lz * NN8;
                const uint32_t dp = smem_u32(ring + lp * G::PLANE + own), dq = smem_u32(qring + lq * G::PLANE + own);
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    cp_async16(dp + v * NT * 16, sp + off[v]);
                    cp_async16(dq + v * NT * 16, sq + off[v]);
                }
                lz = lz + 1 == N ? 0 : lz + 1;
                lp = lp + 1 == DP ? 0 : lp + 1;
                lq = lq + 1 == DQ ? 0 : lq + 1;
                ++issued;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int q = 0; q < 2 + A; ++q) issue();
        // steps 2 .. K: planes before and at the centre, and the centre's momentum
        float2 zm[K > 1 ? K - 1 : 1][V][2], zc[K > 1 ? K - 1 : 1][V][2], pc[K > 1 ? K - 1 : 1][V][2];
#pragma unroll
        for (int s = 0; s < K - 1; ++s)
#pragma unroll
            for (int v = 0; v < V; ++v)
#pragma unroll
                for (int i = 0; i < 2; ++i) zm[s][v][i] = zc[s][v][i] = pc[s][v][i] = make_float2(0.f, 0.f);
        int s0 = 0, sq1 = 1;   // ring slots of psi's plane j and pih's j + 1
        int zo = (za - (K - 1) - (K - 1)) % N;   // the plane of step K
        if (zo < 0) zo += N;
        for (int j = 0; j < J; ++j) {
            asm volatile("cp.async.wait_group %0;" ::"n"(A - 1) : "memory");   // loads up to j + 2 are in
            unsigned char *eb = edges + (j & 1) * G::EDGE;
#pragma unroll
            for (int s = 0; s < K - 1; ++s) {
                st_pair(eb + ((s * NW + w) * 2 + 0) * 512 + lane * 16, zc[s][0]);
                st_pair(eb + ((s * NW + w) * 2 + 1) * 512 + lane * 16, zc[s][V - 1]);
            }
            __syncthreads();
            issue();   // over load j - 1, last read (as a centre) an iteration before the previous barrier
            if (tid == 0 && j == J - 1) *next_item = (int64_t)atomicAdd(&counters[0], 1);
            const int s1 = s0 + 1 >= DP ? s0 + 1 - DP : s0 + 1, s2 = s0 + 2 >= DP ? s0 + 2 - DP : s0 + 2;
            const unsigned char *Pm = ring + s0 * G::PLANE, *Pc = ring + s1 * G::PLANE, *Pp = ring + s2 * G::PLANE;
            const unsigned char *Qc = qring + sq1 * G::PLANE;
            s0 = s1;
            sq1 = sq1 + 1 == DQ ? 0 : sq1 + 1;
            float2 o[V][2], p[V][2];   // the running step's output
            {
                const StepCoefs<float> cf = scoef[0];
                float2 c[V + 2][2];   // rows -1 .. V of the centre plane
                lds_pair(c[0], Pc + above);
                lds_pair(c[V + 1], Pc + below);
#pragma unroll
                for (int v = 0; v < V; ++v) lds_pair(c[v + 1], Pc + own + v * NT * 16);
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    float2 m[2], n[2];
                    lds_pair(m, Pm + own + v * NT * 16);
                    lds_pair(n, Pp + own + v * NT * 16);
                    lds_pair(p[v], Qc + own + v * NT * 16);
                    const float2 left = make_float2(__shfl_up_sync(0xffffffffu, c[v + 1][1].x, 1), __shfl_up_sync(0xffffffffu, c[v + 1][1].y, 1));
                    const float2 right = make_float2(__shfl_down_sync(0xffffffffu, c[v + 1][0].x, 1), __shfl_down_sync(0xffffffffu, c[v + 1][0].y, 1));
                    update_pair(c[v + 1], left, right, c[v], c[v + 2], m, n, p[v], o[v], cf);
                }
            }
#pragma unroll
            for (int s = 0; s < K - 1; ++s) {   // step s + 2
                const StepCoefs<float> cf = scoef[s + 1];
                float2 up[2], dn[2], o2[V][2], p2[V][2];
                lds_pair(up, eb + ((s * NW + wu) * 2 + 1) * 512 + lane * 16);
                lds_pair(dn, eb + ((s * NW + wd) * 2 + 0) * 512 + lane * 16);
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const float2(&c)[2] = zc[s][v];
                    const float2 left = make_float2(__shfl_up_sync(0xffffffffu, c[1].x, 1), __shfl_up_sync(0xffffffffu, c[1].y, 1));
                    const float2 right = make_float2(__shfl_down_sync(0xffffffffu, c[0].x, 1), __shfl_down_sync(0xffffffffu, c[0].y, 1));
                    p2[v][0] = pc[s][v][0];
                    p2[v][1] = pc[s][v][1];
                    update_pair(c, left, right, v > 0 ? zc[s][v > 0 ? v - 1 : 0] : up, v < V - 1 ? zc[s][v < V - 1 ? v + 1 : 0] : dn,
                                zm[s][v], o[v], p2[v], o2[v], cf);
                }
#pragma unroll
                for (int v = 0; v < V; ++v)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        zm[s][v][i] = zc[s][v][i];
                        zc[s][v][i] = o[v][i];
                        pc[s][v][i] = p[v][i];
                        o[v][i] = o2[v][i];
                        p[v][i] = p2[v][i];
                    }
            }
            if (j >= 2 * (K - 1)) {
                char *po = psi_out + (size_t)zo * NN8, *qo = pih_out + (size_t)zo * NN8;
#pragma unroll
                for (int v = 0; v < V; ++v)
                    if ((stores >> v) & 1u) {
                        st_pair(po + off[v], o[v]);
                        st_pair(qo + off[v], p[v]);
                    }
            }
            zo = zo + 1 == N ? 0 : zo + 1;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&counters[1], 1) == (int)gridDim.x - 1) {
            counters[0] = 0;
            counters[1] = 0;
            __threadfence();
        }
    }
}

template <int K, int NW, int VR>
static int prepare_k_t() {
    static PerDevice occ;   // the attribute belongs to the device
    return occ.get([] {
        const auto kern = k_zmarch_k<K, NW, VR>;
        AXS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ZKCfg<K, NW, VR>::SMEM));
        int o = 0;
        AXS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, 32 * NW, ZKCfg<K, NW, VR>::SMEM));
        if (o < 1) fail(AXS_ERR_CUDA, "register-tile z-march kernel <%d,%d> does not fit on an SM", K, NW);
        return o;
    });
}
template <int K, int NW, int VR>
static void launch_k_t(const ZLat *d, int nlat, int64_t items, int *counters, int parity, cudaStream_t st) {
    const int64_t grid = std::min<int64_t>((int64_t)prepare_k_t<K, NW, VR>() * num_sms(), items);
    k_zmarch_k<K, NW, VR><<<(int)grid, 32 * NW, ZKCfg<K, NW, VR>::SMEM, st>>>(d, nlat, items, counters, parity);
    AXS_CUDA(cudaGetLastError());
    count_launches(1);
}

// The kernel of k steps for a tile shape (warps, rows per warp).
template <int NW, int VR, int KMAX>
static bool with_k(int k, bool launch, const ZLat *d, int nlat, int64_t items, int *counters, int parity, cudaStream_t st) {
    if (k < 1 || k > KMAX) return false;
    if constexpr (KMAX > 1)
        if (k < KMAX) return with_k<NW, VR, KMAX - 1>(k, launch, d, nlat, items, counters, parity, st);
    if (launch) launch_k_t<KMAX, NW, VR>(d, nlat, items, counters, parity, st);
    else prepare_k_t<KMAX, NW, VR>();
    return true;
}
static void dispatch_k(int nw, int vr, int k, bool launch, const ZLat *d, int nlat, int64_t items, int *counters, int parity,
                       cudaStream_t st) {
    bool ok = false;
    switch (nw * 10 + vr) {
    case 84: ok = with_k<8, 4, 4>(k, launch, d, nlat, items, counters, parity, st); break;
    case 124: ok = with_k<12, 4, 3>(k, launch, d, nlat, items, counters, parity, st); break;
    case 123: ok = with_k<12, 3, 4>(k, launch, d, nlat, items, counters, parity, st); break;
    }
    if (!ok) fail(AXS_ERR_ARG, "no register-tile kernel with %d x %d rows and %d steps", nw, vr, k);
}
void launch_zmarch_k(int nw, int vr, int k, const ZLat *d, int nlat, int64_t items, int *counters, int parity, cudaStream_t st) {
    dispatch_k(nw, vr, k, true, d, nlat, items, counters, parity, st);
}
void prepare_zmarch_k(int nw, int vr, int kmax) {
    for (int k = 1; k <= kmax; ++k) dispatch_k(nw, vr, k, false, nullptr, 0, 0, nullptr, 0, nullptr);
}

}  // namespace axs
