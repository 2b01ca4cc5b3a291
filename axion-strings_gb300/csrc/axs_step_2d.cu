// 2D leapfrog steps, several per launch (temporal blocking): the 2D form of
// vvsl_field_rescaled (src/standard/s_integrate.cpp:305-348).
//
// A 2D lattice is small: 512^2 fits L2, and one step per launch was bound by
// the launch, the FP64 time coefficients that every thread formed and two
// passes over the state, not by arithmetic. Here a block takes a tile through
// k steps in registers:
//  * it loads psi and pih over the tile plus a k R halo (periodic) once; lane i
//    of a warp holds XS neighbouring sites of V rows, the warps lie above one
//    another, and psi and pih stay in those registers for all k steps;
//  * per step the x neighbours come by shuffles, the y neighbours from the
//    thread's own rows, and only the first and last R rows of each warp go
//    through shared memory (double-buffered: one barrier per step). With psi in
//    a shared tile and every neighbour read from it a step of a row took twice
//    as long (shared-memory wavefronts);
//  * the region that is still right shrinks by R on each side per step (rows
//    past it are skipped, columns past it carry values that nobody reads);
//    after k steps the tile itself is written, psi and pih out of place (other
//    tiles still read the old ones in their halos).
// Each site goes through site_update / site_update_fold with one step's
// coefficients, so k steps in one launch and k launches of one step give the
// same bits.
//
// Measured (GB300, graph of launches, us per step): FP32 radius 1 at 128^2 /
// 512^2 / 1500^2 / 4096^2: 0.48 / 1.03 / 5.0 / 34 with 8 / 6 / 4 / 6 steps
// per launch, against 3.2 / 10 / 23 / 99 with one thread per site and one step per
// launch; FP64 (bound by its FP64 pipe, 9 operations per site and step)
// 1.8 / 7.0 / 44 / 300 against 4 / 16 / 77 / 520 (from 470^2 the march below). A launch costs about 3 us
// before its first step; it was 0.6 us more when every block formed the time
// coefficients (FP64 divisions, one dependent chain): an extra block now forms
// those of the next launch while the others step. Programmatic dependent
// launch gained nothing (the next launch's blocks take slots from this one's).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "axs_internal.h"

namespace axs {

struct Step2dArgs {
    const void *psi;
    void *psi_out;
    const void *pih;
    void *pih_out;
    const double *clock_in;
    double *clock_out;
    const void *tab_in;  // Step2dTable<T>: the coefficients from the clock this launch starts at, if its tag says so
    void *tab_out;       // those from the clock it ends at
    int N, k;            // k steps in this launch
    int ntx, ntiles;     // tiles across, tiles in all
    double dt, inv_dx2, lambda, T0sq3;
    int prs, form;
};
constexpr int kStep2dMaxK = 16;
// The coefficients of the next steps, formed by an extra block of the launch
// before. A table serves a launch only when its tag is the clock and the step
// that launch reads (lambda, T0 and the rest are fixed for a lattice);
// otherwise (a state just set, a resumed run) the launch's blocks form them.
template <typename T>
struct Step2dTable {
    double tau, dt;
    StepCoefs<T> c[kStep2dMaxK];
    T kctr[kStep2dMaxK];
};

// One site's update from its neighbours (x pair and y pair at distances 1..R).
template <typename T, int R>
struct Site2d {
    typedef typename Cplx<T>::type C;
    StepCoefs<T> c;
    T kctr;
    __device__ __forceinline__ void update(C &a, C &p, const C (&xm)[R], const C (&xp)[R], const C (&ym)[R],
                                           const C (&yp)[R]) const {
        if constexpr (sizeof(T) == 4 && R == 1) {
            const float2 s = add2(add2(xm[0], xp[0]), add2(ym[0], yp[0]));
            const float2 L = fma2(make_float2(-4.f, -4.f), a, s);
            const float r = fmaf(a.x, a.x, fmaf(a.y, a.y, c.c0)), g = c.kdt_coef * r;
            p = fma2(make_float2(c.kdt_idx2, c.kdt_idx2), L, fma2(make_float2(g, g), a, p));
            a = fma2(make_float2(c.dt, c.dt), p, a);
        } else if constexpr (R == 1) {
            const T S1 = nsum5<T>(xm[0].x, xp[0].x, ym[0].x, yp[0].x), S2 = nsum5<T>(xm[0].y, xp[0].y, ym[0].y, yp[0].y);
            T an, bn;
            site_update_fold<T>(a.x, a.y, S1, S2, p.x, p.y, an, bn, c, kctr);
            a.x = an;
            a.y = bn;
        } else {
            T a1 = (T)stencil_coef(R - 1, 2, 0) * a.x, a2 = (T)stencil_coef(R - 1, 2, 0) * a.y;
#pragma unroll
            for (int l = 0; l < R; ++l) {
                const T w = (T)stencil_coef(R - 1, 2, l + 1);
                a1 = fma(w, nsum5<T>(xm[l].x, xp[l].x, ym[l].x, yp[l].x), a1);
                a2 = fma(w, nsum5<T>(xm[l].y, xp[l].y, ym[l].y, yp[l].y), a2);
            }
            T an, bn;
            site_update<T>(a.x, a.y, a1, a2, p.x, p.y, an, bn, c);
            a.x = an;
            a.y = bn;
        }
    }
};

__device__ __forceinline__ float2 shfl_c(float2 v, int lane) {
    return make_float2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}
__device__ __forceinline__ double2 shfl_c(double2 v, int lane) {
    return make_double2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}

template <typename T, int XS>
__device__ __forceinline__ void load_sites(const typename Cplx<T>::type *p, typename Cplx<T>::type (&v)[XS]) {
    if constexpr (sizeof(T) == 4 && XS == 2) {
        const float4 q = *reinterpret_cast<const float4 *>(p);
        v[0] = make_float2(q.x, q.y);
        v[1] = make_float2(q.z, q.w);
    } else {
#pragma unroll
        for (int j = 0; j < XS; ++j) v[j] = p[j];
    }
}
template <typename T, int XS>
__device__ __forceinline__ void store_sites(typename Cplx<T>::type *p, const typename Cplx<T>::type (&v)[XS]) {
    if constexpr (sizeof(T) == 4 && XS == 2) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
    } else {
#pragma unroll
        for (int j = 0; j < XS; ++j) p[j] = v[j];
    }
}

// The coefficients n steps from tau (advanced as single steps advance it), and FP64's centre weight.
template <typename T>
__device__ __forceinline__ StepCoefs<T> make_step_coefs(const Step2dArgs &A, double tau, int n, T &kctr) {
    for (int s = 0; s < n; ++s) tau = tau + A.dt;
    const StepCoefs<T> c = make_coefs<T>(tau, A.dt, A.dt, A.inv_dx2, A.lambda, A.T0sq3, A.prs, A.form);
    kctr = sizeof(T) == 8 ? c.kdt_idx2 * (T)-4 : (T)0;
    return c;
}
// Those of step n of this launch, from the table when its tag is this clock and step.
template <typename T>
__device__ __forceinline__ StepCoefs<T> step_coefs(const Step2dArgs &A, int n, T &kctr) {
    const Step2dTable<T> *t = reinterpret_cast<const Step2dTable<T> *>(A.tab_in);
    const double tau = *A.clock_in;
    const bool made = t->tau == tau && t->dt == A.dt;
    const StepCoefs<T> c = t->c[n];
    kctr = t->kctr[n];
    return made ? c : make_step_coefs<T>(A, tau, n, kctr);
}
// The launch's extra block: the next clock and its table.
template <typename T>
__device__ __forceinline__ void next_table(const Step2dArgs &A) {
    const int tid = threadIdx.x;
    if (tid >= kStep2dMaxK) return;
    double tau = *A.clock_in;
    for (int s = 0; s < A.k; ++s) tau = tau + A.dt;
    Step2dTable<T> *t = reinterpret_cast<Step2dTable<T> *>(A.tab_out);
    t->c[tid] = make_step_coefs<T>(A, tau, tid, t->kctr[tid]);
    if (tid == 0) {
        t->tau = tau;
        t->dt = A.dt;
        *A.clock_out = tau;
    }
}

// XS sites per lane, V rows per warp; the block's warps (1 .. 16, at run time)
// lie above one another. R <= V.
template <typename T, int R, int XS, int V>
__global__ void __launch_bounds__(V <= 2 ? 512 : 256) k_step2d(const Step2dArgs A) {
    typedef typename Cplx<T>::type C;
    constexpr int RX = 32 * XS;
    constexpr int E = V < 2 * R ? V : 2 * R;   // rows a warp publishes: its first and last R, or all
    constexpr int LN = (R + XS - 1) / XS;   // lanes to either side that hold x neighbours
    extern __shared__ __align__(16) unsigned char smem[];
    // the first and last R rows of each warp (all, if fewer than 2R), two buffers: [2][warps][E][RX]
    C *edge = reinterpret_cast<C *>(smem);
    __shared__ StepCoefs<T> coefs[kStep2dMaxK];
    __shared__ T kctrs[kStep2dMaxK];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
    const int x = XS * lane, y0 = w * V, RY = V * nw;
    const int N = A.N, k = A.k, H = k * R, HX = (H + XS - 1) / XS * XS;
    const int TX = RX - 2 * HX, TY = RY - 2 * H;
    const C *psi = reinterpret_cast<const C *>(A.psi), *pih = reinterpret_cast<const C *>(A.pih);
    C *po = reinterpret_cast<C *>(A.psi_out), *qo = reinterpret_cast<C *>(A.pih_out);
    if (blockIdx.x == gridDim.x - 1) {
        next_table<T>(A);
        return;
    }
    if (tid < k) {
        T kc;
        coefs[tid] = step_coefs<T>(A, tid, kc);
        if (sizeof(T) == 8) kctrs[tid] = kc;
    }
    for (int tile = blockIdx.x; tile < A.ntiles; tile += gridDim.x - 1) {
        const int ty = tile / A.ntx, gx0 = (tile - ty * A.ntx) * TX, gy0 = ty * TY;
        int gx = (gx0 - HX + x) % N, gy = (gy0 - H + y0) % N;
        if (gx < 0) gx += N;
        if (gy < 0) gy += N;
        C a[V][XS], p[V][XS];
        {
            int yy = gy;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const int o = yy * N + gx;
                load_sites<T, XS>(psi + o, a[v]);
                load_sites<T, XS>(pih + o, p[v]);
                yy = yy + 1 == N ? 0 : yy + 1;
            }
        }
        for (int s = 0; s < k; ++s) {
            C *eb = edge + (s & 1) * nw * E * RX;
            // rows 0 .. R-1 of the warp at 0 .. R-1, rows V-R .. V-1 at the end (E < 2R: row r at r)
#pragma unroll
            for (int e = 0; e < E; ++e) store_sites<T, XS>(eb + (w * E + e) * RX + x, a[e < R ? e : V - E + e]);
            __syncthreads();
            Site2d<T, R> st;
            st.c = coefs[s];
            st.kctr = sizeof(T) == 8 ? kctrs[s] : (T)0;
            const int lo = R * (s + 1), hi = RY - lo;   // rows with all their neighbours
            C up[R][XS], dn[R][XS];   // rows y - 1 .. y - R before this step; rows past the warp's last
            // row y0 - 1 - l is the l-th of the warp above from its end (l < V), of the one above that, ...
#pragma unroll
            for (int l = 0; l < R; ++l) {
                const int wu = max(w - 1 - l / V, 0), wd = min(w + 1 + l / V, nw - 1);
                load_sites<T, XS>(eb + (wu * E + E - 1 - l % V) * RX + x, up[l]);
                load_sites<T, XS>(eb + (wd * E + l % V) * RX + x, dn[l]);
            }
#pragma unroll
            for (int v = 0; v < V; ++v) {
                C old[XS];
#pragma unroll
                for (int j = 0; j < XS; ++j) old[j] = a[v][j];
                const int y = y0 + v;
                if (y >= lo && y < hi) {   // the same in the whole warp
                    C win[XS + 2 * LN * XS];   // sites x - LN XS .. x + XS + LN XS - 1 of the row
#pragma unroll
                    for (int j = 0; j < XS; ++j) win[LN * XS + j] = old[j];
#pragma unroll
                    for (int n = 1; n <= LN; ++n)
#pragma unroll
                        for (int j = 0; j < XS; ++j) {
                            if ((n - 1) * XS + XS - j <= R) win[(LN - n) * XS + j] = shfl_c(old[j], lane - n);
                            if ((n - 1) * XS + j + 1 <= R) win[(LN + n) * XS + j] = shfl_c(old[j], lane + n);
                        }
#pragma unroll
                    for (int j = 0; j < XS; ++j) {
                        C xm[R], xp[R], ym[R], yp[R];
#pragma unroll
                        for (int l = 0; l < R; ++l) {
                            xm[l] = win[LN * XS + j - 1 - l];
                            xp[l] = win[LN * XS + j + 1 + l];
                            ym[l] = up[l][j];
                            yp[l] = v + 1 + l < V ? a[v + 1 + l < V ? v + 1 + l : 0][j] : dn[v + 1 + l < V ? 0 : v + 1 + l - V][j];
                        }
                        st.update(a[v][j], p[v][j], xm, xp, ym, yp);
                    }
                }
#pragma unroll
                for (int l = R - 1; l >= 0; --l)
#pragma unroll
                    for (int j = 0; j < XS; ++j) up[l][j] = l > 0 ? up[l > 0 ? l - 1 : 0][j] : old[j];
            }
        }
        // the tile's sites inside the lattice
        const int ox = gx0 + x - HX;
        if (x >= HX && x < RX - HX && ox < N) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const int y = y0 + v, oy = gy0 + y - H;
                if (y >= H && y < RY - H && oy < N) {
                    store_sites<T, XS>(po + oy * N + ox, a[v]);
                    store_sites<T, XS>(qo + oy * N + ox, p[v]);
                }
            }
        }
        __syncthreads();   // the edge buffers are free for the next tile
    }
}

// One FP64 step of a large lattice: a thread per column of a y-chunk, the y
// neighbours in registers, the x neighbours from L1. FP64 is bound by its pipe,
// so here the tiles' halo columns (2 R k of 32 lanes) cost more than a launch per
// step (kMarch2dSites).
template <int R>
__global__ void __launch_bounds__(128) k_march2d(const Step2dArgs A) {
    typedef double2 C;
    __shared__ StepCoefs<double> sc;
    __shared__ double skctr;
    const int N = A.N, x = blockIdx.x * 128 + threadIdx.x;
    const int chunks = gridDim.y - 1;   // the last row of blocks forms the next launch's coefficients
    if ((int)blockIdx.y == chunks) {
        if (blockIdx.x == 0) next_table<double>(A);
        return;
    }
    if (threadIdx.x == 0) sc = step_coefs<double>(A, 0, skctr);
    const int ya = (int)((int64_t)blockIdx.y * N / chunks), yb = (int)((int64_t)(blockIdx.y + 1) * N / chunks);
    __syncthreads();
    if (x >= N) return;
    Site2d<double, R> st;
    st.c = sc;
    st.kctr = skctr;
    const C *psi = reinterpret_cast<const C *>(A.psi), *pih = reinterpret_cast<const C *>(A.pih);
    C *po = reinterpret_cast<C *>(A.psi_out), *qo = reinterpret_cast<C *>(A.pih_out);
    int xl[R], xr[R];
#pragma unroll
    for (int l = 0; l < R; ++l) {
        xl[l] = x - 1 - l < 0 ? x - 1 - l + N : x - 1 - l;
        xr[l] = x + 1 + l >= N ? x + 1 + l - N : x + 1 + l;
    }
    C yr[2 * R + 1];   // rows y-R .. y+R
#pragma unroll
    for (int d = 0; d < 2 * R; ++d) {
        const int y = ya + d - R;
        yr[d] = psi[(y < 0 ? y + N : (y >= N ? y - N : y)) * N + x];
    }
    for (int y = ya; y < yb; ++y) {
        const int row = y * N;
        yr[2 * R] = psi[(y + R >= N ? y + R - N : y + R) * N + x];
        C p = pih[row + x], a = yr[R], xm[R], xp[R], ym[R], yp[R];
#pragma unroll
        for (int l = 0; l < R; ++l) {
            xm[l] = psi[row + xl[l]];
            xp[l] = psi[row + xr[l]];
            ym[l] = yr[R - 1 - l];
            yp[l] = yr[R + 1 + l];
        }
        st.update(a, p, xm, xp, ym, yp);
        po[row + x] = a;
        qo[row + x] = p;
#pragma unroll
        for (int d = 0; d < 2 * R; ++d) yr[d] = yr[d + 1];
    }
}
// About 16 blocks per SM, in chunks of at least 2 rows (4 from 800^2: 1000^2 takes
// 19.8 us with 4, 20.6 with 2; 512^2 7.4 and 7.0).
template <int R>
static void launch_march2d(const Step2dArgs &a, cudaStream_t st) {
    const int cols = (a.N + 127) / 128;
    const dim3 grid(cols, std::max(1, std::min((16 * num_sms() + cols - 1) / cols, a.N / (a.N < 800 ? 2 : 4))) + 1);
    k_march2d<R><<<grid, 128, 0, st>>>(a);
    AXS_CUDA(cudaGetLastError());
    count_launches(1);
}
// Sites from which FP64 takes it, by radius: us per step of the march and of the
// tiles at radius 1, 426^2 6.5 and 5.9, 512^2 7.0 and 8.3, 1000^2 19.8 and 26,
// 3000^2 158 and 216; radius 2, 256^2 5.5 and 5.4, 340^2 7.1 and 9.1; radius 3, 256^2
// 6.0 and 7.3; radius 4, 126^2 5.5 and 5.9, 64^2 5 and 3.9.
constexpr double kMarch2dSites[4] = {220000.0, 75000.0, 32000.0, 12000.0};

// ---------------------------------------------------------------- dispatch
//
// The shape of a launch (sites per lane, rows per warp, warps, steps) follows
// from an estimate of its time over the shapes below: a launch costs t0; an SM
// takes ceil(tiles / SMs) tiles, in rounds of as many as are resident, a
// round at a load's latency plus a barrier's per step; a tile costs the 32-site
// rows that its shrinking region has over the steps times the cycles of a row
// (a lone block's rows count as its fullest scheduler's, four to the SM); and
// loads and stores go at L2's rate while the state fits half of it (each die's
// share), else HBM's. The
// constants are fitted to 1300 measured launches (N = 64 .. 1500, all radii):
// 5 % rms in FP32, 9 % in FP64, and the shape chosen is within 12 % of the best
// measured one in FP32 and 20 % (one case 32 %) in FP64. More steps per launch
// amortise t0, latency and traffic and cost halo: at 128^2 eight steps per
// launch win in FP32, at 1500^2 four to six; FP64, bound by its pipe, takes one
// to four.
struct Shape2d {
    int xs, v;
    double row;   // SM cycles per 32-site row
};

template <typename T, int R>
static int shapes2d(const Shape2d *&s) {
    static constexpr Shape2d f1[] = {{1, 2, 5.4}, {2, 2, 4.8}, {2, 4, 6.8}, {2, 8, 8.5}};
    static constexpr Shape2d f2[] = {{1, 2, 15.6}, {2, 2, 14.4}, {2, 4, 14.7}, {2, 8, 14.1}};
    static constexpr Shape2d f3[] = {{1, 2, 28.2}, {2, 2, 25.0}, {2, 4, 21.4}};
    static constexpr Shape2d f4[] = {{1, 2, 42.0}, {2, 2, 35.7}, {2, 4, 29.7}};
    static constexpr Shape2d d1[] = {{1, 1, 92.6}, {1, 2, 126.0}, {1, 4, 138.9}};
    static constexpr Shape2d d2[] = {{1, 1, 233.5}, {1, 2, 281.2}};
    static constexpr Shape2d d3[] = {{1, 1, 377.5}, {1, 2, 374.9}};
    static constexpr Shape2d d4[] = {{1, 1, 552.2}, {1, 2, 512.1}};
    if constexpr (sizeof(T) == 4) {
        s = R == 1 ? f1 : R == 2 ? f2 : R == 3 ? f3 : f4;
        return R <= 2 ? 4 : 3;
    } else {
        s = R == 1 ? d1 : R == 2 ? d2 : R == 3 ? d3 : d4;
        return R == 1 ? 3 : 2;
    }
}

// Resident blocks per SM of a shape with nw warps.
template <typename T, int R>
static int resident2d(const Shape2d &s, int nw);

template <typename T, int R>
static Plan2d plan2d_k(int N, int k, int sms) {
    const Shape2d *sh = nullptr;
    const int n = shapes2d<T, R>(sh);
    const bool f32 = sizeof(T) == 4;
    const double t0 = f32 ? 1.8 : 1.9, lat = f32 ? 0.25 : 0.08, step = f32 ? 0.19 : 0.77;   // us
    const double csz = 2.0 * sizeof(T);
    const double bw = 4.0 * N * N * csz < 60e6 ? (f32 ? 15.8e6 : 13.9e6) : 6.5e6;   // bytes per us
    Plan2d best;
    for (int i = 0; i < n; ++i) {
        const int V = sh[i].v, xs = sh[i].xs;
        for (int nw = 4; nw <= (V <= 2 ? 16 : 8); nw += f32 ? 4 : 2) {
            const int rx = 32 * xs, ry = V * nw, h = k * R, hx = (h + xs - 1) / xs * xs;
            const int tx = rx - 2 * hx, ty = ry - 2 * h;
            if (tx < 8 || ty < 2) continue;
            const int ntx = (N + tx - 1) / tx;
            const double tiles = (double)ntx * ((N + ty - 1) / ty), per = tiles / sms;
            // few rows per warp are for lattices of few tiles: with more, their loads are
            // not under other blocks' steps (1500^2 FP32: 5.9 us per step, V = 4 and 8 5.1)
            if (f32 && V == 2 && per > 2.0) continue;
            const int occ = resident2d<T, R>(sh[i], nw);
            double rows = 0.0;
            for (int s = 1; s <= k; ++s) {
                const int a = ry - 2 * R * s;
                int r = a;
                if (per <= 1.0) {
                    const int warps = (a + V - 1) / V + ((R * s) % V && a > V ? 1 : 0);
                    r = std::max(a, 4 * V * ((warps + 3) / 4));
                }
                rows += r;
            }
            const double rounds = per <= 8.0 * occ ? std::ceil(per / occ) : per / occ;
            const double us = t0 + rounds * (lat + step * k) +
                              (per <= 8.0 ? std::ceil(per) : per) * rows * xs * sh[i].row / 1920.0 +
                              tiles * ((double)rx * ry + (double)tx * ty) * 2.0 * csz / bw;
            if (us < best.us) {
                best.xs = xs;
                best.v = V;
                best.nw = nw;
                best.k = k;
                best.ntx = ntx;
                best.ntiles = (int)tiles;
                best.us = us;
            }
        }
    }
    return best;
}

// The plan for at most max_steps steps of a lattice: the steps per launch with
// the least estimated time per step, the launches of an interval evened out.
template <typename T, int R>
static Plan2d plan2d(int N, int max_steps) {
    const int sms = num_sms();
    Plan2d best;
    if (sizeof(T) == 8 && (double)N * N >= kMarch2dSites[R - 1]) return best;   // one step by k_march2d
    for (int k = 1; k <= std::min(12, max_steps); ++k) {
        const Plan2d p = plan2d_k<T, R>(N, k, sms);
        if (p.nw && p.us / k < best.us / best.k) best = p;
    }
    const int launches = (max_steps + best.k - 1) / best.k, k = (max_steps + launches - 1) / launches;
    if (k == best.k) return best;
    const Plan2d p = plan2d_k<T, R>(N, k, sms);
    return p.nw ? p : best;
}

template <typename T, int R, int XS, int V>
static int resident2d_t(int nw) {
    typedef typename Cplx<T>::type C;
    constexpr int E = V < 2 * R ? V : 2 * R;
    constexpr int per_warp = 2 * E * 32 * XS * (int)sizeof(C);
    static PerDevice occ[17];   // the kernel's shared-memory attribute and occupancy belong to the device
    return occ[nw].get([nw] {
        AXS_CUDA(cudaFuncSetAttribute(k_step2d<T, R, XS, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (V <= 2 ? 16 : 8) * per_warp));
        int o = 0;
        AXS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_step2d<T, R, XS, V>, 32 * nw, nw * per_warp));
        return std::max(1, o);
    });
}

template <typename T, int R, int XS, int V>
static void launch2d_t(const Step2dArgs &a, int nw, cudaStream_t st) {
    typedef typename Cplx<T>::type C;
    constexpr int E = V < 2 * R ? V : 2 * R;
    const int smem = nw * 2 * E * 32 * XS * (int)sizeof(C);
    // one more block for the next launch's coefficients
    const int grid = (int)std::min<int64_t>(a.ntiles, (int64_t)resident2d_t<T, R, XS, V>(nw) * num_sms()) + 1;
    k_step2d<T, R, XS, V><<<grid, 32 * nw, smem, st>>>(a);
    AXS_CUDA(cudaGetLastError());
    count_launches(1);
}

// fn<XS, V>() for the shape (xs, v) of shapes2d
template <typename T, int R, class Fn>
static void with_shape2d(int xs, int v, Fn fn) {
    if constexpr (sizeof(T) == 4) {
        if (xs == 1) fn(std::integral_constant<int, 1>(), std::integral_constant<int, 2>());
        else if (v == 2) fn(std::integral_constant<int, 2>(), std::integral_constant<int, 2>());
        else if (v == 4) fn(std::integral_constant<int, 2>(), std::integral_constant<int, 4>());
        else if constexpr (R <= 2) fn(std::integral_constant<int, 2>(), std::integral_constant<int, 8>());
    } else {
        if (v == 1) fn(std::integral_constant<int, 1>(), std::integral_constant<int, 1>());
        else if (v == 2) fn(std::integral_constant<int, 1>(), std::integral_constant<int, 2>());
        else if constexpr (R == 1) fn(std::integral_constant<int, 1>(), std::integral_constant<int, 4>());
    }
}
template <typename T, int R>
static int resident2d(const Shape2d &s, int nw) {
    int o = 1;
    with_shape2d<T, R>(s.xs, s.v, [&](auto xs, auto v) { o = resident2d_t<T, R, xs(), v()>(nw); });
    return o;
}
template <typename T, int R>
static void launch2d(const Step2dArgs &a, const Plan2d &p, cudaStream_t st) {
    if constexpr (sizeof(T) == 8)
        if (p.nw == 0) return launch_march2d<R>(a, st);
    with_shape2d<T, R>(p.xs, p.v, [&](auto xs, auto v) { launch2d_t<T, R, xs(), v()>(a, p.nw, st); });
}

template <typename T, int R>
static int step2d_t(Lattice *L, int max_steps, bool launch) {
    const axs_params &p = L->p;
    auto it = L->plans2d.find(max_steps);
    if (it == L->plans2d.end()) {
        if (L->plans2d.size() >= 64) L->plans2d.clear();
        it = L->plans2d.emplace(max_steps, plan2d<T, R>(p.N, max_steps)).first;
    }
    const Plan2d pl = it->second;
    if (!launch) return pl.k;
    const double dx = p.space_step, T0 = p.T_initial;
    Step2dArgs a;
    a.psi = L->psi[L->cur];
    a.psi_out = L->psi[L->cur ^ 1];
    a.pih = L->pih;
    a.pih_out = L->scratch;
    a.clock_in = L->dclock + L->cur;
    a.clock_out = L->dclock + (L->cur ^ 1);
    a.tab_in = (const char *)L->dstep2d + L->cur * kStep2dSlot;
    a.tab_out = (char *)L->dstep2d + (L->cur ^ 1) * kStep2dSlot;
    a.N = p.N;
    a.k = pl.k;
    a.ntx = pl.ntx;
    a.ntiles = pl.ntiles;
    a.dt = (double)p.time_step;
    a.inv_dx2 = 1.0 / (dx * dx);
    a.lambda = (double)p.lambda;
    a.T0sq3 = (T0 * T0) / 3.0;
    a.prs = p.prs;
    a.form = p.form;
    launch2d<T, R>(a, pl, L->stream);
    return pl.k;
}

static int step2d(Lattice *L, int max_steps, bool launch) {
    static_assert(sizeof(Step2dTable<double>) <= kStep2dSlot, "a slot holds a table");
    const int R = L->p.stencil_setting + 1;
    if (L->esz == 4) {
        switch (R) {
        case 1: return step2d_t<float, 1>(L, max_steps, launch);
        case 2: return step2d_t<float, 2>(L, max_steps, launch);
        case 3: return step2d_t<float, 3>(L, max_steps, launch);
        default: return step2d_t<float, 4>(L, max_steps, launch);
        }
    }
    switch (R) {
    case 1: return step2d_t<double, 1>(L, max_steps, launch);
    case 2: return step2d_t<double, 2>(L, max_steps, launch);
    case 3: return step2d_t<double, 3>(L, max_steps, launch);
    default: return step2d_t<double, 4>(L, max_steps, launch);
    }
}

int step2d_launch(Lattice *L, int max_steps) { return step2d(L, max_steps, true); }
int step2d_steps(Lattice *L, int max_steps) { return step2d(L, max_steps, false); }

}  // namespace axs
