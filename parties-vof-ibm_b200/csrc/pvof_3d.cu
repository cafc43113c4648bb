// CUDA executor of the 3D mode and its entry points (called from the C ABI
// in pvof_api.cu when a context is created with PVOF_GEOM_3D).
//
// Launch shapes: a box of cells is walked row by row, one warp per (j,k)
// row and 32 consecutive i per step, so every field access of a warp is one
// coalesced run along i; grids are capped at a multiple of the SM count and
// stride over the remaining rows.  Reductions write one partial per block
// (a fixed grid of at most NBR blocks) and a one-block scalar kernel adds
// the partials in a fixed order, so every sum is the same from run to run.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <string>
#include <type_traits>
#include <vector>

#include <cuda_runtime.h>

#include "pvof_3d.cuh"
#include "pvof_3d_api.h"

namespace pvof3 {

constexpr int TPB = 256;
constexpr int WPB = TPB / 32;
constexpr int NBR = 148 * 8;        // most blocks of a reduction
constexpr int NBC = 148 * 16;       // most blocks of a cell-wise pass

thread_local std::string g_err3;
const char *last_error() { return g_err3.c_str(); }
static int fail(int code, const std::string &m)
{
    g_err3 = m;
    return code;
}

template <class F>
__global__ void __launch_bounds__(TPB) k3_cells(Range r, const int *gate, F f)
{
    if (gate && *gate == 0) return;
    const int nj = r.j1 - r.j0;
    const long long nrows = (long long)nj * (r.k1 - r.k0);
    const int lane = threadIdx.x & 31;
    for (long long row = (long long)blockIdx.x * WPB + (threadIdx.x >> 5); row < nrows; row += (long long)gridDim.x * WPB) {
        const int j = r.j0 + (int)(row % nj), k = r.k0 + (int)(row / nj);
        for (int i = r.i0 + lane; i < r.i1; i += 32) f(i, j, k);
    }
}

template <int N, bool MAX, class F>
__global__ void __launch_bounds__(TPB) k3_reduce(Range r, const int *gate, double *part, F f)
{
    __shared__ double sh[WPB][N];
    if (gate && *gate == 0) return;
    double acc[N];
#pragma unroll
    for (int q = 0; q < N; q++) acc[q] = 0.0;
    const int nj = r.j1 - r.j0;
    const long long nrows = (long long)nj * (r.k1 - r.k0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long row = (long long)blockIdx.x * WPB + warp; row < nrows; row += (long long)gridDim.x * WPB) {
        const int j = r.j0 + (int)(row % nj), k = r.k0 + (int)(row / nj);
        for (int i = r.i0 + lane; i < r.i1; i += 32) {
            const Vec<N> t = f(i, j, k);
#pragma unroll
            for (int q = 0; q < N; q++) acc[q] = MAX ? fmax(acc[q], t.v[q]) : acc[q] + t.v[q];
        }
    }
#pragma unroll
    for (int q = 0; q < N; q++) {
        double a = acc[q];
        for (int o = 16; o > 0; o >>= 1) {
            const double b = __shfl_down_sync(0xffffffffu, a, o);
            a = MAX ? fmax(a, b) : a + b;
        }
        if (lane == 0) sh[warp][q] = a;
    }
    __syncthreads();
    if (threadIdx.x < N) {
        double a = sh[0][threadIdx.x];
        for (int w = 1; w < WPB; w++) a = MAX ? fmax(a, sh[w][threadIdx.x]) : a + sh[w][threadIdx.x];
        part[(size_t)blockIdx.x * 4 + threadIdx.x] = a;
    }
}

struct Pend {
    int nb[NSLOT], nq[NSLOT], mx[NSLOT];
    unsigned mask;
    int stride;   // partial sums per slot (blocks), times 4 values
};

template <class F>
__global__ void __launch_bounds__(TPB) k3_scalar(const double *part, Pend pd, const int *gate, Sc3 *sc, F f)
{
    __shared__ double sh[TPB];
    if (gate && *gate == 0) return;
    for (int s = 0; s < NSLOT; s++) {
        if (!(pd.mask & (1u << s))) continue;
        for (int q = 0; q < pd.nq[s]; q++) {
            double a = 0.0;
            for (int b = threadIdx.x; b < pd.nb[s]; b += TPB) {
                const double v = part[(size_t)s * pd.stride + (size_t)b * 4 + q];
                a = pd.mx[s] ? fmax(a, v) : a + v;
            }
            sh[threadIdx.x] = a;
            __syncthreads();
            for (int w = TPB / 2; w > 0; w >>= 1) {
                if (threadIdx.x < w) sh[threadIdx.x] = pd.mx[s] ? fmax(sh[threadIdx.x], sh[threadIdx.x + w]) : sh[threadIdx.x] + sh[threadIdx.x + w];
                __syncthreads();
            }
            if (threadIdx.x == 0) sc->sum[s][q] = sh[0];
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) f(sc);
}

// ---------------------------------------------------------------------------
// the pressure PCG iteration (psolve_cg.c:209-253) as three streaming kernels
// over the physical cells: a thread takes two neighbouring cells of a row
// (16-byte loads; i = 0 is 16-byte aligned and every row and plane pitch is
// even) in PKB consecutive planes, a block a 64 x 8 tile of (i, j); PKB
// planes per block keep the end-of-block reduction barrier and the number of
// partial sums small.  Reads at
// ghost and half cells go through the pressure ghost map; the arithmetic is
// that of p_apply_st and of the reference's loops, operand for operand.
// Bound by HBM from about 2 million cells on (256^3: 13 fields, 395 us), below by
// latency and launches.  Three passes: one that forms the direction, applies the
// operator and updates phi together moves nine fields, but its three planes in
// registers leave three blocks per SM, whose last wave is mostly empty just
// above 444 blocks.  Us an iteration, three passes | two: 64^3 24.6 | 27.6, 96^3
// 34.5 | 33.9, 120x97x104 42 | 43, 120^3 57.3 | 72.1, 128^3 66 | 81, 160^3 124 |
// 128, 256x128x64 64 | 79, 256^3 395 | 407.
// ---------------------------------------------------------------------------
constexpr int PKB = 4;   // the momentum passes' too

__device__ __forceinline__ double2 ld2(const double *p) { return *reinterpret_cast<const double2 *>(p); }
__device__ __forceinline__ void st2(double *p, double a, double b) { *reinterpret_cast<double2 *>(p) = make_double2(a, b); }

// the cells (i, i+1) of a pressure field at (j, k), after the ghost update
__device__ __forceinline__ void p_pair(const Dom3 &d, const double *__restrict__ X, int i, int j, int k, double &a,
                                       double &b)
{
    if (j >= 0 && j <= d.NY - 2 && k >= 0 && k <= d.NZ - 2) {
        const double2 v = ld2(X + at(d, i, j, k));
        a = v.x;
        b = v.y;
    } else {
        a = rd<K_PRESSURE>(d, X, i, j, k);
        b = rd<K_PRESSURE>(d, X, i + 1, j, k);
    }
}

// The sums of a block of 256 threads into part[block]; the last block to finish
// adds all the partials in a fixed order (the same whichever block is last) and
// runs the scalar step then(sc, sums...) on one thread, so no separate launch
// is needed between the passes.  The last block's loads go out eight at a time, at
// the last partial again instead of tested beyond it (with a test each the
// pressure iteration took 405 us at 256^3 against 395, 82.5 at 127^3 against 80.3;
// one by one behind the last full eight, the momentum iteration 101.6 at 120^3
// against 98.7).
template <int NV, class F>
__device__ __forceinline__ void block_sum_then(double (&acc)[NV], double *part, Sc3 *sc, F then)
{
    __shared__ double sh[8][NV];
    __shared__ bool last;
    const int t = threadIdx.x + blockDim.x * threadIdx.y, lane = t & 31, warp = t >> 5;
    auto block_sum = [&]() {   // in acc of thread 0
#pragma unroll
        for (int n = 0; n < NV; n++) {
            for (int o = 16; o > 0; o >>= 1) acc[n] += __shfl_down_sync(0xffffffffu, acc[n], o);
            if (lane == 0) sh[warp][n] = acc[n];
        }
        __syncthreads();
        if (t == 0)
#pragma unroll
            for (int n = 0; n < NV; n++)
                for (int q = 1; q < 8; q++) acc[n] += sh[q][n];
    };
    block_sum();
    const unsigned nb = gridDim.x * gridDim.y * gridDim.z;
    if (t == 0) {
        double *p = part + (size_t)(blockIdx.x + gridDim.x * (blockIdx.y + (size_t)gridDim.y * blockIdx.z)) * 4;
#pragma unroll
        for (int n = 0; n < NV; n++) p[n] = acc[n];
        __threadfence();
        last = (atomicAdd(&sc->p_count, 1u) == nb - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int n = 0; n < NV; n++) acc[n] = 0.0;
    for (unsigned b = t; b < nb; b += 8 * 256) {   // beyond the last partial: that one again, not added
        double v[8][NV];
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
            for (int n = 0; n < NV; n++) v[u][n] = __ldcg(part + (size_t)min(b + u * 256, nb - 1) * 4 + n);
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
            for (int n = 0; n < NV; n++) acc[n] += b + u * 256 < nb ? v[u][n] : 0.0;
    }
    __syncthreads();
    block_sum();
    if (t == 0) {
        sc->p_count = 0;
        if constexpr (NV == 1) then(sc, acc[0]);
        else then(sc, acc[0], acc[1]);
    }
}

template <class F>
__global__ void __launch_bounds__(256, 4) k3p_apply(Dom3 d, const double *__restrict__ CX, const double *__restrict__ CY,
                                                    const double *__restrict__ CZ, const double *__restrict__ X,
                                                    double *__restrict__ AD, const int *gate, double *part, Sc3 *sc,
                                                    F then)
{
    if (gate && *gate == 0) return;
    const int ni = d.NX - 1, nj = d.NY - 1, nk = d.NZ - 1;
    const int i = 2 * (blockIdx.x * 32 + threadIdx.x), j = blockIdx.y * 8 + threadIdx.y;
    double acc[1] = {0.0};
    if (i < ni && j < nj) {
        const bool two = i + 1 < ni;
#pragma unroll 1
        for (int kk = 0; kk < PKB; kk++) {
            const int k = blockIdx.z * PKB + kk;
            if (k >= nk) break;
            const long long q = at(d, i, j, k);
            // a row's single last cell goes with the pairs, its second cell (the half
            // cell beyond the row) neither summed nor stored (on a path of its own the
            // rest of the warp waited for it: 127^3 79.7 -> 67.6 us an iteration)
            const double2 c = ld2(X + q);
            const double w0 = (i >= 1) ? X[q - 1] : rd<K_PRESSURE>(d, X, i - 1, j, k);
            const int ie = two ? i + 2 : i + 1;
            const double e1 = (ie <= ni - 1) ? X[q + 2] : rd<K_PRESSURE>(d, X, ie, j, k), e0 = two ? c.y : e1;
            double s0, s1, n0, n1, b0, b1, f0, f1;
            p_pair(d, X, i, j - 1, k, s0, s1);
            p_pair(d, X, i, j + 1, k, n0, n1);
            p_pair(d, X, i, j, k - 1, b0, b1);
            p_pair(d, X, i, j, k + 1, f0, f1);
            const double2 cx = ld2(CX + q), cy = ld2(CY + q), cz = ld2(CZ + q);
            const double2 cym = ld2(CY + q - d.P), czm = ld2(CZ + q - d.S);
            const double cxm = CX[q - 1];
            const double v0 = cx.x * (e0 - c.x) - cxm * (c.x - w0) + cy.x * (n0 - c.x) - cym.x * (c.x - s0) +
                              cz.x * (f0 - c.x) - czm.x * (c.x - b0);
            const double v1 = cx.y * (e1 - c.y) - cx.x * (c.y - c.x) + cy.y * (n1 - c.y) - cym.y * (c.y - s1) +
                              cz.y * (f1 - c.y) - czm.y * (c.y - b1);
            const double ad0 = 1.0 * v0, ad1 = 1.0 * v1;
            acc[0] += c.x * ad0;
            if (two) {
                st2(AD + q, ad0, ad1);
                acc[0] += c.y * ad1;
            } else {
                AD[q] = ad0;
            }
        }
    }
    block_sum_then(acc, part, sc, then);
}

template <class F>
__global__ void __launch_bounds__(256) k3p_update(Dom3 d, double *__restrict__ PHI, double *__restrict__ R,
                                                  const double *__restrict__ DD, const double *__restrict__ AD,
                                                  const double *__restrict__ M, const int *gate, Sc3 *sc,
                                                  double *part, F then)
{
    if (gate && *gate == 0) return;
    const int ni = d.NX - 1, nj = d.NY - 1, nk = d.NZ - 1;
    const int i = 2 * (blockIdx.x * 32 + threadIdx.x), j = blockIdx.y * 8 + threadIdx.y;
    const double alpha = sc->p_alpha;
    double acc[1] = {0.0};
    if (i < ni && j < nj) {
        const bool two = i + 1 < ni;
#pragma unroll
        for (int kk = 0; kk < PKB; kk++) {
            const int k = blockIdx.z * PKB + kk;
            if (k >= nk) break;
            const long long q = at(d, i, j, k);
            if (!two) {
                PHI[q] += alpha * DD[q];
                const double r = R[q] - alpha * AD[q];
                R[q] = r;
                acc[0] += r * (r * M[q]);
                continue;
            }
            const double2 x = ld2(PHI + q), dd = ld2(DD + q), r = ld2(R + q), ad = ld2(AD + q), m = ld2(M + q);
            st2(PHI + q, x.x + alpha * dd.x, x.y + alpha * dd.y);
            const double r0 = r.x - alpha * ad.x, r1 = r.y - alpha * ad.y;
            st2(R + q, r0, r1);
            acc[0] += r0 * (r0 * m.x);
            acc[0] += r1 * (r1 * m.y);
        }
    }
    block_sum_then(acc, part, sc, then);
}

__global__ void __launch_bounds__(256) k3p_dir(Dom3 d, const double *__restrict__ R, const double *__restrict__ M,
                                               double *__restrict__ DD, const int *gate, const Sc3 *sc)
{
    if (gate && *gate == 0) return;
    const int ni = d.NX - 1, nj = d.NY - 1, nk = d.NZ - 1;
    const int i = 2 * (blockIdx.x * 32 + threadIdx.x), j = blockIdx.y * 8 + threadIdx.y;
    if (i >= ni || j >= nj) return;
    const double beta = sc->p_beta;
    const bool two = i + 1 < ni;
#pragma unroll
    for (int kk = 0; kk < PKB; kk++) {
        const int k = blockIdx.z * PKB + kk;
        if (k >= nk) break;
        const long long q = at(d, i, j, k);
        if (!two) {
            DD[q] = R[q] * M[q] + beta * DD[q];
            continue;
        }
        const double2 r = ld2(R + q), m = ld2(M + q), dd = ld2(DD + q);
        st2(DD + q, r.x * m.x + beta * dd.x, r.y * m.y + beta * dd.y);
    }
}

// The momentum PCG's two passes over the faces of component C (one face per
// thread in PKB planes).  First pass: x += alpha d_old of the iteration before,
// the direction d = z + beta d_old, A d and d.Ad; a thread marches its planes with
// the directions of three planes in registers.  KC: the direction's ghost update.
// Second pass: r -= alpha Ad, z = M^-1 r and the sums.  One face a thread leaves
// room for four blocks per SM, where two pressure cells left three.  Bound by HBM
// at 256^3, by latency and launches below.  120x97x104, an iteration: 78 us in
// five launches (the weights already stored) -> 63 us in two.
template <int C, int KC, class F>
__global__ void __launch_bounds__(256, 4) k3v_dir_op(Dom3 d, Range r, double iRe, const double *__restrict__ FT,
                                                  const double *__restrict__ MU, const double *__restrict__ MA,
                                                  const double *__restrict__ MB, const double *__restrict__ Z, double *D0,
                                                  double *D1, double *__restrict__ X, double *__restrict__ AD, const int *gate,
                                                  double *part, Sc3 *sc, F then)
{
    __shared__ double tile[2][8][32];
    if (gate && *gate == 0) return;
    const int i = r.i0 + blockIdx.x * 32 + threadIdx.x, j = r.j0 + blockIdx.y * 8 + threadIdx.y;
    const int done = sc->v_iter;
    const bool first = done == 0;
    const double *__restrict__ DO = (done & 1) ? D1 : D0;
    double *__restrict__ DN = (done & 1) ? D0 : D1;
    const double beta = sc->v_beta, alpha = first ? 0.0 : sc->v_alpha;
    double acc[1] = {0.0};
    // east and west neighbours come from the neighbouring lanes, north and south from
    // the tile in shared memory, and only the tile's edges form a neighbour's
    // direction themselves; the sources and multipliers (y walls) under the ghost
    // rule KC once per thread
    const int tx = threadIdx.x, ty = threadIdx.y;
    const bool live = i < r.i1 && j < r.j1;
    const Map3 &m = d.map[KC];
    const int il = live ? i : r.i0, jl = live ? j : r.j0;
    const int row = jl * d.P, oc = row + il, ow = row + m.x.src[il - 1 + NG], oe = row + m.x.src[il + 1 + NG];
    // the walls' faces of v keep their place under the rule and are no unknowns: zero
    const int js = m.y.src[jl - 1 + NG], jn = m.y.src[jl + 1 + NG], os = js * d.P + il, on = jn * d.P + il;
    const bool hs = js >= r.j0 && js < r.j1, hn = jn >= r.j0 && jn < r.j1;
    const double ms = m.y.mul[jl - 1 + NG], mn = m.y.mul[jl + 1 + NG];
    const bool we = tx == 0, ee = tx == 31 || i + 1 >= r.i1, se = ty == 0, ne = ty == 7 || j + 1 >= r.j1;
    auto dir = [&](long long q) { return first ? Z[q] : Z[q] + beta * DO[q]; };
    const int k0 = r.k0 + blockIdx.z * PKB, k1 = k0 + PKB < r.k1 ? k0 + PKB : r.k1;
    double bk = 0.0, c = 0.0;
    if (live) {
        bk = dir(m.z.src[k0 - 1 + NG] * d.S + oc);
        c = dir(k0 * d.S + oc);
    }
#pragma unroll 1
    for (int k = k0; k < k1; k++) {
        const long long pl = k * d.S, q = pl + oc;
        double f = 0.0, w = 0.0, e = 0.0, s = 0.0, n = 0.0, xo = 0.0;
        if (live) {
            f = dir(m.z.src[k + 1 + NG] * d.S + oc);
            if (we) w = dir(pl + ow);
            if (ee) e = dir(pl + oe);
            if (se && hs) s = ms * dir(pl + os);
            if (ne && hn) n = mn * dir(pl + on);
            if (!first) xo = X[q] + alpha * DO[q];
        }
        tile[k & 1][ty][tx] = c;
        const double wl = __shfl_up_sync(0xffffffffu, c, 1), el = __shfl_down_sync(0xffffffffu, c, 1);
        __syncthreads();
        if (live) {
            if (!we) w = wl;
            if (!ee) e = el;
            if (!se) s = tile[k & 1][ty - 1][tx];
            if (!ne) n = tile[k & 1][ty + 1][tx];
            const double ad = vel_op_w<C>(d, iRe, FT, MU, MA, MB, i, j, k, [&](int a, int b, int g) {
                return a > i ? e : (a < i ? w : (b > j ? n : (b < j ? s : (g > k ? f : (g < k ? bk : c)))));
            });
            if (!first) X[q] = xo;
            DN[q] = c;
            AD[q] = ad;
            acc[0] += c * ad;
            bk = c;
            c = f;
        }
    }
    block_sum_then(acc, part, sc, then);
}

template <class F>
__global__ void __launch_bounds__(256) k3v_resid(Dom3 d, Range r, double *__restrict__ R, const double *__restrict__ AD,
                                                 const double *__restrict__ DG, double *__restrict__ Z, const int *gate, Sc3 *sc,
                                                 double *part, F then)
{
    if (gate && *gate == 0) return;
    const int i = r.i0 + blockIdx.x * 32 + threadIdx.x, j = r.j0 + blockIdx.y * 8 + threadIdx.y;
    const double alpha = sc->v_alpha, eps = sc->v_eps;
    double acc[2] = {0.0, 0.0};
    if (i < r.i1 && j < r.j1) {
#pragma unroll
        for (int kk = 0; kk < PKB; kk++) {
            const int k = r.k0 + blockIdx.z * PKB + kk;
            if (k >= r.k1) break;
            const long long q = at(d, i, j, k);
            const double rv = R[q] - alpha * AD[q], dg = DG[q] + eps;
            R[q] = rv;
            Z[q] = rv / dg;
            acc[0] += rv * rv / dg;
            acc[1] += rv * rv;
        }
    }
    block_sum_then(acc, part, sc, then);
}

// ---------------------------------------------------------------------------
// spectral preconditioner of the 3D pressure PCG (pressure_preconditioner = 1):
// z = s (-L)^-1 (s r), s = sqrt of the Jacobi weights, L the 7-point operator at
// density one with the reference's ghost rules (x, z periodic, mirror walls in
// y).  A real transform along x (N cells) and a complex one along z (K cells)
// diagonalise L into one tridiagonal system in y per (kx, kz), solved by the
// Thomas algorithm from host tables; the constant mode (the operator's null
// space) gets eigenvalue 1 in units of 1/dy^2.  Spectrum layout: element
// (kx, j, kz) at ((kz * ny + j) * H + kx), H = N/2 + 1.
//
// The transforms (power-of-two lengths) keep 8 points of a transform per thread
// in registers: Stockham passes of radix 8, with a last one of 4 or 2 where the
// length is no power of 8, exchanged through shared memory between passes only
// (the first pass takes its inputs from global memory, the last leaves its
// outputs in registers at the same indices).  Bound by HBM (a pass reads and
// writes the spectrum or the box once).  256^3, B200: forward x 275 -> 66 us,
// z 202 -> 53, inverse x 327 -> 96 (radix-2 stages two at a time in shared memory
// before, with a square root per point and direction).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
template <bool INV>
__device__ __forceinline__ double2 crot(double2 a)   // times -i (forward) or i (inverse)
{
    return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ void dft4(double2 &a, double2 &b, double2 &c, double2 &d)   // in natural order, in place
{
    const double2 s = cadd(a, c), t = csub(a, c), u = cadd(b, d), v = crot<INV>(csub(b, d));
    a = cadd(s, u);
    b = cadd(t, v);
    c = csub(s, u);
    d = csub(t, v);
}

template <bool INV>
__device__ __forceinline__ void dft8(double2 (&v)[8])
{
    const double h = 0.70710678118654752440;
    dft4<INV>(v[0], v[2], v[4], v[6]);
    dft4<INV>(v[1], v[3], v[5], v[7]);
    // odd part times exp(-+ 2 pi i k / 8)
    const double2 o1 = INV ? make_double2(h * (v[3].x - v[3].y), h * (v[3].x + v[3].y))
                           : make_double2(h * (v[3].x + v[3].y), h * (v[3].y - v[3].x));
    const double2 o2 = crot<INV>(v[5]);
    const double2 o3 = INV ? make_double2(-h * (v[7].x + v[7].y), h * (v[7].x - v[7].y))
                           : make_double2(h * (v[7].y - v[7].x), -h * (v[7].x + v[7].y));
    const double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = cadd(e0, o0);
    v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1);
    v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2);
    v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3);
    v[7] = csub(e3, o3);
}

// The transform of 2^LOGN points by N / 8 threads: thread b holds points
// b + (N / 8) k in v[k], before and after.  put / get: a point's place in
// shared memory; sync: all threads of the transform.  tw: exp(-2 pi i k / N).
template <int LOGN, bool INV, class Put, class Get, class Sync>
__device__ __forceinline__ void fft_regs(double2 (&v)[8], int b, const double2 *__restrict__ tw, Put put, Get get, Sync sync)
{
    constexpr int N = 1 << LOGN, T = N / 8, P8 = LOGN / 3;
    int s = 1;
#pragma unroll
    for (int f = 0; f < P8; f++, s *= 8) {
        dft8<INV>(v);
        if (3 * (f + 1) == LOGN) return;   // the last pass: no twiddles, outputs in place
        const int p = b / s, q = b - p * s;
        double2 w1 = __ldg(tw + p * s), w2 = __ldg(tw + 2 * p * s), w4 = __ldg(tw + 4 * p * s);
        if (INV) {
            w1.y = -w1.y;
            w2.y = -w2.y;
            w4.y = -w4.y;
        }
        const double2 w3 = cmul(w1, w2);
        v[1] = cmul(v[1], w1);
        v[2] = cmul(v[2], w2);
        v[3] = cmul(v[3], w3);
        v[4] = cmul(v[4], w4);
        v[5] = cmul(v[5], cmul(w4, w1));
        v[6] = cmul(v[6], cmul(w4, w2));
        v[7] = cmul(v[7], cmul(w4, w3));
        sync();   // the previous exchange has been read
#pragma unroll
        for (int k = 0; k < 8; k++) put(q + s * (8 * p + k), v[k]);
        sync();
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = get(b + T * k);
    }
    if constexpr (LOGN % 3 == 2) {
        dft4<INV>(v[0], v[2], v[4], v[6]);
        dft4<INV>(v[1], v[3], v[5], v[7]);
    } else if constexpr (LOGN % 3 == 1) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const double2 x = v[u], y = v[u + 4];
            v[u] = cadd(x, y);
            v[u + 4] = csub(x, y);
        }
    }
}

struct SpecDims {
    int N, logN, K, logK, ny, H;
    int g_x;         // x transforms: pairs of rows per block
    int ch_z;        // z transforms: columns per block
};
constexpr int XT = 256;   // threads per block of the x transforms

// t = s r along two x rows at once (one as the real part, the other as the
// imaginary part of a complex row), forward transform, then the two half
// spectra separated, X_a = (Z_k + conj Z_(N-k)) / 2 and
// X_b = (Z_k - conj Z_(N-k)) / 2i, and stored
template <int LOGN>
__global__ void __launch_bounds__(XT, 2) k3s_fwd_x(Dom3 d, SpecDims sd, const double *__restrict__ R,
                                                   const double *__restrict__ SM, double2 *__restrict__ SP,
                                                   const double2 *__restrict__ TW, const int *gate)
{
    constexpr int N = 1 << LOGN, T = N / 8, G = XT / T, H = N / 2 + 1;
    __shared__ double2 sm[G * (N + N / 8)];
    if (gate && *gate == 0) return;
    const int g = threadIdx.x / T, b = threadIdx.x % T;
    double2 *a = sm + g * (N + N / 8);
    const long long rows = (long long)sd.K * sd.ny;
    const long long ra = 2 * ((long long)blockIdx.x * G + g), rb = ra + 1;   // row = k * ny + j
    const bool la = ra < rows, lb = rb < rows;
    const long long qa = la ? at(d, b, (int)(ra % sd.ny), (int)(ra / sd.ny)) : 0;
    const long long qb = lb ? at(d, b, (int)(rb % sd.ny), (int)(rb / sd.ny)) : 0;
    double2 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++)
        v[k] = make_double2(la ? SM[qa + T * k] * R[qa + T * k] : 0.0, lb ? SM[qb + T * k] * R[qb + T * k] : 0.0);
    auto sync = [] { if (T <= 32) __syncwarp(); else __syncthreads(); };
    auto put = [&](int i, double2 x) { a[i + (i >> 3)] = x; };
    auto get = [&](int i) { return a[i + (i >> 3)]; };
    fft_regs<LOGN, false>(v, b, TW, put, get, sync);
    sync();
#pragma unroll
    for (int k = 0; k < 8; k++) put(b + T * k, v[k]);
    sync();
#pragma unroll
    for (int k = 0; k <= 4; k++) {
        const int kx = b + T * k;
        if (kx >= H) break;
        const double2 zk = get(kx), zn = get((N - kx) & (N - 1));
        if (la) SP[ra * H + kx] = make_double2(0.5 * (zk.x + zn.x), 0.5 * (zk.y - zn.y));
        if (lb) SP[rb * H + kx] = make_double2(0.5 * (zk.y + zn.y), -0.5 * (zk.x - zn.x));
    }
}

// complex transform along z of ch_z neighbouring kx columns at one j;
// neighbouring threads take neighbouring columns
template <int LOGK, bool INV>
__global__ void __launch_bounds__(256) k3s_z(SpecDims sd, double2 *__restrict__ SP, const double2 *__restrict__ TW, const int *gate)
{
    constexpr int K = 1 << LOGK, T = K / 8, CH = 256 / T < 32 ? 256 / T : 32;
    __shared__ double2 sm[K * CH];
    if (gate && *gate == 0) return;
    const int nchunk = (sd.H + CH - 1) / CH;
    const int j = blockIdx.x / nchunk, c = threadIdx.x % CH, kx = (blockIdx.x % nchunk) * CH + c, b = threadIdx.x / CH;
    const bool live = kx < sd.H;
    const long long step = (long long)sd.ny * sd.H;
    double2 *p = SP + (long long)b * step + (long long)j * sd.H + (live ? kx : 0);
    double2 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = live ? p[(long long)(T * k) * step] : make_double2(0.0, 0.0);
    fft_regs<LOGK, INV>(v, b, TW, [&](int i, double2 x) { sm[i * CH + c] = x; }, [&](int i) { return sm[i * CH + c]; },
                        [] { __syncthreads(); });
    if (live)
#pragma unroll
        for (int k = 0; k < 8; k++) p[(long long)(T * k) * step] = v[k];
}

// one tridiagonal system in y per (kx, kz): (m_j)^-1 from the host table (the
// upper coefficient of the eliminated rows is its negative); the right-hand
// side scaled by dy^2 / (N K) (the transforms' norm).  Both sweeps, and the
// constant mode's, in runs of TU rows: a run's loads are all issued before its
// dependent chain of updates.  Bound by HBM: the spectrum is read and written by
// each sweep (256^3 146 us).
__global__ void __launch_bounds__(32) k3s_tri(SpecDims sd, double2 *__restrict__ SP, const double *__restrict__ IM, double scale,
                                               const int *gate)
{
    if (gate && *gate == 0) return;
    const long long sys = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (sys >= (long long)sd.K * sd.H) return;
    const int kz = (int)(sys / sd.H), kx = (int)(sys % sd.H);
    const int ny = sd.ny;
    constexpr int TU = 8;
    auto idx = [&](int j) { return ((long long)kz * ny + j) * sd.H + kx; };
    auto load = [&](double2 (&v)[TU], int j0) {
#pragma unroll
        for (int u = 0; u < TU; u++)
            if (j0 + u < ny) v[u] = SP[idx(j0 + u)];
    };
    auto store = [&](const double2 (&v)[TU], int j0) {
#pragma unroll
        for (int u = 0; u < TU; u++)
            if (j0 + u < ny) SP[idx(j0 + u)] = v[u];
    };
    if (kx == 0 && kz == 0) {
        // the constant mode: the mean-free part by the recurrence of rows
        // 0..ny-2 from u_0 = 0, its mean removed, plus the mean itself
        double2 v[TU], mean = make_double2(0.0, 0.0);
        for (int j0 = 0; j0 < ny; j0 += TU) {
            load(v, j0);
#pragma unroll
            for (int u = 0; u < TU; u++)
                if (j0 + u < ny) mean = cadd(mean, v[u]);
        }
        mean.x *= scale / ny;
        mean.y *= scale / ny;
        double2 um = make_double2(0.0, 0.0), uc = make_double2(0.0, 0.0), su = make_double2(0.0, 0.0);
        for (int j0 = 0; j0 < ny; j0 += TU) {
            load(v, j0);
#pragma unroll
            for (int u = 0; u < TU; u++)
                if (j0 + u < ny) {
                    const double2 dd = make_double2(v[u].x * scale - mean.x, v[u].y * scale - mean.y);
                    const double2 un = j0 + u == 0 ? csub(uc, dd)
                                                   : make_double2(2.0 * uc.x - um.x - dd.x, 2.0 * uc.y - um.y - dd.y);
                    su = cadd(su, uc);
                    v[u] = uc;
                    um = uc;
                    uc = un;
                }
            store(v, j0);
        }
        su.x /= ny;
        su.y /= ny;
        for (int j0 = 0; j0 < ny; j0 += TU) {
            load(v, j0);
#pragma unroll
            for (int u = 0; u < TU; u++)
                if (j0 + u < ny) v[u] = make_double2(v[u].x - su.x + mean.x, v[u].y - su.y + mean.y);
            store(v, j0);
        }
        return;
    }
    double2 dp = make_double2(0.0, 0.0);
    for (int j0 = 0; j0 < ny; j0 += TU) {
        double2 v[TU];
        double m[TU];
        load(v, j0);
#pragma unroll
        for (int u = 0; u < TU; u++)
            if (j0 + u < ny) m[u] = IM[idx(j0 + u)];
#pragma unroll
        for (int u = 0; u < TU; u++)
            if (j0 + u < ny) {
                dp = make_double2((v[u].x * scale + dp.x) * m[u], (v[u].y * scale + dp.y) * m[u]);
                v[u] = dp;
            }
        store(v, j0);
    }
    double2 x = dp;   // u_{ny-1}
    for (int j1 = ny - 2; j1 >= 0; j1 -= TU) {
        double2 v[TU];
        double m[TU];
#pragma unroll
        for (int u = 0; u < TU; u++)
            if (j1 - u >= 0) {
                v[u] = SP[idx(j1 - u)];
                m[u] = IM[idx(j1 - u)];
            }
#pragma unroll
        for (int u = 0; u < TU; u++)
            if (j1 - u >= 0) {
                x = make_double2(v[u].x + m[u] * x.x, v[u].y + m[u] * x.y);
                v[u] = x;
            }
#pragma unroll
        for (int u = 0; u < TU; u++)
            if (j1 - u >= 0) SP[idx(j1 - u)] = v[u];
    }
}

// inverse transform along x of two rows at once (the complex row X_a + i X_b,
// each spectrum extended by its Hermitian symmetry; row a comes back as the
// real part, row b as the imaginary part), z = s u, and r.z
template <int LOGN, class F>
__global__ void __launch_bounds__(XT, 2) k3s_inv_x(Dom3 d, SpecDims sd, const double2 *__restrict__ SP,
                                                   const double *__restrict__ SM, const double *__restrict__ R,
                                                   double *__restrict__ Z, const double2 *__restrict__ TW,
                                                   const int *gate, double *part, Sc3 *sc, F then)
{
    constexpr int N = 1 << LOGN, T = N / 8, G = XT / T, H = N / 2 + 1;
    __shared__ double2 sm[G * (N + N / 8)];
    if (gate && *gate == 0) return;
    const int g = threadIdx.x / T, b = threadIdx.x % T;
    double2 *a = sm + g * (N + N / 8);
    const long long rows = (long long)sd.K * sd.ny;
    const long long ra = 2 * ((long long)blockIdx.x * G + g), rb = ra + 1;
    const bool la = ra < rows, lb = rb < rows;
    double2 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int kx = b + T * k;
        const bool lo = kx < H;
        const int c = lo ? kx : N - kx;
        double2 xa = la ? SP[ra * H + c] : make_double2(0.0, 0.0), xb = lb ? SP[rb * H + c] : make_double2(0.0, 0.0);
        if (!lo) {
            xa.y = -xa.y;
            xb.y = -xb.y;
        }
        v[k] = make_double2(xa.x - xb.y, xa.y + xb.x);
    }
    auto sync = [] { if (T <= 32) __syncwarp(); else __syncthreads(); };
    fft_regs<LOGN, true>(v, b, TW, [&](int i, double2 x) { a[i + (i >> 3)] = x; }, [&](int i) { return a[i + (i >> 3)]; }, sync);
    const long long qa = la ? at(d, b, (int)(ra % sd.ny), (int)(ra / sd.ny)) : 0;
    const long long qb = lb ? at(d, b, (int)(rb % sd.ny), (int)(rb / sd.ny)) : 0;
    double acc[1] = {0.0};
#pragma unroll
    for (int k = 0; k < 8; k++) {
        if (la) {
            const double z = SM[qa + T * k] * v[k].x;
            acc[0] += R[qa + T * k] * z;
            Z[qa + T * k] = z;
        }
        if (lb) {
            const double z = SM[qb + T * k] * v[k].y;
            acc[0] += R[qb + T * k] * z;
            Z[qb + T * k] = z;
        }
    }
    block_sum_then(acc, part, sc, then);
}

// d = z + beta d (the spectral form's direction)
__global__ void __launch_bounds__(256) k3p_dir_z(Dom3 d, const double *__restrict__ Z, double *__restrict__ DD,
                                                 const int *gate, const Sc3 *sc)
{
    if (gate && *gate == 0) return;
    const int ni = d.NX - 1, nj = d.NY - 1, nk = d.NZ - 1;
    const int i = 2 * (blockIdx.x * 32 + threadIdx.x), j = blockIdx.y * 8 + threadIdx.y;
    if (i >= ni || j >= nj) return;
    const double beta = sc->p_beta;
    const bool two = i + 1 < ni;
    for (int kk = 0; kk < PKB; kk++) {
        const int k = blockIdx.z * PKB + kk;
        if (k >= nk) break;
        const long long q = at(d, i, j, k);
        if (!two) {
            DD[q] = Z[q] + beta * DD[q];
            continue;
        }
        const double2 z = ld2(Z + q), dd = ld2(DD + q);
        st2(DD + q, z.x + beta * dd.x, z.y + beta * dd.y);
    }
}

// host block (reference layout) <-> padded field
__global__ void k3_unpack(Dom3 d, double *fld, const double *blk, int ng)
{
    const int nx = ng ? d.NX : d.NX + 2 * NG, ny = ng ? d.NY : d.NY + 2 * NG, nz = ng ? d.NZ : d.NZ + 2 * NG;
    const int o = ng ? 0 : NG;
    const long long n = (long long)nx * ny * nz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % nx), j = (int)((t / nx) % ny), k = (int)(t / ((long long)nx * ny));
        fld[at(d, i - o, j - o, k - o)] = blk[t];
    }
}

// the reference's array after its ghost update, into the host block layout;
// xf: 0 the field, 1 C_G, 2 rho, 3 mu of C_L
template <int K>
__global__ void k3_pack(Dom3 d, Phase ph, const double *fld, double *blk, int ng, int xf)
{
    const int nx = ng ? d.NX : d.NX + 2 * NG, ny = ng ? d.NY : d.NY + 2 * NG, nz = ng ? d.NZ : d.NZ + 2 * NG;
    const int o = ng ? 0 : NG;
    const long long n = (long long)nx * ny * nz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % nx) - o, j = (int)((t / nx) % ny) - o, k = (int)(t / ((long long)nx * ny)) - o;
        double v = ng ? fld[at(d, i, j, k)] : rd<K>(d, fld, i, j, k);
        if (xf == 1) v = ph.cg(v);
        else if (xf == 2) v = ph.rho(v);
        else if (xf == 3) v = ph.mu(v);
        // rho and mu are computed on the G range only: the positions their
        // ghost update leaves alone keep the zeros of the allocation
        if (xf >= 2 && !written<K>(d, i, j, k)) v = 0.0;
        blk[t] = v;
    }
}

__global__ void k3_flush(double *buf, size_t n, double v)
{
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) buf[t] = v;
}

struct GpuExec {
    cudaStream_t stream = nullptr;
    Sc3 *sc = nullptr;         // device scalars
    Sc3 *sc_host = nullptr;    // pinned mirror
    int *int_host = nullptr;   // pinned word
    double *part = nullptr;    // NSLOT x pstride partial sums
    size_t pstride = 0;        // doubles per slot: 4 per block of the largest reduction grid
    Pend pend{};
    long long launches = 0;
    cudaError_t err = cudaSuccess;
    size_t field_elems = 0;    // doubles per padded field
    long long origin = 0;      // offset of element (0,0,0) in a field
    // per-solver device time (pvof_set_solver_timing): events around each solve
    int timing = 0;
    cudaEvent_t tev[2] = {nullptr, nullptr};
    double sol_ms[3] = {0.0, 0.0, 0.0};

    void tic()
    {
        if (timing) cudaEventRecord(tev[0], stream);
    }
    void toc(int solver)
    {
        if (!timing) return;
        float t = 0.f;
        if (cudaEventRecord(tev[1], stream) == cudaSuccess && cudaEventSynchronize(tev[1]) == cudaSuccess &&
            cudaEventElapsedTime(&t, tev[0], tev[1]) == cudaSuccess)
            sol_ms[solver] += t;
    }

    void note()
    {
        launches++;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess && err == cudaSuccess) err = e;
    }
    static int blocks(const Range &r, int cap)
    {
        const long long nrows = (long long)(r.j1 - r.j0) * (r.k1 - r.k0);
        long long b = (nrows + WPB - 1) / WPB;
        if (b < 1) b = 1;
        if (b > cap) b = cap;
        return (int)b;
    }
    static bool empty(const Range &r) { return r.i1 <= r.i0 || r.j1 <= r.j0 || r.k1 <= r.k0; }

    template <class F>
    void cells(const Range &r, const int *gate, F f)
    {
        if (empty(r)) return;
        k3_cells<<<blocks(r, NBC), TPB, 0, stream>>>(r, gate, f);
        note();
    }
    template <int N, bool MAX = false, class F>
    void reduce(const Range &r, const int *gate, int slot, F f)
    {
        const int nb = blocks(r, NBR);
        k3_reduce<N, MAX><<<nb, TPB, 0, stream>>>(r, gate, part + (size_t)slot * pstride, f);
        note();
        pend.nb[slot] = empty(r) ? 0 : nb;
        pend.nq[slot] = N;
        pend.mx[slot] = MAX ? 1 : 0;
        pend.mask |= 1u << slot;
    }
    template <class F>
    void scalar(const int *gate, F f)
    {
        pend.stride = pstride;
        k3_scalar<<<1, TPB, 0, stream>>>(part, pend, gate, sc, f);
        note();
        pend.mask = 0;
    }
    // the pressure PCG iteration's three passes (k3p_*)
    static dim3 pgrid(const Dom3 &d)
    {
        return dim3((unsigned)((d.NX - 1 + 63) / 64), (unsigned)((d.NY - 1 + 7) / 8), (unsigned)((d.NZ - 1 + PKB - 1) / PKB));
    }
    // the momentum PCG's (k3v_*)
    static dim3 vgrid(const Range &r)
    {
        return dim3((unsigned)((r.i1 - r.i0 + 31) / 32), (unsigned)((r.j1 - r.j0 + 7) / 8), (unsigned)((r.k1 - r.k0 + PKB - 1) / PKB));
    }
    // the partials of these passes use the last slot, which the generic
    // reductions of the solves do not touch
    double *last_slot() { return part + (size_t)(NSLOT - 1) * pstride; }
    template <class F>
    void p_apply(const Dom3 &d, const double *CX, const double *CY, const double *CZ, const double *X, double *AD,
                 const int *gate, F then)
    {
        k3p_apply<<<pgrid(d), dim3(32, 8), 0, stream>>>(d, CX, CY, CZ, X, AD, gate, last_slot(), sc, then);
        note();
    }
    template <class F>
    void p_update(const Dom3 &d, double *PHI, double *R, const double *DD, const double *AD, const double *M,
                  const int *gate, F then)
    {
        k3p_update<<<pgrid(d), dim3(32, 8), 0, stream>>>(d, PHI, R, DD, AD, M, gate, sc, last_slot(), then);
        note();
    }
    void p_dir(const Dom3 &d, const double *R, const double *M, double *DD, const int *gate)
    {
        k3p_dir<<<pgrid(d), dim3(32, 8), 0, stream>>>(d, R, M, DD, gate, sc);
        note();
    }
    void p_dir_z(const Dom3 &d, const double *Z, double *DD, const int *gate)
    {
        k3p_dir_z<<<pgrid(d), dim3(32, 8), 0, stream>>>(d, Z, DD, gate, sc);
        note();
    }
    template <int C, int KC, class F>
    void v_dir_op(const Dom3 &d, const Range &r, double iRe, const double *FT, const double *MU, const double *MA, const double *MB,
                  const double *Z, double *D0, double *D1, double *X, double *AD, const int *gate, F then)
    {
        k3v_dir_op<C, KC><<<vgrid(r), dim3(32, 8), 0, stream>>>(d, r, iRe, FT, MU, MA, MB, Z, D0, D1, X, AD, gate, last_slot(), sc,
                                                               then);
        note();
    }
    template <class F>
    void v_resid(const Dom3 &d, const Range &r, double *R, const double *AD, const double *DG, double *Z, const int *gate, F then)
    {
        k3v_resid<<<vgrid(r), dim3(32, 8), 0, stream>>>(d, r, R, AD, DG, Z, gate, sc, last_slot(), then);
        note();
    }
    // spectral preconditioner: spectrum, tridiagonal tables, launch shapes
    double2 *spec = nullptr;
    double *tri_im = nullptr;
    SpecDims sd{};
    double spec_scale = 0.0;
    double2 *tw_x = nullptr, *tw_z = nullptr;   // exp(-2 pi i q / n), q < n
    // z = s (-L)^-1 (s r) over the physical cells (the k3s_* kernels), then
    // r.z and the scalar step then(sc, r.z) in the last block
    // x transforms: one pair of rows per nt_x threads, g_x pairs per block
    static long long spec_xblocks(const SpecDims &sd)
    {
        return (((long long)sd.K * sd.ny + 1) / 2 + sd.g_x - 1) / sd.g_x;
    }
    template <int LOGN>
    void launch_fwd_x(unsigned grid, const Dom3 &d, const double *R, const double *SM, const int *gate)
    {
        k3s_fwd_x<LOGN><<<grid, XT, 0, stream>>>(d, sd, R, SM, spec, tw_x, gate);
        note();
    }
    template <int LOGN, class F>
    void launch_inv_x(unsigned grid, const Dom3 &d, const double *R, const double *SM, double *Z, const int *gate, F then)
    {
        k3s_inv_x<LOGN><<<grid, XT, 0, stream>>>(d, sd, spec, SM, R, Z, tw_x, gate, last_slot(), sc, then);
        note();
    }
    template <int LOGK>
    void launch_z(bool inverse, const int *gate)
    {
        constexpr int T = (1 << LOGK) / 8;
        const unsigned grid = (unsigned)(sd.ny * ((sd.H + sd.ch_z - 1) / sd.ch_z));
        if (inverse) k3s_z<LOGK, true><<<grid, T * sd.ch_z, 0, stream>>>(sd, spec, tw_z, gate);
        else k3s_z<LOGK, false><<<grid, T * sd.ch_z, 0, stream>>>(sd, spec, tw_z, gate);
        note();
    }
    // f with the transform length 2^log as a compile-time constant (3 .. 10)
    template <class F>
    static void with_log(int log, F f)
    {
        switch (log) {
        case 3: f(std::integral_constant<int, 3>()); break;
        case 4: f(std::integral_constant<int, 4>()); break;
        case 5: f(std::integral_constant<int, 5>()); break;
        case 6: f(std::integral_constant<int, 6>()); break;
        case 7: f(std::integral_constant<int, 7>()); break;
        case 8: f(std::integral_constant<int, 8>()); break;
        case 9: f(std::integral_constant<int, 9>()); break;
        default: f(std::integral_constant<int, 10>()); break;
        }
    }
    template <class F>
    void spec_apply(const Dom3 &d, const double *R, const double *SM, double *Z, const int *gate, F then)
    {
        const unsigned gx = (unsigned)spec_xblocks(sd);
        // one thread per system, a few thousand systems: blocks of 32 spread them over every SM
        const unsigned gt = (unsigned)(((long long)sd.K * sd.H + 31) / 32);
        with_log(sd.logN, [&](auto L) { launch_fwd_x<decltype(L)::value>(gx, d, R, SM, gate); });
        with_log(sd.logK, [&](auto L) { launch_z<decltype(L)::value>(false, gate); });
        k3s_tri<<<gt, 32, 0, stream>>>(sd, spec, tri_im, spec_scale, gate);
        note();
        with_log(sd.logK, [&](auto L) { launch_z<decltype(L)::value>(true, gate); });
        with_log(sd.logN, [&](auto L) { launch_inv_x<decltype(L)::value>(gx, d, R, SM, Z, gate, then); });
    }
    int read_int(const int *p)
    {
        if (cudaMemcpyAsync(int_host, p, sizeof(int), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
            cudaStreamSynchronize(stream) != cudaSuccess) {
            if (err == cudaSuccess) err = cudaGetLastError();
            return 0;
        }
        return *int_host;
    }
    double read_double(const double *p)
    {
        Sc3 s = read_scalars();
        const char *base = reinterpret_cast<const char *>(sc);
        return *reinterpret_cast<const double *>(reinterpret_cast<const char *>(&s) + (reinterpret_cast<const char *>(p) - base));
    }
    Sc3 read_scalars()
    {
        if (cudaMemcpyAsync(sc_host, sc, sizeof(Sc3), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
            cudaStreamSynchronize(stream) != cudaSuccess) {
            if (err == cudaSuccess) err = cudaGetLastError();
        }
        return *sc_host;
    }
    void zero(double *fld)
    {
        const cudaError_t e = cudaMemsetAsync(fld - origin, 0, field_elems * sizeof(double), stream);
        if (e != cudaSuccess && err == cudaSuccess) err = e;
    }
    int status()
    {
        if (err != cudaSuccess) return fail(PVOF_ECUDA, std::string("CUDA: ") + cudaGetErrorString(err));
        return PVOF_OK;
    }
};

struct Handle {
    Box3<GpuExec> b;
    int device = 0;
    double *mem = nullptr;      // all fields
    double *tables = nullptr;   // metrics, weights, maps (doubles)
    int *itables = nullptr;     // map sources
    double *stage = nullptr;    // staging block for host copies
    size_t stage_elems = 0;
    double *flush = nullptr;
    size_t flush_elems = 0;
    cudaEvent_t ev[2] = {nullptr, nullptr};
};

static size_t block_elems(const Dom3 &d, bool ng)
{
    return ng ? (size_t)d.NX * d.NY * d.NZ : (size_t)(d.NX + 2 * NG) * (d.NY + 2 * NG) * (d.NZ + 2 * NG);
}

#define CK3(call)                                                                              \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess) return fail(PVOF_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

int destroy(Handle *h)
{
    if (!h) return PVOF_OK;
    cudaSetDevice(h->device);
    GpuExec &x = h->b.x;
    if (x.stream) cudaStreamSynchronize(x.stream);
    cudaFree(h->mem);
    cudaFree(h->tables);
    cudaFree(h->itables);
    cudaFree(h->stage);
    cudaFree(h->flush);
    cudaFree(x.sc);
    cudaFree(x.part);
    cudaFree(x.spec);
    cudaFree(x.tri_im);
    cudaFree(x.tw_x);
    cudaFree(x.tw_z);
    cudaFreeHost(x.sc_host);
    cudaFreeHost(x.int_host);
    for (int q = 0; q < 2; q++) {
        if (h->ev[q]) cudaEventDestroy(h->ev[q]);
        if (x.tev[q]) cudaEventDestroy(x.tev[q]);
    }
    if (x.stream) cudaStreamDestroy(x.stream);
    delete h;
    return PVOF_OK;
}

// the spectral preconditioner's launch shapes, tables and spectrum (host
// tables in FP64 from the same modified wave numbers as the operator)
static int spec_setup(GpuExec &x, const Dom3 &d, const pvof_grid_desc *g)
{
    SpecDims &sd = x.sd;
    sd.N = d.NX - 1;
    sd.K = d.NZ - 1;
    sd.ny = d.NY - 1;
    sd.H = sd.N / 2 + 1;
    sd.logN = 0;
    while ((1 << sd.logN) < sd.N) sd.logN++;
    sd.logK = 0;
    while ((1 << sd.logK) < sd.K) sd.logK++;
    sd.g_x = XT / (sd.N / 8);
    sd.ch_z = std::min(32, 256 / (sd.K / 8));
    const double idy2 = d.idy2;
    x.spec_scale = (1.0 / idy2) / ((double)sd.N * (double)sd.K);
    const size_t n = (size_t)sd.K * sd.ny * sd.H;
    std::vector<double> im(n);
    const double pi = 3.14159265358979323846;
    for (int kz = 0; kz < sd.K; kz++)
        for (int kx = 0; kx < sd.H; kx++) {
            const double lam = (d.idx2 * (2.0 - 2.0 * std::cos(2.0 * pi * kx / sd.N)) +
                                d.idz2 * (2.0 - 2.0 * std::cos(2.0 * pi * kz / sd.K))) / idy2;
            double cprev = 0.0;
            for (int j = 0; j < sd.ny; j++) {
                const double b = ((j == 0 || j == sd.ny - 1) ? 1.0 : 2.0) + lam;
                const double m = b + cprev;
                const size_t q = ((size_t)kz * sd.ny + j) * sd.H + kx;
                im[q] = 1.0 / m;
                cprev = -im[q];
            }
        }
    (void)g;
    std::vector<double2> twx((size_t)sd.N), twz((size_t)sd.K);
    for (int q = 0; q < sd.N; q++) twx[q] = make_double2(std::cos(2.0 * pi * q / sd.N), -std::sin(2.0 * pi * q / sd.N));
    for (int q = 0; q < sd.K; q++) twz[q] = make_double2(std::cos(2.0 * pi * q / sd.K), -std::sin(2.0 * pi * q / sd.K));
    if (cudaMalloc(&x.tw_x, twx.size() * sizeof(double2)) != cudaSuccess ||
        cudaMalloc(&x.tw_z, twz.size() * sizeof(double2)) != cudaSuccess ||
        cudaMemcpy(x.tw_x, twx.data(), twx.size() * sizeof(double2), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(x.tw_z, twz.data(), twz.size() * sizeof(double2), cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(PVOF_ENOMEM, "twiddle tables");
    if (cudaMalloc(&x.spec, n * sizeof(double2)) != cudaSuccess ||
        cudaMalloc(&x.tri_im, n * sizeof(double)) != cudaSuccess)
        return fail(PVOF_ENOMEM, "device memory for the spectral preconditioner");
    if (cudaMemcpy(x.tri_im, im.data(), n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(PVOF_ECUDA, "spectral tables upload");
    return PVOF_OK;
}

int create(const pvof_grid_desc *g, const pvof_params *p, int device, Handle **out)
{
    *out = nullptr;
    if (!g->periodic[0] || g->periodic[1] || !g->periodic[2])
        return fail(PVOF_EINVAL, "the 3D mode needs x and z periodic and walls in y");
    if (g->NXM < 8 || g->NYM < 8 || g->NZM < 8) return fail(PVOF_EINVAL, "the 3D mode needs at least 8 cells per direction");
    if (p->pressure_warm_start) return fail(PVOF_EINVAL, "the pressure warm starts are 2D only");
    if (p->pressure_preconditioner < 0 || p->pressure_preconditioner > 1)
        return fail(PVOF_EINVAL, "pressure_preconditioner must be 0 (Jacobi) or 1 (spectral)");
    if (p->pressure_preconditioner) {
        auto pow2 = [](int n) { return n >= 2 && n <= 1024 && (n & (n - 1)) == 0; };
        if (!pow2(g->NXM) || !pow2(g->NZM) || g->NYM > 4096)
            return fail(PVOF_EINVAL, "the 3D spectral preconditioner needs power-of-two x and z cell counts up to 1024");
    }
    if (p->stencil_fp32 < 0 || p->stencil_fp32 > 1) return fail(PVOF_EINVAL, "stencil_fp32 must be 0 or 1");
    const double hx = (g->xmax - g->xmin) / g->NXM, hy = (g->ymax - g->ymin) / g->NYM, hz = (g->zmax - g->zmin) / g->NZM;
    if (!(hx > 0 && hy > 0 && hz > 0)) return fail(PVOF_EINVAL, "empty box");
    CK3(cudaSetDevice(device));
    Handle *h = new Handle();
    h->device = device;
    Box3<GpuExec> &b = h->b;
    b.g = *g;
    b.p = *p;
    b.ph.rho_g = p->rho2 / p->rho1;
    b.ph.mu_g = p->mu2 / p->mu1;
    Dom3 &d = b.d;
    d.NX = g->NXM + 1;
    d.NY = g->NYM + 1;
    d.NZ = g->NZM + 1;
    d.P = ((OX + d.NX + NG) + 7) / 8 * 8;
    d.S = (long long)d.P * (d.NY + 2 * NG);
    GpuExec &x = b.x;
    x.field_elems = (size_t)d.S * (size_t)(d.NZ + 2 * NG);
    x.origin = (long long)NG * d.S + (long long)NG * d.P + OX;
    auto bail = [&](int rc) { destroy(h); return rc; };
    if (cudaStreamCreateWithFlags(&x.stream, cudaStreamNonBlocking) != cudaSuccess) return bail(fail(PVOF_ECUDA, "stream"));
    // fields (zeroed once: never-written positions read as the reference's zero-initialised arrays)
    const int nfields = F3_COUNT;
    if (cudaMalloc(&h->mem, x.field_elems * sizeof(double) * nfields) != cudaSuccess)
        return bail(fail(PVOF_ENOMEM, "device memory for the 3D fields"));
    if (cudaMemsetAsync(h->mem, 0, x.field_elems * sizeof(double) * nfields, x.stream) != cudaSuccess)
        return bail(fail(PVOF_ECUDA, "memset"));
    for (int q = 0; q < F3_COUNT; q++) b.f[q] = h->mem + (size_t)q * x.field_elems + x.origin;
    // tables: metrics per axis (8 arrays), weights, map multipliers; map sources
    HostAxis ax[3];
    const bool per[3] = {true, false, true};
    const double lo[3] = {g->xmin, g->ymin, g->zmin}, hi[3] = {g->xmax, g->ymax, g->zmax};
    const int N[3] = {d.NX, d.NY, d.NZ};
    for (int a = 0; a < 3; a++) {
        host_axis_metrics(ax[a], N[a], lo[a], hi[a], per[a]);
        host_axis_maps(ax[a], N[a], per[a], false, false, false, a, g->wall[PVOF_BOTTOM], g->wall[PVOF_TOP]);
    }
    std::vector<double> dt_;
    std::vector<int> it_;
    std::vector<size_t> doff, ioff;
    auto addd = [&](const std::vector<double> &v) { doff.push_back(dt_.size()); dt_.insert(dt_.end(), v.begin(), v.end()); };
    auto addi = [&](const std::vector<int> &v) { ioff.push_back(it_.size()); it_.insert(it_.end(), v.begin(), v.end()); };
    for (int a = 0; a < 3; a++) {
        addd(ax[a].idf); addd(ax[a].idc); addd(ax[a].df); addd(ax[a].dc); addd(ax[a].w);
        for (int kind = 0; kind < K_COUNT; kind++) {
            addd(ax[a].mul[kind]);
            addi(ax[a].src[kind]);
        }
    }
    if (cudaMalloc(&h->tables, dt_.size() * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&h->itables, it_.size() * sizeof(int)) != cudaSuccess)
        return bail(fail(PVOF_ENOMEM, "device memory for the tables"));
    if (cudaMemcpy(h->tables, dt_.data(), dt_.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->itables, it_.data(), it_.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess)
        return bail(fail(PVOF_ECUDA, "table upload"));
    size_t qd = 0, qi = 0;
    for (int a = 0; a < 3; a++) {
        const double *idf = h->tables + doff[qd++] + NG, *idc = h->tables + doff[qd++] + NG;
        const double *df = h->tables + doff[qd++] + NG, *dc = h->tables + doff[qd++] + NG;
        const double *w = h->tables + doff[qd++] + NG;
        if (a == 0) { d.idx_u = idf; d.idx_c = idc; d.dx_u = df; d.dx_c = dc; d.wx = w; }
        if (a == 1) { d.idy_v = idf; d.idy_c = idc; d.dy_v = df; d.dy_c = dc; d.wy = w; }
        if (a == 2) { d.idz_w = idf; d.idz_c = idc; d.dz_w = df; d.dz_c = dc; d.wz = w; }
        for (int kind = 0; kind < K_COUNT; kind++) {
            Axis A{h->itables + ioff[qi++], h->tables + doff[qd++]};
            if (a == 0) d.map[kind].x = A;
            if (a == 1) d.map[kind].y = A;
            if (a == 2) d.map[kind].z = A;
        }
    }
    d.idx2 = ax[0].idc[1 + NG] * ax[0].idc[1 + NG];
    d.idy2 = ax[1].idc[1 + NG] * ax[1].idc[1 + NG];
    d.idz2 = ax[2].idc[1 + NG] * ax[2].idc[1 + NG];
    d.idx_u1 = ax[0].idf[1 + NG];
    if (p->pressure_preconditioner && spec_setup(x, d, g) < 0) return bail(PVOF_ENOMEM);
    {
        // one partial sum per block of the largest reduction grid: the
        // generic sums, the momentum and pressure passes (a pressure block takes
        // twice a momentum block's cells) and the spectral inverse-x pass
        const dim3 vg = GpuExec::vgrid(Range{0, d.NX, 0, d.NY, 0, d.NZ});
        size_t nb = std::max((size_t)NBR, (size_t)vg.x * vg.y * vg.z);
        if (p->pressure_preconditioner) nb = std::max(nb, (size_t)GpuExec::spec_xblocks(x.sd));
        x.pstride = 4 * nb;
    }
    if (cudaMalloc(&x.sc, sizeof(Sc3)) != cudaSuccess || cudaMalloc(&x.part, sizeof(double) * NSLOT * x.pstride) != cudaSuccess)
        return bail(fail(PVOF_ENOMEM, "device scalars"));
    cudaMemsetAsync(x.sc, 0, sizeof(Sc3), x.stream);
    cudaMemsetAsync(x.part, 0, sizeof(double) * NSLOT * x.pstride, x.stream);
    if (cudaMallocHost(&x.sc_host, sizeof(Sc3)) != cudaSuccess || cudaMallocHost(&x.int_host, sizeof(int)) != cudaSuccess)
        return bail(fail(PVOF_ENOMEM, "pinned scalars"));
    h->stage_elems = block_elems(d, false);
    if (cudaMalloc(&h->stage, h->stage_elems * sizeof(double)) != cudaSuccess)
        return bail(fail(PVOF_ENOMEM, "staging block"));
    for (int q = 0; q < 2; q++)
        if (cudaEventCreate(&h->ev[q]) != cudaSuccess || cudaEventCreate(&x.tev[q]) != cudaSuccess)
            return bail(fail(PVOF_ECUDA, "event"));
    if (cudaStreamSynchronize(x.stream) != cudaSuccess) return bail(fail(PVOF_ECUDA, "set-up"));
    *out = h;
    return PVOF_OK;
}

// field of the ABI -> (slot, ghost kind, no-ghost, derived quantity)
struct FieldRef {
    int slot, kind, ng, xf;
};
static bool field_ref(const Handle *h, int field, bool upload, FieldRef &r)
{
    r = FieldRef{-1, K_SCALAR, 0, 0};
    switch (field) {
    case PVOF_F_C_L: r.slot = F3_CL; break;
    case PVOF_F_F: r.slot = (upload || !h->b.initialized) ? F3_F : F3_CL; break;
    case PVOF_F_C_G: if (upload) return false; r.slot = F3_CL; r.xf = 1; break;
    case PVOF_F_RHO: if (upload) return false; r.slot = F3_CL; r.xf = 2; break;
    case PVOF_F_MU: if (upload) return false; r.slot = F3_CL; r.xf = 3; break;
    case PVOF_F_PSI_LG: r.slot = F3_PSI; break;
    case PVOF_F_CH_RHS_N:
    case PVOF_F_CH_RHS_CUR: r.slot = F3_RN; break;
    case PVOF_F_U: r.slot = F3_U; r.kind = K_U; break;
    case PVOF_F_V: r.slot = F3_V; r.kind = K_V; break;
    case PVOF_F_W: r.slot = F3_W; r.kind = K_W; break;
    case PVOF_F_P: r.slot = F3_P; r.kind = K_PRESSURE; break;
    case PVOF_F_DELTAP: r.slot = F3_DP; r.kind = K_PRESSURE; break;
    case PVOF_F_P_RHS: r.slot = F3_PRHS; r.kind = K_WRAP_C; break;
    case PVOF_F_U_EXPLICIT: case PVOF_F_U_EXPLICIT_OLD: r.slot = F3_U_EXO; r.ng = 1; break;
    case PVOF_F_V_EXPLICIT: case PVOF_F_V_EXPLICIT_OLD: r.slot = F3_V_EXO; r.ng = 1; break;
    case PVOF_F_W_EXPLICIT: case PVOF_F_W_EXPLICIT_OLD: r.slot = F3_W_EXO; r.ng = 1; break;
    case PVOF_F_U_VISC_EXPLICIT: case PVOF_F_U_VISC_EXPLICIT_OLD: r.slot = F3_U_VXO; r.ng = 1; break;
    case PVOF_F_V_VISC_EXPLICIT: case PVOF_F_V_VISC_EXPLICIT_OLD: r.slot = F3_V_VXO; r.ng = 1; break;
    case PVOF_F_W_VISC_EXPLICIT: case PVOF_F_W_VISC_EXPLICIT_OLD: r.slot = F3_W_VXO; r.ng = 1; break;
    case PVOF_F_U_RHS: r.slot = F3_U_RHS; r.ng = 1; break;
    case PVOF_F_V_RHS: r.slot = F3_V_RHS; r.ng = 1; break;
    case PVOF_F_W_RHS: r.slot = F3_W_RHS; r.ng = 1; break;
    case PVOF_F_FSIG_OLD_X: r.slot = F3_FSO_X; r.ng = 1; break;
    case PVOF_F_FSIG_OLD_Y: r.slot = F3_FSO_Y; r.ng = 1; break;
    case PVOF_F_FSIG_OLD_Z: r.slot = F3_FSO_Z; r.ng = 1; break;
    case PVOF_F_FSIG_NEW_X: r.slot = F3_FSN_X; r.ng = 1; break;
    case PVOF_F_FSIG_NEW_Y: r.slot = F3_FSN_Y; r.ng = 1; break;
    case PVOF_F_FSIG_NEW_Z: r.slot = F3_FSN_Z; r.ng = 1; break;
    default: return false;
    }
    return true;
}

static bool is_ng_field(int field)
{
    return (field >= PVOF_F_U_EXPLICIT && field <= PVOF_F_FSIG_NEW_Y) || (field >= PVOF_F_W_EXPLICIT && field <= PVOF_F_FSIG_NEW_Z);
}

size_t block_count(const Handle *h, int field)
{
    if (field < 0 || field >= PVOF_F_COUNT) return 0;
    return block_elems(h->b.d, is_ng_field(field));
}

int upload(Handle *h, int field, const double *host, size_t count)
{
    FieldRef r;
    if (!field_ref(h, field, true, r)) return fail(PVOF_EINVAL, "this field cannot be uploaded in the 3D mode");
    const size_t n = block_elems(h->b.d, r.ng);
    if (count != n) return fail(PVOF_EINVAL, "block size mismatch");
    CK3(cudaSetDevice(h->device));
    GpuExec &x = h->b.x;
    CK3(cudaMemcpyAsync(h->stage, host, n * sizeof(double), cudaMemcpyHostToDevice, x.stream));
    k3_unpack<<<592, 256, 0, x.stream>>>(h->b.d, h->b.f[r.slot], h->stage, r.ng);
    x.note();
    CK3(cudaStreamSynchronize(x.stream));
    return x.status();
}

int download(Handle *h, int field, double *host, size_t count)
{
    FieldRef r;
    if (!field_ref(h, field, false, r)) return fail(PVOF_EINVAL, "this field is not kept in the 3D mode");
    const size_t n = block_elems(h->b.d, r.ng);
    if (count != n) return fail(PVOF_EINVAL, "block size mismatch");
    CK3(cudaSetDevice(h->device));
    GpuExec &x = h->b.x;
    const Dom3 &d = h->b.d;
    const double *fld = h->b.f[r.slot];
    switch (r.kind) {
    case K_U: k3_pack<K_U><<<592, 256, 0, x.stream>>>(d, h->b.ph, fld, h->stage, r.ng, r.xf); break;
    case K_V: k3_pack<K_V><<<592, 256, 0, x.stream>>>(d, h->b.ph, fld, h->stage, r.ng, r.xf); break;
    case K_W: k3_pack<K_W><<<592, 256, 0, x.stream>>>(d, h->b.ph, fld, h->stage, r.ng, r.xf); break;
    case K_PRESSURE: k3_pack<K_PRESSURE><<<592, 256, 0, x.stream>>>(d, h->b.ph, fld, h->stage, r.ng, r.xf); break;
    case K_WRAP_C: k3_pack<K_WRAP_C><<<592, 256, 0, x.stream>>>(d, h->b.ph, fld, h->stage, r.ng, r.xf); break;
    default: k3_pack<K_SCALAR><<<592, 256, 0, x.stream>>>(d, h->b.ph, fld, h->stage, r.ng, r.xf); break;
    }
    x.note();
    CK3(cudaMemcpyAsync(host, h->stage, n * sizeof(double), cudaMemcpyDeviceToHost, x.stream));
    CK3(cudaStreamSynchronize(x.stream));
    return x.status();
}

int synchronize(Handle *h)
{
    CK3(cudaSetDevice(h->device));
    CK3(cudaStreamSynchronize(h->b.x.stream));
    return h->b.x.status();
}

int set_stage(Handle *h, int stage, double dt)
{
    if (stage < 0 || stage > 2 || !(dt > 0.0)) return fail(PVOF_EINVAL, "stage must be 0..2 and dt positive");
    h->b.stage = stage;
    h->b.dt = dt;
    return PVOF_OK;
}

int initialize(Handle *h)
{
    CK3(cudaSetDevice(h->device));
    const int rc = h->b.initialize();
    if (rc < 0) return rc;
    CK3(cudaStreamSynchronize(h->b.x.stream));
    return h->b.x.status();
}

int substep(Handle *h, pvof_stats *st)
{
    CK3(cudaSetDevice(h->device));
    if (!h->b.initialized) return fail(PVOF_EINVAL, "pvof_initialize() first");
    if (!(h->b.dt > 0.0)) return fail(PVOF_EINVAL, "pvof_set_stage() first");
    const int rc = h->b.substep(st);
    if (rc == PVOF_EDIVERGED) return fail(rc, "the outer Poisson loop did not reach div < 1e-6 in 10 passes");
    return rc;
}

int run_steps(Handle *h, int nsteps, double dt, pvof_stats *st)
{
    CK3(cudaSetDevice(h->device));
    if (!h->b.initialized) return fail(PVOF_EINVAL, "pvof_initialize() first");
    if (nsteps < 0 || !(dt > 0.0)) return fail(PVOF_EINVAL, "nsteps >= 0 and dt > 0");
    const int rc = h->b.run_steps(nsteps, dt, st);
    if (rc == PVOF_EDIVERGED) return fail(rc, "the outer Poisson loop did not reach div < 1e-6 in 10 passes");
    return rc;
}

int liquid_mass(Handle *h, double *m)
{
    CK3(cudaSetDevice(h->device));
    return h->b.liquid_mass(m);
}

long long launch_count(const Handle *h) { return h->b.x.launches; }

int set_solver_timing(Handle *h, int on)
{
    h->b.x.timing = on ? 1 : 0;
    for (int k = 0; k < 3; k++) {
        h->b.x.sol_ms[k] = 0.0;
        h->b.sol_launches[k] = h->b.sol_iters[k] = h->b.sol_cell_iters[k] = 0;
    }
    return PVOF_OK;
}

int solver_timing(const Handle *h, int solver, double *ms, long long *launches, long long *iters, long long *cell_iters)
{
    if (solver < 0 || solver > 2) return fail(PVOF_EINVAL, "bad solver index");
    if (ms) *ms = h->b.x.sol_ms[solver];
    if (launches) *launches = h->b.sol_launches[solver];
    if (iters) *iters = h->b.sol_iters[solver];
    if (cell_iters) *cell_iters = h->b.sol_cell_iters[solver];
    return PVOF_OK;
}
double clamp_total(const Handle *h) { return h->b.clamp_total; }

int timer_start(Handle *h)
{
    CK3(cudaSetDevice(h->device));
    CK3(cudaEventRecord(h->ev[0], h->b.x.stream));
    return PVOF_OK;
}

int timer_stop(Handle *h, double *ms)
{
    CK3(cudaSetDevice(h->device));
    CK3(cudaEventRecord(h->ev[1], h->b.x.stream));
    CK3(cudaEventSynchronize(h->ev[1]));
    float t = 0.f;
    CK3(cudaEventElapsedTime(&t, h->ev[0], h->ev[1]));
    *ms = t;
    return h->b.x.status();
}

// writes a buffer twice the size of the L2 so the next launch starts cold
int flush_l2(Handle *h)
{
    CK3(cudaSetDevice(h->device));
    if (!h->flush) {
        int l2 = 0;
        CK3(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, h->device));
        h->flush_elems = (size_t)2 * (size_t)l2 / sizeof(double);
        CK3(cudaMalloc(&h->flush, h->flush_elems * sizeof(double)));
    }
    k3_flush<<<592, 256, 0, h->b.x.stream>>>(h->flush, h->flush_elems, 0.0);
    CK3(cudaGetLastError());
    return PVOF_OK;
}

}  // namespace pvof3
