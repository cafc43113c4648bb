// Constant-density Poisson solver by Fourier transform in the periodic x
// direction and tridiagonal systems in the wall-normal y direction:
// Pressure_solve_xz_period (Eulerian/lsolver/psolve_fft.c:638-983) with its
// coefficients (Pressure_calc_coeff, :467-591) and tridiagonal solves
// (tridiag, :141-163), for the planar 2D mode (one z plane: the z transform
// of the reference is the identity there).
//
//   1. rows: real forward transform of length N = NX-1 times 1/N, two rows as
//      one complex transform, stored as N/2 + 1 complex numbers;
//   2. every wave number: the tridiagonal system along y of
//      (as, ap - 2 (1 - cos(2 pi k / N)) / dx^2, an), the mean mode pinned to
//      zero at j = 0 (Neumann walls).  On the uniform grid the mirror walls'
//      eigenvectors are cosines, so a column is a cosine transform, a division
//      by the eigenvalues and the transform back (k_fft_solve_y), in shared
//      memory; columns too long for that or with a large prime factor take the
//      Thomas algorithm, one thread per wave number (k_fft_thomas);
//   3. rows: unnormalised inverse transform, two at a time.
//
// The transforms are Stockham passes of radix 4, 2, 3, 5 and any larger prime
// factor between two buffers in shared memory, twiddles from one table per
// axis.  Bound by the passes' shared-memory traffic and the latency of their
// barriers; the plane itself stays in L2.  B200, device time of the three
// kernels: 1024x2048 1373 -> 86 us, 200x800 882 -> 21 us (Thomas chains of
// 800 to 2048 dependent divisions on 2 to 8 blocks, and a direct transform
// with a sincospi per term where N was no power of two).
#include <cmath>

#include "pvof_device.cuh"
#include "pvof_kernels.cuh"

namespace pvof {

namespace {

constexpr int FT = 256;    // threads per block of the x transforms
constexpr int FTY = 512;   // of the y solve, whose two buffers leave room for one or two blocks per SM

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// times -i (forward) or i (inverse)
template <bool INV>
__device__ __forceinline__ double2 crot(double2 a) { return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x); }
template <bool INV>
__device__ __forceinline__ double2 twiddle(const double2 *__restrict__ tw, int k)
{
    double2 w = __ldg(tw + k);
    if (INV) w.y = -w.y;
    return w;
}

// One Stockham pass of radix R over `count` transforms of n points each
// (transform g at x + g n): with s the product of the radices done so far and
// m = n / (s R), butterfly (p, q) reads x[q + s (p + m k)] and writes
// y[q + s (R p + k)], times exp(-+2 pi i p k / (n / s)) = tw[p k s].
template <int R, bool INV>
__device__ void fft_pass(const double2 *x, double2 *y, int n, int s, int count, const double2 *__restrict__ tw)
{
    const unsigned nb = (unsigned)n / R, m = nb / (unsigned)s;
    for (unsigned t = threadIdx.x; t < nb * (unsigned)count; t += blockDim.x) {
        const unsigned g = t / nb, b = t - g * nb, p = b / (unsigned)s, q = b - p * (unsigned)s;
        const double2 *xi = x + (size_t)g * n + q + s * p;
        double2 *yo = y + (size_t)g * n + q + (size_t)s * R * p;
        double2 v[R];
#pragma unroll
        for (int k = 0; k < R; k++) v[k] = xi[(size_t)s * m * k];
        double2 o[R];
        if constexpr (R == 2) {
            o[0] = cadd(v[0], v[1]);
            o[1] = csub(v[0], v[1]);
        } else if constexpr (R == 4) {
            const double2 a = cadd(v[0], v[2]), c = csub(v[0], v[2]), d = cadd(v[1], v[3]), e = crot<INV>(csub(v[1], v[3]));
            o[0] = cadd(a, d);
            o[1] = cadd(c, e);
            o[2] = csub(a, d);
            o[3] = csub(c, e);
        } else if constexpr (R == 3) {
            const double h = 0.86602540378443864676;
            const double2 a = cadd(v[1], v[2]), e = crot<INV>(csub(v[1], v[2]));
            const double2 c = make_double2(v[0].x - 0.5 * a.x, v[0].y - 0.5 * a.y), d = make_double2(h * e.x, h * e.y);
            o[0] = cadd(v[0], a);
            o[1] = cadd(c, d);
            o[2] = csub(c, d);
        } else {
            const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
            const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
            const double2 a = cadd(v[1], v[4]), b5 = cadd(v[2], v[3]);
            const double2 d = crot<INV>(csub(v[1], v[4])), e = crot<INV>(csub(v[2], v[3]));
            const double2 f = make_double2(v[0].x + c1 * a.x + c2 * b5.x, v[0].y + c1 * a.y + c2 * b5.y);
            const double2 h = make_double2(v[0].x + c2 * a.x + c1 * b5.x, v[0].y + c2 * a.y + c1 * b5.y);
            const double2 u = make_double2(s1 * d.x + s2 * e.x, s1 * d.y + s2 * e.y);
            const double2 w = make_double2(s2 * d.x - s1 * e.x, s2 * d.y - s1 * e.y);
            o[0] = cadd(v[0], cadd(a, b5));
            o[1] = cadd(f, u);
            o[4] = csub(f, u);
            o[2] = cadd(h, w);
            o[3] = csub(h, w);
        }
        yo[0] = o[0];
#pragma unroll
        for (int k = 1; k < R; k++) yo[(size_t)s * k] = p == 0 ? o[k] : cmul(o[k], twiddle<INV>(tw, (int)(p * k * s)));
    }
}

// the same pass for any other prime factor r: one output per thread
template <bool INV>
__device__ void fft_pass_any(const double2 *x, double2 *y, int n, int r, int s, int count, const double2 *__restrict__ tw)
{
    const unsigned m = (unsigned)(n / (s * r));
    for (unsigned t = threadIdx.x; t < (unsigned)(n * count); t += blockDim.x) {
        const unsigned g = t / (unsigned)n, b = t - g * n, q = b % (unsigned)s, pk = b / (unsigned)s, p = pk / (unsigned)r, k = pk - p * r;
        const double2 *xi = x + (size_t)g * n + q + (size_t)s * p;
        double2 a = xi[0];
        unsigned e = 0;   // k j (n / r) mod n
        for (int j = 1; j < r; j++) {
            e += k * (unsigned)(n / r);
            if (e >= (unsigned)n) e -= n;
            a = cadd(a, cmul(xi[(size_t)s * m * j], twiddle<INV>(tw, (int)e)));
        }
        y[t] = cmul(a, twiddle<INV>(tw, (int)(p * k * s)));   // t = g n + q + s (r p + k)
    }
}

// `count` transforms of n points at a (b: as much scratch); returns where the
// result is
template <bool INV>
__device__ double2 *fft_run(double2 *a, double2 *b, const FftRadices &R, int n, int count, const double2 *__restrict__ tw)
{
    int s = 1;
    for (int f = 0; f < R.n; f++) {
        const int r = R.r[f];
        if (r == 4) fft_pass<4, INV>(a, b, n, s, count, tw);
        else if (r == 2) fft_pass<2, INV>(a, b, n, s, count, tw);
        else if (r == 3) fft_pass<3, INV>(a, b, n, s, count, tw);
        else if (r == 5) fft_pass<5, INV>(a, b, n, s, count, tw);
        else fft_pass_any<INV>(a, b, n, r, s, count, tw);
        __syncthreads();
        double2 *t = a;
        a = b;
        b = t;
        s *= r;
    }
    return a;
}

}  // namespace

// The radices of an n-point transform: fours, a two, threes, fives, then the
// other primes.
FftRadices fft_radices(int n)
{
    FftRadices R;
    R.n = 0;
    R.largest = 1;
    auto take = [&](int r) {
        while (n % r == 0 && n > 1) {
            R.r[R.n++] = r;
            n /= r;
            if (r > R.largest) R.largest = r;
        }
    };
    for (int r : {4, 2, 3, 5}) take(r);
    for (int r = 7; r * r <= n; r += 2) take(r);
    if (n > 1) take(n);
    return R;
}

// step 1: spectrum k of row j at hat[j][k] (complex, row pitch of the planes)
__global__ void __launch_bounds__(FT) k_fft_forward(Dom d, FftArgs A, const double *__restrict__ rhs, double *__restrict__ hat)
{
    extern __shared__ double2 sm[];
    const int P = d.P, N = A.N, M = A.M, G = A.pairs, g0 = blockIdx.x * G;
    double2 *a = sm, *b = sm + (size_t)G * N;
    for (int t = threadIdx.x; t < G * N; t += blockDim.x) {
        const int g = t / N, i = t - g * N, j = 2 * (g0 + g);
        a[t] = make_double2(j < M ? AT_(rhs, i, j) : 0.0, j + 1 < M ? AT_(rhs, i, j + 1) : 0.0);
    }
    __syncthreads();
    const double2 *z = fft_run<false>(a, b, A.rx, N, G, A.twx);
    const int H = N / 2 + 1;
    const double sc = 0.5 * A.inx;
    for (int t = threadIdx.x; t < G * H; t += blockDim.x) {
        const int g = t / H, k = t - g * H, j = 2 * (g0 + g);
        const double2 zk = z[(size_t)g * N + k], zn = z[(size_t)g * N + (k ? N - k : 0)];
        if (j < M) reinterpret_cast<double2 *>(&AT_(hat, 0, j))[k] = make_double2((zk.x + zn.x) * sc, (zk.y - zn.y) * sc);
        if (j + 1 < M)
            reinterpret_cast<double2 *>(&AT_(hat, 0, j + 1))[k] = make_double2((zk.y + zn.y) * sc, (zn.x - zk.x) * sc);
    }
}

// step 2, by cosine transforms: `cols` wave numbers per block.  A column x of
// M rows in the order v_n = x_2n, v_(M-1-n) = x_(2n+1) has, with V its
// transform and w_k = exp(-i pi k / 2M), the cosine transform
// Z_k = (w_k V_k + conj(w_k) V_(M-k)) / 2, and back V_k = conj(w_k) (Z_k -
// i Z_(M-k)) (J. Makhoul, A fast cosine transform in one and two dimensions,
// IEEE Trans. ASSP 28, 1980); both are linear, so a complex column is one
// transform.  The mean mode: its first row's equation is replaced by x_0 = 0,
// i.e. the right-hand side made compatible through that row, the column's
// constant left at zero and x_0 taken off.
__global__ void __launch_bounds__(FTY) k_fft_solve_y(Dom d, FftArgs A, double *__restrict__ hat)
{
    extern __shared__ double2 sm[];
    __shared__ double red[FTY / 32];
    const int P = d.P, M = A.M, H = A.N / 2 + 1, C = A.cols, c0 = blockIdx.x * C, nc = H - c0 < C ? H - c0 : C;
    double2 *a = sm, *b = sm + (size_t)C * M;
    double part = 0.0;   // the mean mode's sum over the rows above the first
    for (int t = threadIdx.x; t < nc * M; t += blockDim.x) {
        const int j = t / nc, c = t - j * nc;
        const double2 v = reinterpret_cast<const double2 *>(&AT_(hat, 0, j))[c0 + c];
        if (c0 + c == 0 && j > 0) part += v.x;
        a[(size_t)c * M + (j & 1 ? M - 1 - (j >> 1) : j >> 1)] = v;
    }
    if (c0 == 0) {
        for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int q = 0; q < FTY / 32; q++) s += red[q];
            a[0] = make_double2(-s, 0.0);
        }
    }
    __syncthreads();
    double2 *z = fft_run<false>(a, b, A.ry, M, nc, A.twy);
    const double im = 1.0 / (double)M;
    const int half = M / 2 + 1;
    for (int t = threadIdx.x; t < nc * half; t += blockDim.x) {
        const int c = t / half, k = t - c * half, k2 = k ? M - k : 0;
        double2 *v = z + (size_t)c * M;
        const double2 V = v[k], U = v[k2], w = A.wy[k];
        const double lx = A.mw[c0 + c];
        // with w' = w_(M-k) = -i conj(w_k)
        const double2 zk = make_double2(0.5 * ((w.x * V.x - w.y * V.y) + (w.x * U.x + w.y * U.y)),
                                        0.5 * ((w.x * V.y + w.y * V.x) + (w.x * U.y - w.y * U.x)));
        const double ek = -(A.ly[k] + lx), fk = (c0 + c == 0 && k == 0) ? 0.0 : im / ek;
        const double2 Z = make_double2(zk.x * fk, zk.y * fk);
        if (k == 0) {
            v[0] = Z;
            continue;
        }
        const double2 x = make_double2(-w.y, -w.x);   // w'
        const double2 zn = make_double2(0.5 * ((x.x * U.x - x.y * U.y) + (x.x * V.x + x.y * V.y)),
                                        0.5 * ((x.x * U.y + x.y * U.x) + (x.x * V.y - x.y * V.x)));
        const double fn = im / -(A.ly[k2] + lx);
        const double2 Y = make_double2(zn.x * fn, zn.y * fn);
        // conj(w) (Z - i Y), conj(w') (Y - i Z)
        const double2 p = make_double2(Z.x + Y.y, Z.y - Y.x), q = make_double2(Y.x + Z.y, Y.y - Z.x);
        v[k] = make_double2(w.x * p.x + w.y * p.y, w.x * p.y - w.y * p.x);
        if (k2 != k) v[k2] = make_double2(x.x * q.x + x.y * q.y, x.x * q.y - x.y * q.x);
    }
    __syncthreads();
    z = fft_run<true>(z, z == a ? b : a, A.ry, M, nc, A.twy);
    const double pin = z[0].x;   // the mean mode's first row
    for (int t = threadIdx.x; t < nc * M; t += blockDim.x) {
        const int j = t / nc, c = t - j * nc;
        double2 v = z[(size_t)c * M + (j & 1 ? M - 1 - (j >> 1) : j >> 1)];
        if (c0 + c == 0) v = make_double2(v.x - pin, 0.0);
        reinterpret_cast<double2 *>(&AT_(hat, 0, j))[c0 + c] = v;
    }
}

// step 2, by the Thomas algorithm (psolve_fft.c:141-163) along y for every
// wave number k; as/ap/an per row, mw[k] the modified wavenumber; gam is scratch
__global__ void k_fft_thomas(Dom d, FftArgs A, const double *__restrict__ as_, const double *__restrict__ ap_,
                             const double *__restrict__ an_, double *__restrict__ hat, double *__restrict__ gam)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x, M = A.M;
    if (k > A.N / 2) return;
    const int P = d.P;
    auto X = [&](int j) -> double2 & { return reinterpret_cast<double2 *>(&AT_(hat, 0, j))[k]; };
    auto pinned = [&](int j) { return k == 0 && j == 0; };
    double bet = pinned(0) ? 1.0 : ap_[0] - A.mw[k];
    double2 x = pinned(0) ? make_double2(0.0, 0.0) : make_double2(X(0).x / bet, X(0).y / bet);
    X(0) = x;
    for (int j = 1; j < M; j++) {
        const double g = (pinned(j - 1) ? 0.0 : an_[j - 1]) / bet;
        AT_(gam, k, j) = g;
        bet = ap_[j] - A.mw[k] - as_[j] * g;
        const double2 r = X(j);
        x = make_double2((r.x - as_[j] * x.x) / bet, (r.y - as_[j] * x.y) / bet);
        X(j) = x;
    }
    for (int j = M - 2; j >= 0; j--) {
        const double g = AT_(gam, k, j + 1);
        const double2 r = X(j);
        x = make_double2(r.x - g * x.x, r.y - g * x.y);
        X(j) = x;
    }
}

// step 3: out[j][0..N) = unnormalised inverse transform of the rows' spectra
__global__ void __launch_bounds__(FT) k_fft_inverse(Dom d, FftArgs A, const double *__restrict__ hat, double *__restrict__ out)
{
    extern __shared__ double2 sm[];
    const int P = d.P, N = A.N, M = A.M, G = A.pairs, g0 = blockIdx.x * G, H = N / 2 + 1;
    double2 *a = sm, *b = sm + (size_t)G * N;
    for (int t = threadIdx.x; t < G * H; t += blockDim.x) {
        const int g = t / H, k = t - g * H, j = 2 * (g0 + g);
        double2 xa = make_double2(0.0, 0.0), xb = xa;
        if (j < M) xa = reinterpret_cast<const double2 *>(&AT_(hat, 0, j))[k];
        if (j + 1 < M) xb = reinterpret_cast<const double2 *>(&AT_(hat, 0, j + 1))[k];
        if (k == 0 || 2 * k == N) xa.y = xb.y = 0.0;   // real
        a[(size_t)g * N + k] = make_double2(xa.x - xb.y, xa.y + xb.x);
        if (k > 0 && 2 * k < N) a[(size_t)g * N + N - k] = make_double2(xa.x + xb.y, xb.x - xa.y);
    }
    __syncthreads();
    const double2 *z = fft_run<true>(a, b, A.rx, N, G, A.twx);
    for (int t = threadIdx.x; t < G * N; t += blockDim.x) {
        const int g = t / N, i = t - g * N, j = 2 * (g0 + g);
        const double2 v = z[t];
        if (j < M) AT_(out, i, j) = v.x;
        if (j + 1 < M) AT_(out, i, j + 1) = v.y;
    }
}

cudaError_t fft_solve_launch(const Dom &d, const FftArgs &A, const double *thomas, const double *rhs, double *hat, double *gam,
                             double *out, cudaStream_t st)
{
    const size_t smx = 2 * sizeof(double2) * (size_t)A.pairs * A.N, smy = 2 * sizeof(double2) * (size_t)A.cols * A.M;
    if (!raise_dynamic_smem((const void *)k_fft_forward, smx) || !raise_dynamic_smem((const void *)k_fft_inverse, smx) ||
        (A.cols && !raise_dynamic_smem((const void *)k_fft_solve_y, smy)))
        return cudaErrorInvalidValue;
    const unsigned nx = (unsigned)(((A.M + 1) / 2 + A.pairs - 1) / A.pairs);
    k_fft_forward<<<nx, FT, smx, st>>>(d, A, rhs, hat);
    if (A.cols) k_fft_solve_y<<<(unsigned)((A.N / 2 + A.cols) / A.cols), FTY, smy, st>>>(d, A, hat);
    else k_fft_thomas<<<(unsigned)((A.N / 2 + 128) / 128), 128, 0, st>>>(d, A, thomas, thomas + A.M, thomas + 2 * A.M, hat, gam);
    k_fft_inverse<<<nx, FT, smx, st>>>(d, A, hat, out);
    return cudaGetLastError();
}

}  // namespace pvof
