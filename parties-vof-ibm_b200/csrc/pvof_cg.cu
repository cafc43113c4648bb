// Persistent iterative solvers of the two-phase substep.
//
// Each solve is ONE cooperative launch that runs the reference's whole CG
// loop on the device: the blocks step through the iterations together, and the
// exchange of the inner products' sums (grid_exchange) is the barrier between
// its phases.  The sums are added in a fixed tree, by every block or by the
// first one for all, so all blocks hold the same totals and take the same
// convergence decisions.  Cells are assigned to threads by the same
// grid-stride mapping in every phase, so a thread reads back its own cells'
// private values (diagonal, Ad) without a barrier.
//
// Two exchanges per iteration (three in the biharmonic solve through a field):
// the new search direction d_k = z_k + beta d_{k-1} is not written in a phase of
// its own; the matrix-vector phase writes it for its own cells into the second
// direction buffer and evaluates it on the fly at the stencil neighbours (from
// z and d_{k-1}, with the reference's ghost update of d applied through the
// same source maps).  The arithmetic per value is the reference's, so the
// iterates are those of the reference's loop.
//
// The waits are bounded (cooperative_groups::grid_group::sync's are not): if the
// other blocks never arrive, an error is recorded in DevScalars::error and every
// block leaves the solver.  Ranges of at most one cell per resident thread keep
// the whole momentum or pressure solve in registers.
#include "pvof_device.cuh"
#include "pvof_exchange.cuh"
#include "pvof_kernels.cuh"

namespace pvof {

struct Range {
    int i0, j0, w, n;
    __device__ __forceinline__ void ij(int q, int &i, int &j) const { i = i0 + q % w; j = j0 + q / w; }
};

// source of (i,j) under a ghost map (identity in the interior)
__device__ __forceinline__ void src_of(const BcMap &m, int NX, int NY, int i, int j, int &si, int &sj, double &mul)
{
    if (i >= 1 && i <= NX - 2 && j >= 1 && j <= NY - 2) {
        si = i; sj = j; mul = 1.0;
        return;
    }
    si = m.x.src[i + NG];
    sj = m.y.src[j + NG];
    mul = m.x.mul[i + NG] * m.y.mul[j + NG];
}

// ---------------------------------------------------------------------------
// diffuse_solve_biharmonic_pcg (Eulerian/VOF_DIFFUSE.c:339-429): CG on
// [a_dt I + bih L.L] x = b.  The reference iterates over the G range, whose
// half cells (i = NX-1, j = NY-1) hold exact copies of their boundary source
// cells at every iteration; here every physical cell carries the summed measure
// W of itself and its copies.
// Two forms of L(L(p)), the same operands in the same operations.  FLY: both
// Laplacians on the fly, two exchanges an iteration, five inner Laplacians per
// cell (1400 instructions, 140 loads).  Otherwise L(p) goes through a field of its
// own and L of that makes Ap behind a third exchange.  The context picks by the
// number of cells (biharmonic_on_the_fly).  Bound by the latency of the exchanges
// on small ranges, by L2 from about 300 000 cells on: 1024x1024, six solves, on
// the fly 7.7 ms, through the field 4.7.
// ---------------------------------------------------------------------------
template <bool FLY>
__device__ __forceinline__ void cg_biharmonic(const BihArgs &A)
{
    const Dom &d = A.d;
    const int P = d.P, NX = d.NX, NY = d.NY;
    Slots sl{reinterpret_cast<unsigned long long *>(A.partials), &A.scal->error, gridDim.x, blockIdx.x, 1, 0};
    const Range R{0, 0, NX - 1, (NX - 1) * (NY - 1)};
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    const double nk = (double)d.nk;

    // L at a cell of a field given at physical cells, through the scalar ghost
    // update (VOF_DIFFUSE_compute_laplacian)
    auto lap = [&](int i, int j, auto f) {
        return lap_at(d, i, j, [&](int a, int b) {
            int si, sj;
            double mul;
            src_of(A.msc, NX, NY, a, b, si, sj, mul);
            return f(si, sj);
        });
    };
    auto auxf = [&](int a, int b) { return AT_(A.aux, a, b); };
    // L(L(f)) without and with the field
    auto twice = [&](int i, int j, auto f) { return lap(i, j, [&](int a, int b) { return lap(a, b, f); }); };

    double one[1] = {0.0};
    auto xf = [&](int a, int b) { return AT_(A.x, a, b); };
    if (!FLY) {
        for (int q = tid; q < R.n; q += nth) {
            int i, j;
            R.ij(q, i, j);
            AT_(A.aux, i, j) = lap(i, j, xf);
        }
        if (!grid_exchange<1, true>(sl, one)) return;
    }
    double sbb = 0.0, srr = 0.0;
    for (int q = tid; q < R.n; q += nth) {
        int i, j;
        R.ij(q, i, j);
        double ap = A.a_dt * AT_(A.x, i, j) + A.bih * (FLY ? twice(i, j, xf) : lap(i, j, auxf));
        double bv = AT_(A.b, i, j);
        double rv = bv - ap;
        AT_(A.r, i, j) = rv;
        AT_(A.p1, i, j) = rv;
        double m = d.m.wx[i] * d.m.wy[j] * d.wz;
        sbb += m * bv * bv;
        srr += m * rv * rv;
    }
    double both[2] = {sbb, srr};
    if (!grid_exchange<2, true>(sl, both)) return;
    double rhs_norm = sqrt(nk * both[0]);
    if (rhs_norm < 1e-30) rhs_norm = 1.0;
    double rz = nk * both[1];
    double rel = sqrt(rz) / rhs_norm;
    int iter = 0;
    if (rel < A.tol) {
        if (blockIdx.x == 0 && threadIdx.x == 0) { A.scal->ch_iters = 0; A.scal->ch_rel = rel; }
        return;
    }
    double *pcur = A.p1, *pnxt = A.p2;
    double beta = 0.0, alpha = 0.0;
    bool first = true, pending = false;   // pending: x += alpha p_cur still to be applied
    while (iter < A.maxit) {
        // p = z + beta p (z = r); Ap = a_dt p + bih L(L(p))
        double spap = 0.0;
        const double bt = beta, al = alpha;
        const double *pold = pcur;
        for (int q = tid; q < R.n; q += nth) {
            int i, j;
            R.ij(q, i, j);
            const double po = AT_(pold, i, j);
            double pv = po, l;
            if (first) {
                auto p = [&](int a, int b) { return AT_(pold, a, b); };
                l = FLY ? twice(i, j, p) : lap(i, j, p);
            } else {
                pv = AT_(A.r, i, j) + bt * po;
                AT_(pnxt, i, j) = pv;
                AT_(A.x, i, j) += al * po;   // the update of the iteration before
                auto p = [&](int a, int b) { return AT_(A.r, a, b) + bt * AT_(pold, a, b); };
                l = FLY ? twice(i, j, p) : lap(i, j, p);
            }
            if (FLY) {
                const double ap = A.a_dt * pv + A.bih * l;
                AT_(A.Ap, i, j) = ap;
                spap += d.m.wx[i] * d.m.wy[j] * d.wz * pv * ap;
            } else {
                AT_(A.aux, i, j) = l;
            }
        }
        if (!first) { double *t = pcur; pcur = pnxt; pnxt = t; }
        first = false;
        if (!FLY) {
            one[0] = 0.0;
            if (!grid_exchange<1, true>(sl, one)) return;
            for (int q = tid; q < R.n; q += nth) {
                int i, j;
                R.ij(q, i, j);
                const double pv = AT_(pcur, i, j);
                const double ap = A.a_dt * pv + A.bih * lap(i, j, auxf);
                AT_(A.Ap, i, j) = ap;
                spap += d.m.wx[i] * d.m.wy[j] * d.wz * pv * ap;
            }
        }
        // the update reads its own cells' Ap only: the sum alone
        one[0] = spap;
        pending = false;
        if (!grid_exchange<1, false>(sl, one)) return;
        double pAp = nk * one[0];
        if (fabs(pAp) < 1e-30) break;
        alpha = rz / pAp;
        pending = true;
        double srr2 = 0.0;
        for (int q = tid; q < R.n; q += 2 * nth) {   // two cells per trip
            const int q1 = q + nth;
            const bool two = q1 < R.n;
            int i, j, i1 = 0, j1 = 0;
            R.ij(q, i, j);
            const double r0 = AT_(A.r, i, j), a0 = AT_(A.Ap, i, j);
            double r1 = 0.0, a1 = 0.0;
            if (two) {
                R.ij(q1, i1, j1);
                r1 = AT_(A.r, i1, j1); a1 = AT_(A.Ap, i1, j1);
            }
            const double rv = r0 - alpha * a0, rw = r1 - alpha * a1;
            AT_(A.r, i, j) = rv;
            srr2 += d.m.wx[i] * d.m.wy[j] * d.wz * rv * rv;
            if (two) {
                AT_(A.r, i1, j1) = rw;
                srr2 += d.m.wx[i1] * d.m.wy[j1] * d.wz * rw * rw;
            }
        }
        one[0] = srr2;
        if (!grid_exchange<1, true>(sl, one)) return;
        ++iter;
        double rr = nk * one[0];
        rel = sqrt(rr) / rhs_norm;
        if (rel < A.tol) break;
        double rz_new = rr;  // z == r: the same weighted sum
        beta = rz_new / (rz + 1e-30);
        rz = rz_new;
    }
    if (pending)
        for (int q = tid; q < R.n; q += nth) {
            int i, j;
            R.ij(q, i, j);
            AT_(A.x, i, j) += alpha * AT_(pcur, i, j);
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) { A.scal->ch_iters = iter; A.scal->ch_rel = rel; }
}

__global__ void __launch_bounds__(512, 2) k_cg_biharmonic(BihArgs A) { cg_biharmonic<false>(A); }
// one block per SM: at 64 registers (two) it spills, 256x256 75.0 us against 70.9
__global__ void __launch_bounds__(512) k_cg_biharmonic_fly(BihArgs A) { cg_biharmonic<true>(A); }

// ---------------------------------------------------------------------------
// One cell per thread: every value of the solve that belongs to the cell stays
// in the thread's registers, the direction at the four stencil neighbours
// included (each thread advances d = z + beta d at all five points, the same
// operation on the same operands as the owner's), so an iteration moves one
// store of z and four loads of the neighbours' z per cell through L2 and is
// bound by the latency of its two grid-wide sums.  The sum behind the step
// length needs no data of other blocks and skips the fences.  Iterates and
// sums are those of the grid-stride passes, bit for bit.
// ---------------------------------------------------------------------------

// the velocity solve with one cell per thread (B200, 241x482: 13.9 -> 9.2 us
// per iteration)
__global__ void __launch_bounds__(512, 2) k_cg_velocity_res(VelArgs A)
{
    const Dom &d = A.d;
    const int P = d.P, NX = d.NX, NY = d.NY;
    const Range R{A.i0, A.j0, A.i1 - A.i0, (A.i1 - A.i0) * (A.j1 - A.j0)};
    const double EPS = 1e-14;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = q < R.n;
    int i = A.i0, j = A.j0;
    if (on) R.ij(q, i, j);
    const int comp = A.comp;
    Slots sl{reinterpret_cast<unsigned long long *>(A.partials), &A.scal->error, gridDim.x, blockIdx.x, 1, 0};
    double r = 0.0, dg = 1.0, ft = 0.0, x = 0.0, z = 0.0;
    double m0 = 0.0, m1 = 0.0, m2 = 0.0, m3 = 0.0;   // viscosities of the x+, x-, y+, y- faces
    ptrdiff_t off[4];
    double mul[4];
    double v[2];
    v[0] = 0.0;
    if (on) {
        dg = vel_diag(d, comp, A.rho, A.mu, i, j, A.iRe, A.alpha_dt) + EPS;
        const double *__restrict__ mu = A.mu;
        if (comp == 0) {
            ft = 0.5 * (AT_(A.rho, i, j) + AT_(A.rho, i - 1, j)) / A.alpha_dt;
            m0 = AT_(mu, i, j);
            m1 = AT_(mu, i - 1, j);
            m2 = harm(avg2(AT_(mu, i - 1, j + 1), AT_(mu, i, j + 1)), avg2(AT_(mu, i - 1, j), AT_(mu, i, j)));
            m3 = harm(avg2(AT_(mu, i - 1, j), AT_(mu, i, j)), avg2(AT_(mu, i - 1, j - 1), AT_(mu, i, j - 1)));
        } else {
            ft = 0.5 * (AT_(A.rho, i, j) + AT_(A.rho, i, j - 1)) / A.alpha_dt;
            m0 = harm(avg2(AT_(mu, i + 1, j - 1), AT_(mu, i + 1, j)), avg2(AT_(mu, i, j - 1), AT_(mu, i, j)));
            m1 = harm(avg2(AT_(mu, i, j - 1), AT_(mu, i, j)), avg2(AT_(mu, i - 1, j - 1), AT_(mu, i - 1, j)));
            m2 = AT_(mu, i, j);
            m3 = AT_(mu, i, j - 1);
        }
        const double ad = vel_op(d, comp, A.rho, A.mu, i, j, A.iRe, A.alpha_dt, [&](int a, int b) { return AT_(A.x, a, b); });
        x = AT_(A.x, i, j);
        r = AT_(A.rhs, i, j) - ad;
        z = r / dg;
        v[0] = r * z;
        AT_(A.z, i, j) = z;
        const int di[4] = {1, -1, 0, 0}, dj[4] = {0, 0, 1, -1};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            int si, sj;
            src_of(A.mcg, NX, NY, i + di[k], j + dj[k], si, sj, mul[k]);
            if (si < A.i0 || si >= A.i1 || sj < A.j0 || sj >= A.j1) mul[k] = 0.0;
            off[k] = mul[k] == 0.0 ? (ptrdiff_t)j * P + i : (ptrdiff_t)sj * P + si;
        }
    }
    double one[1] = {v[0]};
    if (!grid_exchange<1, true>(sl, one)) return;
    double rz = one[0], RMS = 0.0, beta = 0.0, dc = 0.0, dn[4] = {0.0, 0.0, 0.0, 0.0};
    int iters = 0;
    while (iters < A.maxit) {
        iters++;
        double ad = 0.0;
        one[0] = 0.0;
        if (on) {
            dc = z + beta * dc;
            double f[4];
#pragma unroll
            for (int k = 0; k < 4; k++) dn[k] = __ldcg(A.z + off[k]) + beta * dn[k];
#pragma unroll
            for (int k = 0; k < 4; k++) f[k] = mul[k] == 0.0 ? 0.0 : mul[k] * dn[k];
            // vel_op_w at the cell
            const double Ax = ft * dc;
            double op = 0.0;
            if (comp == 0) {
                const double fxp = m0 * (f[0] - dc) * d.m.idx_u[i], fxm = m1 * (dc - f[1]) * d.m.idx_u[i - 1];
                const double fyp = m2 * (f[2] - dc) * d.m.idy_c[j], fym = m3 * (dc - f[3]) * d.m.idy_c[j - 1];
                op += A.iRe * u_cv_x_div(d, i, fxp, fxm);
                op += A.iRe * (fyp - fym) * d.m.idy_v[j];
                op += axisym_ur_term(d, i, A.iRe * 0.5 * (m0 + m1), dc);
            } else {
                const double fxp = m0 * (f[0] - dc) * d.m.idx_c[i], fxm = m1 * (dc - f[1]) * d.m.idx_c[i - 1];
                const double fyp = m2 * (f[2] - dc) * d.m.idy_v[j], fym = m3 * (dc - f[3]) * d.m.idy_v[j - 1];
                op += A.iRe * v_cv_x_div(d, i, fxp, fxm);
                op += A.iRe * (fyp - fym) * d.m.idy_c[j - 1];
            }
            ad = Ax - op;
            one[0] = dc * ad;
        }
        if (!grid_exchange<1, false>(sl, one)) return;
        const double alpha = rz / (one[0] + A.step_eps);
        v[0] = v[1] = 0.0;
        if (on) {
            x += alpha * dc;
            r = r - alpha * ad;
            z = r / dg;
            AT_(A.z, i, j) = z;
            v[0] = r * r / dg;
            v[1] = r * r;
        }
        if (!grid_exchange<2, true>(sl, v)) return;
        RMS = sqrt(A.in_tot * v[1]);
        if (RMS < A.tol) break;
        beta = v[0] / (rz + A.step_eps);
        rz = v[0];
    }
    if (on) AT_(A.x, i, j) = x;
    if (blockIdx.x == 0 && threadIdx.x == 0) { A.scal->vel_iters[comp] = iters; A.scal->vel_rms[comp] = RMS; }
}

// ---------------------------------------------------------------------------
// Velocity_solve_cg (Eulerian/lsolver/msolve_cg.c:525-722): Jacobi PCG with
// the RMS residual stop, one velocity component.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(512, 2) k_cg_velocity(VelArgs A)
{
    const Dom &d = A.d;
    const int P = d.P, NX = d.NX, NY = d.NY;
    Slots sl{reinterpret_cast<unsigned long long *>(A.partials), &A.scal->error, gridDim.x, blockIdx.x, 1, 0};
    const Range R{A.i0, A.j0, A.i1 - A.i0, (A.i1 - A.i0) * (A.j1 - A.j0)};
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    const double EPS = 1e-14;
    auto active = [&](int a, int b) { return a >= A.i0 && a < A.i1 && b >= A.j0 && b < A.j1; };

    double srz = 0.0;
    for (int q = tid; q < R.n; q += nth) {
        int i, j;
        R.ij(q, i, j);
        double dg = vel_diag(d, A.comp, A.rho, A.mu, i, j, A.iRe, A.alpha_dt) + EPS;
        AT_(A.diag, i, j) = dg;
        vel_weights(d, A.comp, A.rho, A.mu, A.ft, A.mc, i, j, A.i0, A.j0, A.alpha_dt);
        double ad = vel_op(d, A.comp, A.rho, A.mu, i, j, A.iRe, A.alpha_dt, [&](int a, int b) { return AT_(A.x, a, b); });
        double rv = AT_(A.rhs, i, j) - ad;
        AT_(A.r, i, j) = rv;
        double dv = rv / dg;
        AT_(A.dir, i, j) = dv;
        AT_(A.z, i, j) = dv;
        srz += rv * dv;
    }
    double one[1] = {srz}, both[2];
    if (!grid_exchange<1, true>(sl, one)) return;
    double rz = one[0];
    double RMS = 0.0, beta = 0.0;
    int iters = 0;
    double *dcur = A.dir, *dnxt = A.dir2;
    bool first = true;
    double alpha = 0.0;   // the step of the update x += alpha d_cur still to be applied
    while (iters < A.maxit) {
        iters++;
        // d = M^-1 r + beta d, Ad = A d with the VEL_TYPE_CG ghost update of d
        double sdad = 0.0;
        const double bt = beta, al = alpha;
        const double *dold = dcur;
        for (int q = tid; q < R.n; q += nth) {
            int i, j;
            R.ij(q, i, j);
            double dv, ad;
            if (first) {
                dv = AT_(dold, i, j);
                ad = vel_op_w(d, A.comp, A.ft, A.mc, A.mu, i, j, A.iRe, [&](int a, int b) {
                    int si, sj;
                    double mul;
                    src_of(A.mcg, NX, NY, a, b, si, sj, mul);
                    if (mul == 0.0 || !active(si, sj)) return 0.0;
                    return mul * AT_(dold, si, sj);
                });
            } else {
                dv = AT_(A.z, i, j) + bt * AT_(dold, i, j);
                AT_(dnxt, i, j) = dv;
                ad = vel_op_w(d, A.comp, A.ft, A.mc, A.mu, i, j, A.iRe, [&](int a, int b) {
                    int si, sj;
                    double mul;
                    src_of(A.mcg, NX, NY, a, b, si, sj, mul);
                    if (mul == 0.0 || !active(si, sj)) return 0.0;
                    return mul * (AT_(A.z, si, sj) + bt * AT_(dold, si, sj));
                });
            }
            if (!first) AT_(A.x, i, j) += al * AT_(dold, i, j);   // the update of the iteration before
            AT_(A.Ad, i, j) = ad;
            sdad += dv * ad;
        }
        if (!first) { double *t = dcur; dcur = dnxt; dnxt = t; }
        first = false;
        one[0] = sdad;   // the update reads its own cells' Ad only
        if (!grid_exchange<1, false>(sl, one)) return;
        alpha = rz / (one[0] + A.step_eps);
        double s0 = 0.0, s1 = 0.0;
        // two cells per trip, their loads before either's stores
        for (int q = tid; q < R.n; q += 2 * nth) {
            const int q1 = q + nth;
            const bool two = q1 < R.n;
            int i, j, i1 = 0, j1 = 0;
            R.ij(q, i, j);
            const double r0 = AT_(A.r, i, j), a0 = AT_(A.Ad, i, j), g0 = AT_(A.diag, i, j);
            double r1 = 0.0, a1 = 0.0, g1 = 1.0;
            if (two) {
                R.ij(q1, i1, j1);
                r1 = AT_(A.r, i1, j1); a1 = AT_(A.Ad, i1, j1); g1 = AT_(A.diag, i1, j1);
            }
            const double ri = r0 - alpha * a0, rj = r1 - alpha * a1;
            AT_(A.r, i, j) = ri;
            AT_(A.z, i, j) = ri / g0;
            s0 += ri * ri / g0;
            s1 += ri * ri;
            if (two) {
                AT_(A.r, i1, j1) = rj;
                AT_(A.z, i1, j1) = rj / g1;
                s0 += rj * rj / g1;
                s1 += rj * rj;
            }
        }
        both[0] = s0;
        both[1] = s1;
        if (!grid_exchange<2, true>(sl, both)) return;
        double rz_new = both[0], rr = both[1];
        RMS = sqrt(A.in_tot * rr);
        if (RMS < A.tol) break;
        beta = rz_new / (rz + A.step_eps);
        rz = rz_new;
    }
    if (!first)
        for (int q = tid; q < R.n; q += nth) {
            int i, j;
            R.ij(q, i, j);
            AT_(A.x, i, j) += alpha * AT_(dcur, i, j);
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) { A.scal->vel_iters[A.comp] = iters; A.scal->vel_rms[A.comp] = RMS; }
}

// ---------------------------------------------------------------------------
// Pressure_solve_cg (Eulerian/lsolver/psolve_cg.c:130-293): Jacobi PCG on the
// variable-density Poisson operator, absolute stop on sqrt(r.M^-1 r), mean
// removed at the end.
//
// One cell per thread (cg_pressure_resident): ranges of at most one cell per
// resident thread (151 552 cells on a B200), the context's and the
// no-allocation entry point's.  Bound by the latency of the two grid-wide
// sums; per iteration 241x482 12.1 -> 7.7 us, 48x96 7.0 -> 2.4 us.
//
// Larger ranges (cg_pressure): the operator's face weights 2 / (rho_P +
// rho_N) are computed once, in the set-up phase, into the planes A.bx / A.by,
// so an iteration multiplies instead of dividing four times per cell.  The
// pressure ghost rules copy with weight 1 (psolve_cg.c:374-460: Neumann
// copies, periodic wrap) and leave the solve range [0, NX-2] x [0, NY-2]
// unmapped, so a neighbour's source differs from it only at the four ends of
// the axes: those sources are read once from the maps and the stencil is
// gathered without branches.  The update phi += alpha d of an iteration is
// applied in the next iteration's direction pass, which reads d at the cell
// anyway (the same operands and operation, one pass later; before the mean
// removal after the last iteration), so the update pass reads three planes
// instead of five.  Measured per iteration on B200 without the planes and the
// deferred update 31.7 us at 1024x1024 and 154 us at 2048x2048, with them
// 20.8 and 96.6 us; two cells per trip of the direction pass ran 16% slower
// at 2048x2048 (64 registers, loads in flight lost).  PAIR (k_cg_pressure_fwp):
// both passes over pairs of neighbouring cells with 16-byte accesses, for
// ranges of at least two cells per resident thread (the context picks it by
// size): 2048x2048 94.0 -> 86.9 us, 1024x1024 20.7 -> 19.9 us.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cg_pressure_resident(const PresArgs &A, const Range &R)
{
    const Dom &d = A.d;
    const int P = d.P, NX = d.NX, NY = d.NY;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = q < R.n;
    int i = 0, j = 0;
    if (on) R.ij(q, i, j);
    Slots sl{reinterpret_cast<unsigned long long *>(A.partials), &A.scal->error, gridDim.x, blockIdx.x, 1, 0};
    double r = 0.0, m = 0.0, z = 0.0, ph = 0.0, rw = 1.0;
    double cxm = 0.0, cxp = 0.0, cym = 0.0, cyp = 0.0;
    const ptrdiff_t cC = (ptrdiff_t)j * P + i;
    ptrdiff_t cE = cC, cW = cC, cN = cC, cS = cC;
    double s[1] = {0.0};
    if (on) {
        // sources of the neighbours under the pressure ghost rules
        cW = (ptrdiff_t)j * P + (i > 0 ? i - 1 : A.mp.x.src[NG - 1]);
        cE = (ptrdiff_t)j * P + (i < NX - 2 ? i + 1 : A.mp.x.src[NX - 1 + NG]);
        cS = (ptrdiff_t)(j > 0 ? j - 1 : A.mp.y.src[NG - 1]) * P + i;
        cN = (ptrdiff_t)(j < NY - 2 ? j + 1 : A.mp.y.src[NY - 1 + NG]) * P + i;
        const double *__restrict__ rho = A.rho;
        const double r0 = rho[cC];
        const double bxp = 2.0 / (r0 + rho[cC + 1]), bxm = 2.0 / (r0 + rho[cC - 1]);
        const double byp = 2.0 / (r0 + rho[cC + P]), bym = 2.0 / (r0 + rho[cC - P]);
        face_coeffs(d, i, bxm, bxp, bym, byp, cxm, cxp, cym, cyp);
        rw = row_weight(d, i);
        const double ad = pressure_op(d, rho, i, j, [&](int a, int b) { return remap(A.mp, A.phi, P, NX, NY, a, b); });
        // the axisymmetric right-hand side carries the row weight r_c of the
        // operator (psolve_hypre.c:184-200)
        r = (d.axisym ? A.rhs[cC] * d.m.r_c[i] : A.rhs[cC]) - ad;
        m = A.M[cC];
        ph = A.phi[cC];
        z = r * m;
        A.z[cC] = z;
        s[0] = r * z;
    }
    if (!grid_exchange<1, true>(sl, s)) return;
    double gamma = s[0], gamma_new = 0.0, beta = 0.0;
    if (sqrt(gamma) < A.tol) {
        if (blockIdx.x == 0 && threadIdx.x == 0) { A.scal->p_iters = 0; A.scal->p_res = sqrt(gamma); }
        return;
    }
    double dc = 0.0, dE = 0.0, dW = 0.0, dN = 0.0, dS = 0.0;
    int iters;
    for (iters = 1; iters <= A.maxit; iters++) {
        double ad = 0.0;
        s[0] = 0.0;
        if (on) {
            const double zE = __ldcg(A.z + cE), zW = __ldcg(A.z + cW), zN = __ldcg(A.z + cN), zS = __ldcg(A.z + cS);
            dc = z + beta * dc;
            dE = zE + beta * dE;
            dW = zW + beta * dW;
            dN = zN + beta * dN;
            dS = zS + beta * dS;
            const double val = cxp * (dE - dc) - cxm * (dc - dW) + cyp * (dN - dc) - cym * (dc - dS);
            ad = rw * val;
            s[0] = dc * ad;
        }
        if (!grid_exchange<1, false>(sl, s)) return;
        const double alpha = gamma / (s[0] + 1e-30);
        s[0] = 0.0;
        if (on) {
            r = r - alpha * ad;
            z = r * m;
            A.z[cC] = z;
            ph += alpha * dc;
            s[0] = r * z;
        }
        if (!grid_exchange<1, true>(sl, s)) return;
        gamma_new = s[0];
        if (sqrt(gamma_new) < A.tol) break;
        beta = gamma_new / (gamma + 1e-30);
        gamma = gamma_new;
    }
    // remove the mean (every face Neumann or periodic), psolve_cg.c:255-279
    s[0] = on ? ph : 0.0;
    if (!grid_exchange<1, false>(sl, s)) return;
    if (on) A.phi[cC] = ph - s[0] / (double)R.n;
    if (iters > A.maxit) iters = A.maxit;
    if (blockIdx.x == 0 && threadIdx.x == 0) { A.scal->p_iters = iters; A.scal->p_res = sqrt(gamma_new); }
}

// WEIGHTS: the face weights come from the planes A.bx / A.by, filled by the
// set-up phase; otherwise each is computed where it is needed (the no-allocation
// entry point on a device too small for a cell per thread: its scratch has no
// room for them).
template <bool PAIR, bool WEIGHTS>
__device__ __forceinline__ void cg_pressure(const PresArgs &A)
{
    const Dom &d = A.d;
    const int P = d.P, NX = d.NX, NY = d.NY;
    const Range R{0, 0, NX - 1, (NX - 1) * (NY - 1)};
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    // sources of the neighbours beyond the ends of the solve range
    const int xw = A.mp.x.src[NG - 1], xe = A.mp.x.src[NX - 1 + NG];
    const int ys = A.mp.y.src[NG - 1], yn = A.mp.y.src[NY - 1 + NG];
    const double *__restrict__ rho = A.rho;
    const double *__restrict__ bx = A.bx;
    const double *__restrict__ by = A.by;
    Slots sl{reinterpret_cast<unsigned long long *>(A.partials), &A.scal->error, gridDim.x, blockIdx.x, 1, 0};
    if (!PAIR && WEIGHTS && R.n <= nth) {   // one cell per thread
        cg_pressure_resident(A, R);
        return;
    }

    double sg = 0.0;
    for (int q = tid; q < R.n; q += nth) {
        int i, j;
        R.ij(q, i, j);
        if (WEIGHTS) pressure_face_weights(d, rho, A.bx, A.by, i, j);
        double ad = pressure_op(d, rho, i, j, [&](int a, int b) { return remap(A.mp, A.phi, P, NX, NY, a, b); });
        // the axisymmetric right-hand side carries the row weight r_c of the
        // operator (psolve_hypre.c:184-200)
        double rv = (d.axisym ? AT_(A.rhs, i, j) * d.m.r_c[i] : AT_(A.rhs, i, j)) - ad;
        AT_(A.res, i, j) = rv;
        double z = rv * AT_(A.M, i, j);
        AT_(A.dir, i, j) = z;
        AT_(A.z, i, j) = z;
        sg += rv * z;
    }
    double one[1] = {sg};
    if (!grid_exchange<1, true>(sl, one)) return;
    double gamma = one[0], gamma_new = 0.0, beta = 0.0;
    if (sqrt(gamma) < A.tol) {
        if (blockIdx.x == 0 && threadIdx.x == 0) { A.scal->p_iters = 0; A.scal->p_res = sqrt(gamma); }
        return;
    }

    // d = z + beta d_old at the five points of cell q (d_old alone on the
    // first iteration) and A d at the cell
    auto direction = [&](int q, bool first, const double *__restrict__ zp, const double *__restrict__ dold, double bt,
                         double &dv, double &ad) {
        int i, j;
        R.ij(q, i, j);
        const int iw = i > 0 ? i - 1 : xw, ie = i < NX - 2 ? i + 1 : xe;
        const int js = j > 0 ? j - 1 : ys, jn = j < NY - 2 ? j + 1 : yn;
        const ptrdiff_t row = (ptrdiff_t)j * P;
        const ptrdiff_t cC = row + i, cE = row + ie, cW = row + iw;
        const ptrdiff_t cN = (ptrdiff_t)jn * P + i, cS = (ptrdiff_t)js * P + i;
        double vc, ve, vw, vn, vs;
        if (first) {
            vc = dold[cC]; ve = dold[cE]; vw = dold[cW]; vn = dold[cN]; vs = dold[cS];
        } else {
            vc = zp[cC] + bt * dold[cC];
            ve = zp[cE] + bt * dold[cE];
            vw = zp[cW] + bt * dold[cW];
            vn = zp[cN] + bt * dold[cN];
            vs = zp[cS] + bt * dold[cS];
        }
        double bxm, bxp, bym, byp;
        if (WEIGHTS) {
            bxm = bx[cC - 1]; bxp = bx[cC]; bym = by[cC - P]; byp = by[cC];
        } else {
            const double r0 = rho[cC];
            bxm = 2.0 / (r0 + rho[cC - 1]); bxp = 2.0 / (r0 + rho[cC + 1]);
            bym = 2.0 / (r0 + rho[cC - P]); byp = 2.0 / (r0 + rho[cC + P]);
        }
        double cxm, cxp, cym, cyp;
        face_coeffs(d, i, bxm, bxp, bym, byp, cxm, cxp, cym, cyp);
        const double val = cxp * (ve - vc) - cxm * (vc - vw) + cyp * (vn - vc) - cym * (vc - vs);
        dv = vc;
        ad = row_weight(d, i) * val;
    };

    // PAIR: the two passes over pairs of cells (2k, 2k+1) of a row with
    // 16-byte loads and stores (the planes' rows start on 16-byte boundaries
    // and i = 0 sits at an even column); a row of odd length ends in a single
    // cell, whose stores are 8 bytes wide.  The values are those of the
    // single-cell passes: the same operands in the same operations.
    const int W = NX - 1, Wp = (W + 1) / 2, Np = Wp * (NY - 1);
    auto ld2 = [](const double *p) { return *reinterpret_cast<const double2 *>(p); };
    auto st2 = [](double *p, double a, double b) { *reinterpret_cast<double2 *>(p) = make_double2(a, b); };
    auto direction_pair = [&](int p, bool first, const double *__restrict__ zp, const double *__restrict__ dold,
                              double *__restrict__ dn, double bt, double al, double &sdad) {
        const int j = p / Wp, i0 = 2 * (p - j * Wp), i1 = i0 + 1;
        const bool has1 = i1 < W;
        const int iw = i0 > 0 ? i0 - 1 : xw, ie = i0 + 2 <= NX - 2 ? i0 + 2 : xe;
        const int js = j > 0 ? j - 1 : ys, jn = j < NY - 2 ? j + 1 : yn;
        const ptrdiff_t r = (ptrdiff_t)j * P + i0, rn = (ptrdiff_t)jn * P + i0, rs = (ptrdiff_t)js * P + i0;
        const ptrdiff_t rw = (ptrdiff_t)j * P + iw, re = (ptrdiff_t)j * P + ie;
        const double2 oc = ld2(dold + r), on = ld2(dold + rn), os = ld2(dold + rs);
        const double ow = dold[rw], oe = dold[re];
        double2 vc = oc, vn = on, vs = os;
        double vw = ow, ve = oe;
        if (!first) {
            const double2 zc = ld2(zp + r), zn = ld2(zp + rn), zs = ld2(zp + rs);
            const double zw = zp[rw], ze = zp[re];
            vc = make_double2(zc.x + bt * oc.x, zc.y + bt * oc.y);
            vn = make_double2(zn.x + bt * on.x, zn.y + bt * on.y);
            vs = make_double2(zs.x + bt * os.x, zs.y + bt * os.y);
            vw = zw + bt * ow;
            ve = ze + bt * oe;
        }
        const double2 bxc = ld2(bx + r), byc = ld2(by + r), bys = ld2(by + r - P);
        const double bxw = bx[r - 1];
        double cxm, cxp, cym, cyp;
        face_coeffs(d, i0, bxw, bxc.x, bys.x, byc.x, cxm, cxp, cym, cyp);
        const double e0 = has1 ? vc.y : ve;
        const double ad0 = row_weight(d, i0) *
                           (cxp * (e0 - vc.x) - cxm * (vc.x - vw) + cyp * (vn.x - vc.x) - cym * (vc.x - vs.x));
        face_coeffs(d, i1, bxc.x, bxc.y, bys.y, byc.y, cxm, cxp, cym, cyp);
        const double ad1 = row_weight(d, i1) *
                           (cxp * (ve - vc.y) - cxm * (vc.y - vc.x) + cyp * (vn.y - vc.y) - cym * (vc.y - vs.y));
        if (has1) {
            if (!first) {
                const double2 ph = ld2(A.phi + r);
                st2(A.phi + r, ph.x + al * oc.x, ph.y + al * oc.y);
            }
            if (!first) st2(dn + r, vc.x, vc.y);
            st2(A.Ad + r, ad0, ad1);
            sdad += vc.x * ad0;
            sdad += vc.y * ad1;
        } else {
            if (!first) A.phi[r] = A.phi[r] + al * oc.x;
            if (!first) dn[r] = vc.x;
            A.Ad[r] = ad0;
            sdad += vc.x * ad0;
        }
    };
    auto update_pair = [&](int p, double alpha, double &sgn) {
        const int j = p / Wp, i0 = 2 * (p - j * Wp);
        const bool has1 = i0 + 1 < W;
        const ptrdiff_t r = (ptrdiff_t)j * P + i0;
        const double2 rr = ld2(A.res + r), aa = ld2(A.Ad + r), mm = ld2(A.M + r);
        const double rv0 = rr.x - alpha * aa.x, z0 = rv0 * mm.x;
        const double rv1 = rr.y - alpha * aa.y, z1 = rv1 * mm.y;
        if (has1) {
            st2(A.res + r, rv0, rv1);
            st2(A.z + r, z0, z1);
            sgn += rv0 * z0;
            sgn += rv1 * z1;
        } else {
            A.res[r] = rv0;
            A.z[r] = z0;
            sgn += rv0 * z0;
        }
    };

    double *dcur = A.dir, *dnxt = A.dir2;
    bool first = true;
    double alpha = 0.0;   // the step of the update phi += alpha d_cur still to be applied
    int iters;
    for (iters = 1; iters <= A.maxit; iters++) {
        // d = z + beta d (z = M r), Ad with the pressure ghost update of d;
        // phi += alpha d_old from the previous iteration at the cell
        double sdad = 0.0;
        const double bt = beta, al = alpha;
        const double *dold = dcur;
        if (PAIR)
            for (int p = tid; p < Np; p += nth) direction_pair(p, first, A.z, dold, dnxt, bt, al, sdad);
        else
        for (int q = tid; q < R.n; q += nth) {
            double dv, ad;
            direction(q, first, A.z, dold, bt, dv, ad);
            int i, j;
            R.ij(q, i, j);
            double ph0 = 0.0, do0 = 0.0;
            if (!first) { ph0 = AT_(A.phi, i, j); do0 = AT_(dold, i, j); }
            if (!first) AT_(dnxt, i, j) = dv;
            AT_(A.Ad, i, j) = ad;
            if (!first) AT_(A.phi, i, j) = ph0 + al * do0;
            sdad += dv * ad;
        }
        if (!first) { double *t = dcur; dcur = dnxt; dnxt = t; }
        first = false;
        one[0] = sdad;   // the update reads its own cells' Ad only
        if (!grid_exchange<1, false>(sl, one)) return;
        alpha = gamma / (one[0] + 1e-30);
        double sgn = 0.0;
        if (PAIR)
            for (int p = tid; p < Np; p += nth) update_pair(p, alpha, sgn);
        else
        for (int q = tid; q < R.n; q += 2 * nth) {
            const int q1 = q + nth;
            const bool two = q1 < R.n;
            int i0, j0, i1 = 0, j1 = 0;
            R.ij(q, i0, j0);
            double r0 = AT_(A.res, i0, j0), a0 = AT_(A.Ad, i0, j0), m0 = AT_(A.M, i0, j0);
            double r1 = 0.0, a1 = 0.0, m1 = 0.0;
            if (two) {
                R.ij(q1, i1, j1);
                r1 = AT_(A.res, i1, j1); a1 = AT_(A.Ad, i1, j1); m1 = AT_(A.M, i1, j1);
            }
            {
                const double rv = r0 - alpha * a0, z = rv * m0;
                AT_(A.res, i0, j0) = rv;
                AT_(A.z, i0, j0) = z;
                sgn += rv * z;
            }
            if (two) {
                const double rv = r1 - alpha * a1, z = rv * m1;
                AT_(A.res, i1, j1) = rv;
                AT_(A.z, i1, j1) = z;
                sgn += rv * z;
            }
        }
        one[0] = sgn;
        if (!grid_exchange<1, true>(sl, one)) return;
        gamma_new = one[0];
        if (sqrt(gamma_new) < A.tol) break;
        beta = gamma_new / (gamma + 1e-30);
        gamma = gamma_new;
    }
    // remove the mean (every face Neumann or periodic), psolve_cg.c:255-279,
    // after the last iteration's pending update
    double ssum = 0.0;
    const bool pending = !first;
    for (int q = tid; q < R.n; q += nth) {
        int i, j;
        R.ij(q, i, j);
        if (pending) AT_(A.phi, i, j) += alpha * AT_(dcur, i, j);
        ssum += AT_(A.phi, i, j);
    }
    one[0] = ssum;
    if (!grid_exchange<1, false>(sl, one)) return;
    double avg = one[0] / (double)R.n;
    for (int q = tid; q < R.n; q += nth) {
        int i, j;
        R.ij(q, i, j);
        AT_(A.phi, i, j) -= avg;
    }
    if (iters > A.maxit) iters = A.maxit;
    if (blockIdx.x == 0 && threadIdx.x == 0) { A.scal->p_iters = iters; A.scal->p_res = sqrt(gamma_new); }
}

// the no-allocation entry point's solve: at most one cell per resident thread, or
// a walk of the range where the device holds fewer threads
__global__ void __launch_bounds__(512) k_cg_pressure(PresArgs A)
{
    cg_pressure_resident(A, Range{0, 0, A.d.NX - 1, (A.d.NX - 1) * (A.d.NY - 1)});
}
__global__ void __launch_bounds__(512) k_cg_pressure_walk(PresArgs A) { cg_pressure<false, false>(A); }
__global__ void __launch_bounds__(512, 2) k_cg_pressure_fw(PresArgs A) { cg_pressure<false, true>(A); }
__global__ void __launch_bounds__(512, 2) k_cg_pressure_fwp(PresArgs A) { cg_pressure<true, true>(A); }

}  // namespace pvof
