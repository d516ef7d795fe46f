// k_cg_coop.cuh — the plain FP64 CG as one cooperative launch (included by k_fp64.cu).
//
// The two-kernel iteration (k_cg_spmv*, k_cg_update) costs two launches, two ramps and two
// last-block reductions, whatever the grid: about 17-20 us on grids whose data the L2 holds and
// whose arithmetic takes 1-2 us.  Here every CTA stays resident for the whole solve, and an iteration's
// grid-wide sums, one (k_cg_one) or two (p.q and r.r), are also the barriers that publish its vectors.
#pragma once
#include "k_coop.cuh"

namespace suli {

// the scalars of the solve, the same in every thread
struct CoopCG {
    double rr, rr_start, alpha, beta, pq;
    int iters, done, status;
    // after p.q
    __device__ __forceinline__ void dot(double t) {
        rr_start = rr;
        pq = t;
        alpha = rr / t;
        if (!isfinite(alpha)) { status = SULI_ERR_NAN; done = 1; }
    }
    // after r.r: beta and the stopping test of k_cg_update
    __device__ __forceinline__ void residual(double t, int mode, double thr, int maxit) {
        beta = t / rr;
        rr = t;
        iters += 1;
        bool go = (mode == 0) ? fabs(rr_start) > thr : t > thr;
        if (iters >= maxit) { go = false; status = SULI_WARN_CG_MAXIT; }
        if (!isfinite(t)) { go = false; status = SULI_ERR_NAN; }
        done = go ? 0 : 1;
    }
};
__device__ __forceinline__ CoopCG coop_load(const CGState* st) {
    return CoopCG{st->rr, st->rr_start, st->alpha, st->beta, st->pq, st->iters, st->done, st->status};
}
// the end of a CTA's part of the solve: its failure, and from CTA 0 the state
__device__ __forceinline__ void coop_store(const CoopCG& s, bool failed, CGState* st) {
    if (threadIdx.x != 0) return;
    if (failed) st->gave_up = 1;
    if (blockIdx.x != 0) return;
    st->rr = s.rr; st->rr_start = s.rr_start; st->alpha = s.alpha; st->beta = s.beta; st->pq = s.pq;
    st->iters = s.iters;
    st->done = 1;
    st->status = failed ? SULI_ERR_CUDA : s.status;
}

// Small grids: a thread owns U cells for the whole solve and keeps everything but r in
// registers: the cell's e, r, p, q, its six coefficients, and p at its six neighbours, which it
// advances itself (p_nb = r_nb + beta p_nb, the owner's expression), so an iteration loads only r
// at the neighbours and stores only r.  The directions end in cg_pa (resumed solves read it).
// Cells are numbered along x, so the loads of a warp run along rows.  Bound by the latencies of
// its two sums and of the neighbours' loads (25x50x45: 6.1 us an iteration, 19.7 with two kernels).
template <int U, int NT>
__device__ __forceinline__ void cg_reg(const Geo& G, const BC& bc, double* r, double* pa, double* e,
                                       const double* __restrict__ ax, const double* __restrict__ ay,
                                       const double* __restrict__ az, CGState* st, double* work, int polls, double* sh) {
    CoopCG s = coop_load(st);
    const double thr = st->thr;
    const int mode = st->mode, maxit = st->maxit;
    CoopGrid S(work, sh, polls);
    const int px = G.px, pxy = (int)G.pxy;
    const int total = G.nx * G.ny * G.nz, step = gridDim.x * NT;
    int c[U], nb[U][6];
    double a[U][6], pn[U][6], p[U], rc[U], ec[U], q[U];
    const bool fresh = (s.iters == 0);
    if (fresh) s.beta = 0.;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int id = blockIdx.x * NT + threadIdx.x + u * step;
        c[u] = -1;
        p[u] = rc[u] = ec[u] = q[u] = 0.;
#pragma unroll
        for (int m = 0; m < 6; ++m) { a[u][m] = 0.; pn[u][m] = 0.; nb[u][m] = 0; }
        if (id < total) {
            const int i = id % G.nx + 1, j = (id / G.nx) % G.ny + 1, k = id / (G.nx * G.ny) + 1;
            const int cc = G.idx32(i, j, k);
            const Nb o = neighbours(G, bc, i, j, k);
            c[u] = cc;
            nb[u][0] = cc + o.xp; nb[u][1] = cc + o.xm; nb[u][2] = cc + o.yp;
            nb[u][3] = cc + o.ym; nb[u][4] = cc + o.zp; nb[u][5] = cc + o.zm;
            a[u][0] = ax[cc + 1]; a[u][1] = ax[cc]; a[u][2] = ay[cc + px];
            a[u][3] = ay[cc]; a[u][4] = az[cc + pxy]; a[u][5] = az[cc];
            rc[u] = r[cc];
            ec[u] = e[cc];
            if (!fresh) {
                p[u] = pa[cc];
#pragma unroll
                for (int m = 0; m < 6; ++m) pn[u][m] = pa[nb[u][m]];
            }
        }
    }
    while (!s.done && !S.failed) {
        double rn[U][6];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c[u] >= 0) {
#pragma unroll
                for (int m = 0; m < 6; ++m) rn[u][m] = __ldcg(r + nb[u][m]);
            }
        double dot = 0.;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c[u] >= 0) {
                p[u] = rc[u] + s.beta * p[u];
#pragma unroll
                for (int m = 0; m < 6; ++m) pn[u][m] = rn[u][m] + s.beta * pn[u][m];
                q[u] = p[u] - pn[u][0] * a[u][0] - pn[u][1] * a[u][1] - pn[u][2] * a[u][2] - pn[u][3] * a[u][3] -
                       pn[u][4] * a[u][4] - pn[u][5] * a[u][5];
                dot += p[u] * q[u];
            }
        s.dot(coop_sum(S, dot));
        if (s.done || S.failed) break;
        double rr = 0.;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c[u] >= 0) {
                ec[u] = ec[u] - s.alpha * p[u];
                rc[u] = rc[u] - s.alpha * q[u];
                __stcg(r + c[u], rc[u]);
                rr += rc[u] * rc[u];
            }
        s.residual(coop_sum(S, rr), mode, thr, maxit);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (c[u] >= 0) {
            e[c[u]] = ec[u];
            pa[c[u]] = p[u];
        }
    coop_store(s, S.failed, st);
}
template <int U, int NT>
__global__ void __launch_bounds__(NT, 1) k_cg_reg(Geo G, BC bc, double* r, double* pa, double* e,
                                                  const double* __restrict__ ax, const double* __restrict__ ay,
                                                  const double* __restrict__ az, CGState* st, double* work, int polls) {
    __shared__ double sh[kCoopShared];
    if (st->done) return;
    cg_reg<U, NT>(G, bc, r, pa, e, ax, ay, az, st, work, polls, sh);
}

// Small grids whose operator is symmetric: the same iteration in Chronopoulos and Gear's form
// (J. Comput. Appl. Math. 25, 1989), which needs one grid-wide sum: with w = A~ r,
//   s = w + beta s (= A~ p),  alpha = r.r / (r.w - beta r.r / alpha_old),
// r.r and r.w come from one sum after the updates.  A thread keeps e, r, p, s and w of its U cells
// and r and s at their six neighbours, which it advances itself (the owner's expressions), so an
// iteration loads only w at the neighbours and stores only w, in two arrays in turn (a CTA may be
// one sum ahead).  e, p and the coefficients sit in shared memory, the rest in registers.
// In exact arithmetic the iterates are k_cg_reg's.  An asymmetric operator (a periodic axis with the
// reference's clamped end faces, 8_derivadas.f90:318-323, when the density varies across it) makes p.A~p
// another number, so those solves keep k_cg_reg.  So does a system without a solution: every
// boundary is a Neumann one, the null vector of A~ is sqrt(d), and the part of r along it
// (CGState.null2, its square) stays in r for good.  Once r is little more than that part, p.A~p is
// the small difference of two large terms and can come out negative: a channel with an unbalanced
// outflow took up to ten times the iterations and left three to ten times the divergence of the two-sum
// form.  Restated on the CPU (density ratio 833, tolerances 1e-4 to 1e-18, warm and cold starts),
// the two forms agree in iterations and in the true residual wherever null2 <= 1e-2 thr, and part from
// 1e-1 thr on; kNullPart leaves a factor of ten.  A balanced system has null2 of rounding, about
// 1e-38 b~.b~.
// A resumed solve reads p and s, which end in cg_pa and cg_q; one whose threshold the divergence test
// lowered past the rule goes on in the two-sum form from r, e and p.
// Bound by the latency of its one sum, whose last part the neighbours' loads overlap: 3.4 us an
// iteration at 25x50x45 where k_cg_reg takes 6.1, 3.7 at 64x32x48 against 6.7.
constexpr double kNullPart = 1e-3;
template <int U, int NT>
__global__ void __launch_bounds__(NT, 1) k_cg_one(Geo G, BC bc, double* r, double* pa, double* wa, double* wb, double* e,
                                                  const double* __restrict__ ax, const double* __restrict__ ay,
                                                  const double* __restrict__ az, CGState* st, double* work, int polls) {
    extern __shared__ double cells[];   // [8 U][NT]: six coefficients, e, p
    __shared__ double sh[kCoopShared];
    if (st->done) return;
    const double thr = st->thr;
    if (!(st->null2 <= kNullPart * thr)) {   // the same for every CTA
        cg_reg<U, NT>(G, bc, r, pa, e, ax, ay, az, st, work, polls, sh);
        return;
    }
    CoopCG t = coop_load(st);
    const int mode = st->mode, maxit = st->maxit;
    CoopGrid S(work, sh, polls);
    const int px = G.px, pxy = (int)G.pxy;
    const int total = G.nx * G.ny * G.nz, step = gridDim.x * NT;
    const bool fresh = (t.iters == 0);
    int c[U], nb[U][6];
    double rn[U][6], sn[U][6], rc[U], sc[U], wc[U];
    double* own = cells + threadIdx.x;   // value v of cell u: own[(8 u + v) NT]
    double dot = 0.;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int id = blockIdx.x * NT + threadIdx.x + u * step;
        c[u] = -1;
        rc[u] = sc[u] = wc[u] = 0.;
#pragma unroll
        for (int m = 0; m < 6; ++m) { nb[u][m] = 0; rn[u][m] = sn[u][m] = 0.; }
        if (id < total) {
            const int i = id % G.nx + 1, j = (id / G.nx) % G.ny + 1, k = id / (G.nx * G.ny) + 1;
            const int cc = G.idx32(i, j, k);
            const Nb o = neighbours(G, bc, i, j, k);
            c[u] = cc;
            nb[u][0] = cc + o.xp; nb[u][1] = cc + o.xm; nb[u][2] = cc + o.yp;
            nb[u][3] = cc + o.ym; nb[u][4] = cc + o.zp; nb[u][5] = cc + o.zm;
            const double a[6] = {ax[cc + 1], ax[cc], ay[cc + px], ay[cc], az[cc + pxy], az[cc]};
            rc[u] = r[cc];
            double q = rc[u];
#pragma unroll
            for (int m = 0; m < 6; ++m) {
                own[(8 * u + m) * NT] = a[m];
                rn[u][m] = r[nb[u][m]];
                q = q - rn[u][m] * a[m];
                if (!fresh) sn[u][m] = wa[nb[u][m]];
            }
            if (!fresh) sc[u] = wa[cc];
            own[(8 * u + 6) * NT] = e[cc];
            own[(8 * u + 7) * NT] = fresh ? 0. : pa[cc];
            wc[u] = q;
            dot += rc[u] * q;
        }
    }
    // w goes to cg_pb first: other CTAs may still read s of a resumed solve in cg_q
    double *w = wb, *wnext = wa;
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (c[u] >= 0) __stcg(w + c[u], wc[u]);
    double alpha_old = t.alpha;
    bool first = true;
    coop_begin(S, 0., dot);
    for (;;) {
        double wn[U][6];   // in flight while the partials are added
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c[u] >= 0) {
#pragma unroll
                for (int m = 0; m < 6; ++m) wn[u][m] = __ldcg(w + nb[u][m]);
            }
        const double2 d = coop_end(S);
        if (S.failed) break;
        if (!first) t.residual(d.x, mode, thr, maxit);
        else if (fresh) t.beta = 0.;
        first = false;
        if (t.done) break;
        t.rr_start = t.rr;
        t.pq = (t.iters == 0) ? d.y : d.y - t.beta * t.rr / alpha_old;   // p.A~p
        t.alpha = t.rr / t.pq;
        if (!isfinite(t.alpha)) { t.status = SULI_ERR_NAN; break; }
        const double alpha = t.alpha, beta = t.beta;
        double rr = 0., rw = 0.;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c[u] >= 0) {
                const double p = rc[u] + beta * own[(8 * u + 7) * NT];
                own[(8 * u + 7) * NT] = p;
                own[(8 * u + 6) * NT] = own[(8 * u + 6) * NT] - alpha * p;
                sc[u] = wc[u] + beta * sc[u];
                rc[u] = rc[u] - alpha * sc[u];
                double q = rc[u];
#pragma unroll
                for (int m = 0; m < 6; ++m) {
                    sn[u][m] = wn[u][m] + beta * sn[u][m];
                    rn[u][m] = rn[u][m] - alpha * sn[u][m];
                    q = q - rn[u][m] * own[(8 * u + m) * NT];
                }
                wc[u] = q;
                __stcg(wnext + c[u], q);
                rr += rc[u] * rc[u];
                rw += rc[u] * q;
            }
        alpha_old = alpha;
        double* x = w;
        w = wnext;
        wnext = x;
        coop_begin(S, rr, rw);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (c[u] >= 0) {
            r[c[u]] = rc[u];
            e[c[u]] = own[(8 * u + 6) * NT];
            pa[c[u]] = own[(8 * u + 7) * NT];
            wa[c[u]] = sc[u];
        }
    coop_store(t, S.failed, st);
}

// Larger grids: the iteration's two passes over units dealt to the threads in turn (a unit is a
// pair of x cells, 16-byte loads, and a column of KZ planes).  Every other iteration the first pass
// also applies the last two iterations' e -= alpha p (it reads the newer p anyway, and the older
// where it writes its own), so the second only forms r; it takes the units in reverse order,
// newest in the L2 first.  Iteration n (from 1) writes its direction into pa for odd n, pb for even
// n.  Bound by the loads a thread's 64 registers keep in flight: 11.5 passes in 78 us at
// 256x128x128 (the two kernels' 13 in 110), the first pass 8.5 in 60 us, 4.7 TB/s, the second 3 in 18
// us, 5.6 TB/s.  Measured there with e updated in every iteration (83.4 us): 512 threads of the same
// 87.7-97, 4 planes a unit 96, 8 planes 105, 1 plane 89.
template <int KZ, int NT>
__global__ void __launch_bounds__(NT, 1) k_cg_two(Geo G, BC bc, double* r, double* pa, double* pb, double* q, double* e,
                                                  const double* __restrict__ ax, const double* __restrict__ ay,
                                                  const double* __restrict__ az, CGState* st, double* work, int polls) {
    __shared__ double sh[kCoopShared];
    CoopCG s = coop_load(st);
    if (s.done) return;
    const double thr = st->thr;
    const int mode = st->mode, maxit = st->maxit;
    CoopGrid S(work, sh, polls);
    const int nx = G.nx, ny = G.ny, nz = G.nz, px = G.px, pxy = (int)G.pxy;
    const int ux = (nx + 1) / 2, uxy = ux * ny, units = uxy * ((nz + KZ - 1) / KZ);
    const int first = blockIdx.x * NT + threadIdx.x, step = gridDim.x * NT;
    const int last = first < units ? first + (units - 1 - first) / step * step : -1;
    if (s.iters == 0) s.beta = 0.;
    auto lg2 = [](const double* a) { return __ldcg(reinterpret_cast<const double2*>(a)); };
    auto ld2 = [](const double* a) { return *reinterpret_cast<const double2*>(a); };
    // nx odd: the last pair of a row holds one cell
    auto put = [](double* a, double2 v, bool two) {
        if (two) __stcg(reinterpret_cast<double2*>(a), v);
        else __stcg(a, v.x);
    };
    int pending = 0;          // iterations whose update e lacks, the older with step alpha_old
    double alpha_old = 0.;
    while (!s.done && !S.failed) {
        double* pn_ = (s.iters & 1) ? pb : pa;                                   // iteration s.iters + 1
        const double* po = (s.iters == 0) ? r : ((s.iters & 1) ? pa : pb);
        const double beta = s.beta, alpha0 = s.alpha;
        double dot = 0.;
        for (int u = first; u < units; u += step) {
            const int kz = u / uxy, rem = u - kz * uxy, jj = rem / ux, j = jj + 1, i0 = 2 * (rem - jj * ux) + 1, k0 = kz * KZ + 1;
            const bool two = i0 < nx;
            const int lastx = two ? 1 : 0;                                         // the pair's last cell
            const int oxm = (i0 > 1) ? -1 : (bc.perx ? nx - 1 : 0);
            const int oxp = lastx + ((i0 + lastx < nx) ? 1 : (bc.perx ? -(nx - 1) : 0));
            const int oym = (j > 1) ? -px : (bc.pery ? (ny - 1) * px : 0);
            const int oyp = (j < ny) ? px : (bc.pery ? -(ny - 1) * px : 0);
            const int c0 = kBase + (i0 - 1) + px * j;
            auto pn2 = [&](int c) {
                const double2 a = lg2(r + c), b = lg2(po + c);
                return make_double2(a.x + beta * b.x, a.y + beta * b.y);
            };
            double2 col[KZ + 2];
#pragma unroll
            for (int m = 0; m < KZ + 2; ++m) col[m] = pn2(c0 + pxy * map_any(k0 - 1 + m, nz, bc.perz));
#pragma unroll
            for (int m = 0; m < KZ; ++m) {
                const int k = k0 + m;
                if (k > nz) break;
                const int c = c0 + pxy * k;
                const double pxm = __ldcg(r + c + oxm) + beta * __ldcg(po + c + oxm);
                const double pxp = __ldcg(r + c + oxp) + beta * __ldcg(po + c + oxp);
                const double2 pym = pn2(c + oym), pyp = pn2(c + oyp);
                const double2 pc = col[m + 1], pzm = col[m], pzp = col[m + 2];
                const double2 axc = ld2(ax + c), ayc = ld2(ay + c), ayp = ld2(ay + c + px), azc = ld2(az + c),
                              azp = ld2(az + c + pxy);
                const double ax2 = ax[c + 2];
                const double q0 = pc.x - (two ? pc.y : pxp) * axc.y - pxm * axc.x - pyp.x * ayp.x - pym.x * ayc.x -
                                  pzp.x * azp.x - pzm.x * azc.x;
                const double q1 = pc.y - pxp * ax2 - pc.x * axc.y - pyp.y * ayp.y - pym.y * ayc.y - pzp.y * azp.y -
                                  pzm.y * azc.y;
                if (pending == 2) {   // the older direction is the one this iteration's replaces
                    double2 ev = lg2(e + c);
                    const double2 pw = lg2(pn_ + c), pv = lg2(po + c);
                    ev.x = (ev.x - alpha_old * pw.x) - alpha0 * pv.x;
                    ev.y = (ev.y - alpha_old * pw.y) - alpha0 * pv.y;
                    put(e + c, ev, two);
                }
                put(q + c, make_double2(q0, q1), two);
                put(pn_ + c, pc, two);
                dot += pc.x * q0;
                if (two) dot += pc.y * q1;
            }
        }
        if (pending == 2) pending = 0;
        s.dot(coop_sum(S, dot));
        if (s.done || S.failed) break;
        const double alpha = s.alpha;
        double rr = 0.;
        for (int u = last; u >= 0; u -= step) {
            const int kz = u / uxy, rem = u - kz * uxy, jj = rem / ux, j = jj + 1, i0 = 2 * (rem - jj * ux) + 1, k0 = kz * KZ + 1;
            const bool two = i0 < nx;
            const int c0 = kBase + (i0 - 1) + px * j;
#pragma unroll
            for (int m = 0; m < KZ; ++m) {
                const int k = k0 + m;
                if (k > nz) break;
                const int c = c0 + pxy * k;
                double2 rv = lg2(r + c);
                const double2 qv = lg2(q + c);
                rv.x = rv.x - alpha * qv.x;
                rv.y = rv.y - alpha * qv.y;
                put(r + c, rv, two);
                rr += rv.x * rv.x;
                if (two) rr += rv.y * rv.y;
            }
        }
        if (pending == 0) alpha_old = alpha;
        ++pending;
        s.residual(coop_sum(S, rr), mode, thr, maxit);
    }
    if (pending > 0) {   // the last iterations' updates of e
        const double* p1 = ((s.iters - pending + 1) & 1) ? pa : pb;
        const double* p2 = (s.iters & 1) ? pa : pb;
        for (int u = first; u < units; u += step) {
            const int kz = u / uxy, rem = u - kz * uxy, jj = rem / ux, i0 = 2 * (rem - jj * ux) + 1, k0 = kz * KZ + 1;
            for (int k = k0; k < k0 + KZ && k <= nz; ++k) {
                const int c = kBase + (i0 - 1) + px * (jj + 1) + pxy * k;
                double2 ev = lg2(e + c);
                double2 pv = lg2(p1 + c);
                ev.x = ev.x - alpha_old * pv.x;
                ev.y = ev.y - alpha_old * pv.y;
                if (pending == 2) {
                    pv = lg2(p2 + c);
                    ev.x = ev.x - s.alpha * pv.x;
                    ev.y = ev.y - s.alpha * pv.y;
                }
                put(e + c, ev, i0 < nx);
            }
        }
    }
    coop_store(s, S.failed, st);
}

}  // namespace suli
