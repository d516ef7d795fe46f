// k_cg_coop.cuh — the plain FP64 CG as one cooperative launch (included by k_fp64.cu).
//
// The two-kernel iteration (k_cg_spmv*, k_cg_update) costs two launches, two ramps and two
// last-block reductions, whatever the grid: about 16-20 us on grids whose data the L2 holds and
// whose arithmetic takes 1-2 us.  Here every CTA stays resident for the whole solve and an
// iteration is two grid-wide sums (p.q, r.r), each also the barrier that publishes r (or p).
//
// Grid-wide sum: every CTA has an inbox with one 8-byte slot a CTA.  A CTA writes its partial into
// its slot of every inbox (release), polls its own inbox until no slot holds the "empty" pattern
// and adds the partials in CTA order (fixed order, so a run is bit-reproducible): one store and
// one load latency a sum, no atomics, and no two CTAs poll the same lines (with one shared slot
// a CTA, polled by all, a sum took 2 us longer at 110 CTAs than at 55).  Three inbox sets take
// turns: before a CTA publishes in one set it empties its own inbox of the next, which it read two
// sums ago and which nobody writes before having seen that publication.  Each wait is bounded; a
// wait that runs out ends the solve with SULI_ERR_CUDA.
#pragma once

namespace suli {

constexpr long long kSlotEmpty = -1;          // all bits set: no partial sum is published as this NaN
constexpr int kCoopSpin = 1 << 22;            // polls of a bounded wait (each about an L2 latency)

struct CoopSum {
    long long* slots;   // [3][nctas][pitch], all empty at launch
    int n;              // CTAs
    int pitch;          // slots an inbox, rounded up to whole 128-byte lines
    int round;          // sums done, modulo 3
    double* sh;         // shared scratch: warp partials, the total, the failure flag
    bool failed;
};
constexpr int kCoopShared = 34;
__host__ __device__ inline int coop_pitch(int n) { return (n + 15) & ~15; }

template <bool ACQUIRE>
__device__ __forceinline__ long long slot_load(const long long* p) {
    long long v;
    if (ACQUIRE) asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    else asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void slot_store(long long* p, long long v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Sum of v over the grid; every thread gets it.  PUBLISH: every global store of the CTA before the
// call is visible to every CTA's loads (from L2) after it; without it the sum orders nothing (and
// waits for no store).  Of two successive sums at least one publishes: its fence also orders the
// emptied slots, which are emptied one sum after they were read and written again one sum later.
template <bool PUBLISH>
__device__ __forceinline__ double coop_sum(CoopSum& S, double v) {
    const int tid = threadIdx.x, lane = tid & 31, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) S.sh[tid >> 5] = v;
    __syncthreads();
    if (tid < 32) {
        v = (lane < nw) ? S.sh[lane] : 0.;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const int prev = (S.round == 0) ? 2 : S.round - 1;
        const long long mine = isnan(v) ? 0x7ff8000000000000ll : __double_as_longlong(v);
        long long* set = S.slots + (long long)S.round * S.n * S.pitch;
        long long* clear = S.slots + ((long long)prev * S.n + blockIdx.x) * S.pitch;
        if (!PUBLISH)
            for (int q = lane; q < S.n; q += 32) slot_store(set + (long long)q * S.pitch + blockIdx.x, mine);
        for (int q = lane; q < S.n; q += 32) slot_store(clear + q, kSlotEmpty);
        if (PUBLISH) {
            __threadfence();
            for (int q = lane; q < S.n; q += 32) slot_store(set + (long long)q * S.pitch + blockIdx.x, mine);
        }
        set += (long long)blockIdx.x * S.pitch;
        double t = 0.;
        bool ok = true;
        for (int q0 = lane; q0 < S.n; q0 += 5 * 32) {   // five slots a lane in flight
            long long w[5];
            int spin = 0;
            bool all;
            do {
                all = true;
#pragma unroll
                for (int m = 0; m < 5; ++m) {
                    const int q = q0 + 32 * m;
                    w[m] = (q < S.n) ? slot_load<PUBLISH>(set + q) : 0;
                }
#pragma unroll
                for (int m = 0; m < 5; ++m) all = all && (w[m] != kSlotEmpty);
            } while (!all && ++spin < kCoopSpin);
            ok = ok && all;
#pragma unroll
            for (int m = 0; m < 5; ++m)
                if (q0 + 32 * m < S.n) t += __longlong_as_double(w[m]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        ok = __all_sync(0xffffffffu, ok);
        if (lane == 0) {
            S.sh[32] = t;
            S.sh[33] = ok ? 0. : 1.;
        }
    }
    __syncthreads();
    S.round = (S.round == 2) ? 0 : S.round + 1;
    S.failed = S.failed || S.sh[33] != 0.;
    return S.sh[32];
}

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
__device__ __forceinline__ void coop_store(const CoopCG& s, bool failed, CGState* st) {
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
// its two sums and of the neighbours' loads (25x50x45: 5.1 us an iteration, 17.5 with two kernels);
// four cells a thread, so that fewer CTAs (55 there) take part in the sums.
template <int U, int NT>
__global__ void __launch_bounds__(NT, 1) k_cg_reg(Geo G, BC bc, double* r, double* pa, double* e,
                                                  const double* __restrict__ ax, const double* __restrict__ ay,
                                                  const double* __restrict__ az, CGState* st, long long* slots) {
    __shared__ double sh[kCoopShared];
    CoopCG s = coop_load(st);
    if (s.done) return;
    const double thr = st->thr;
    const int mode = st->mode, maxit = st->maxit;
    CoopSum S{slots, (int)gridDim.x, coop_pitch((int)gridDim.x), 0, sh, false};
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
        s.dot(coop_sum<false>(S, dot));
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
        s.residual(coop_sum<true>(S, rr), mode, thr, maxit);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (c[u] >= 0) {
            e[c[u]] = ec[u];
            pa[c[u]] = p[u];
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) coop_store(s, S.failed, st);
}

// Larger grids: the iteration's two passes over units dealt to the threads in turn (a unit is a
// pair of x cells, 16-byte loads, and a column of KZ planes).  The first pass also applies the
// previous iteration's e -= alpha p, whose p it reads anyway, so the second only forms r; it
// takes the units in reverse order, newest in the L2 first.  Iteration n (from 1) writes its
// direction into pa for odd n, pb for even n.  Bound by the loads a thread's 64 registers keep in
// flight: 12 passes in 83.8 us at 256x128x128, 4.8 TB/s (the two kernels' 13 passes: 103.4 us).
// Measured there: 512 threads of the same 87.7-97, 4 planes a unit 96, 8 planes 105, 1 plane 89.
template <int KZ, int NT>
__global__ void __launch_bounds__(NT, 1) k_cg_two(Geo G, BC bc, double* r, double* pa, double* pb, double* q, double* e,
                                                  const double* __restrict__ ax, const double* __restrict__ ay,
                                                  const double* __restrict__ az, CGState* st, long long* slots) {
    __shared__ double sh[kCoopShared];
    CoopCG s = coop_load(st);
    if (s.done) return;
    const double thr = st->thr;
    const int mode = st->mode, maxit = st->maxit;
    CoopSum S{slots, (int)gridDim.x, coop_pitch((int)gridDim.x), 0, sh, false};
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
    bool pending = false;   // e lacks the previous iteration's update
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
                put(q + c, make_double2(q0, q1), two);
                put(pn_ + c, pc, two);
                dot += pc.x * q0;
                if (two) dot += pc.y * q1;
                if (pending) {
                    double2 ev = lg2(e + c);
                    const double2 pv = lg2(po + c);
                    ev.x = ev.x - alpha0 * pv.x;
                    ev.y = ev.y - alpha0 * pv.y;
                    put(e + c, ev, two);
                }
            }
        }
        pending = false;
        s.dot(coop_sum<true>(S, dot));
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
        pending = true;
        s.residual(coop_sum<true>(S, rr), mode, thr, maxit);
    }
    if (pending) {   // the last iteration's e -= alpha p
        const double* p = (s.iters & 1) ? pa : pb;
        for (int u = first; u < units; u += step) {
            const int kz = u / uxy, rem = u - kz * uxy, jj = rem / ux, i0 = 2 * (rem - jj * ux) + 1, k0 = kz * KZ + 1;
            for (int k = k0; k < k0 + KZ && k <= nz; ++k) {
                const int c = kBase + (i0 - 1) + px * (jj + 1) + pxy * k;
                double2 ev = lg2(e + c);
                const double2 pv = lg2(p + c);
                ev.x = ev.x - s.alpha * pv.x;
                ev.y = ev.y - s.alpha * pv.y;
                put(e + c, ev, i0 < nx);
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) coop_store(s, S.failed, st);
}

}  // namespace suli
