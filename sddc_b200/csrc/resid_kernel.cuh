// A residual evaluation (compresid, compresid.f90:1-80 and what it calls) with
// one thread per line of solution points, as the time step's stages work
// (line_kernel.cuh), and the face traces of a state by the same split.
//
// resid_kernel, per tile of cells:
//   1  staging by TMA and asynchronous copies; the ghost and received states
//      of the faces without a neighbour in this context go to the places of
//      the neighbours' traces;
//   2  nablaQsp (compflux.f90:107-157): the line's sums of three variables'
//      gradients at a time from the face-averaged states, the exchange between
//      the lines that cross at a point, coalesced stores;
//   3  the fluxes and their derivative sums, the exchange, sources; the
//      residual to memory by TMA;
//   4  the AV smoothness sensor per cell (AV.f90:14-83).
// Three variables at a time, because the sums of all nine (18N doubles) leave
// no registers for the line's states, which would be read from shared memory
// again at every flux point.
//
// What bounds it: latency, at 2 warps of up to 255 registers per scheduler in
// double (2.5 of 168 spill: 412 bytes at N = 5, no faster).  us per
// evaluation of a context, by tiles and by lines: FP64 N = 5, 16^2 cells 35
// and 27, 64^2 54 and 44, 200x150 222 and 170; N = 6, 200x150 373 and 280;
// mixed N = 5, 200x150 160 and 147; exact N = 5, 64^2 66 and 67 (the second
// wave of CTAs has 91 of 592), 200x150 290 and 264.  With the caller's memory,
// 90x90 cells, N = 5, FP64: 120 and 87, where half of the gain is the launches
// around it (one copy back, none in).
#pragma once

#include "line_kernel.cuh"

namespace sddc {

template <int N, typename R> struct ResidSmem {
    static constexpr int CPB = line_tile_cells(N);
    static constexpr int NQ = 9 * N * N, NN = N * N, NL = N - 1;
    static constexpr bool kPad = N % 2 == 0;  // two doubles per cell against bank conflicts
    static constexpr int QS = kPad ? NQ + 2 : NQ;
    static constexpr int MS = MetLayout<N>::kSize;
    static constexpr int TS = 4 * trace_stride<N, R>() + 16 / (int)sizeof(R);  // in R
    static constexpr int XS = QS;  // exchanged sums and what comes of them, then the sensor's values
    static_assert(2 * (NL * NL + NL * N + NN) <= XS, "the sensor's values fit the exchange region");
    static constexpr size_t kBytes =
        (size_t)CPB * (8 * (QS + MS + XS + NN) + TS * sizeof(R)) + 16 * 2 * line_threads(N, CPB) + 8 * (2 * NL * N + 4 * 32);
};
// Whether a thread holds its line's states in registers through the fluxes (as
// line_hold; in the exact form at N = 5 they spill)
template <int N, typename R, bool EX> __host__ __device__ constexpr bool resid_hold() { return sizeof(R) == 4 || N <= (EX ? 4 : 5); }
template <int N, typename R> constexpr int resid_min_blocks()
{
    const int w = (sizeof(R) == 4 || N == 2 ? 12 : 8) /
                  (line_threads(N, ResidSmem<N, R>::CPB) / 32);
    const int m = (int)(228 * 1024 / (ResidSmem<N, R>::kBytes + 1280));
    const int b = w < m ? w : m;
    return b < 1 ? 1 : b;
}

template <int N, typename R, bool EXACT>
__global__ void __launch_bounds__(line_threads(N, ResidSmem<N, R>::CPB), (resid_min_blocks<N, R>()))
    resid_kernel(const StageArgs a, const Ops ops)
{
    constexpr bool EX = EXACT && sizeof(R) == sizeof(double);
    using S = ResidSmem<N, R>;
    using ML = MetLayout<N>;
    constexpr int CPB = S::CPB, NT = line_threads(N, CPB), NQ = S::NQ, NN = S::NN, QS = S::QS, MS = S::MS, TS = S::TS,
                  XS = S::XS, NH = (N + 1) / 2;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *sQ = reinterpret_cast<double *>(smem_raw);  // [CPB][QS]
    double *sMet = sQ + CPB * QS;                        // [CPB][MS] normals, Jac
    double *sX = sMet + CPB * MS;                        // [CPB][XS]
    double *sJz = sX + CPB * XS;                         // [CPB][NN] Jz^2
    R *sT = reinterpret_cast<R *>(sJz + CPB * NN);       // [CPB][TS] the other sides' traces
    // the partners' normals at the ends r = 0 and r = N of each thread's line
    double2 *sP = reinterpret_cast<double2 *>(sT + CPB * TS);  // [2][NT]
    double *sOpH = reinterpret_cast<double *>(sP + 2 * NT);    // [N-1][N]  AV projection
    double *sOpHL = sOpH + (N - 1) * N;                        // [N][N-1]  AV prolongation
    double *sRed = sOpHL + N * (N - 1);                        // [4][32]
    __shared__ __align__(8) unsigned long long sBar;
    __shared__ int sAbort;

    const int tid = threadIdx.x, tile = blockIdx.x;
    int c0, ncl, cs;
    bool first_tile;
    if (a.tiles) {
        const int4 tl = a.tiles[tile];
        c0 = tl.x;
        ncl = tl.y;
        cs = tl.z;
        first_tile = tl.w != 0;
    } else {
        c0 = tile * CPB;
        ncl = min(CPB, a.ncell - c0);
        cs = 0;
        first_tile = tile == 0;
    }
    double *maxima = a.maxima + 10 * cs;
    // this thread's line (as in line_kernel) and the records of its end faces
    const int fam = tid >= N * CPB ? 1 : 0;
    const int lt = tid - fam * N * CPB, lc = lt % CPB;
    const bool act = tid < 2 * N * CPB && lc < ncl;
    const int c = act ? lc : 0, l = act ? lt / CPB : 0;
    const int lf0 = fam == 0 ? 4 : 1, lfN = fam == 0 ? 2 : 3;
    const int np0 = fam == 0 ? N - 1 - l : l, npN = fam == 0 ? l : N - 1 - l;  // 0-based
    int2 rec0 = make_int2(0, 0), recN = make_int2(0, 0);
    if (act) {
        rec0 = __ldg(a.faces + (size_t)(c0 + c) * 4 + lf0 - 1);
        recN = __ldg(a.faces + (size_t)(c0 + c) * 4 + lfN - 1);
    }
    const int pt0 = fam == 0 ? N * l : l, pts = fam == 0 ? 1 : N;  // point t of the line: pt0 + pts*t
    const int q0 = c * QS + 9 * pt0, qstr = 9 * pts;
    const int par = (l ^ fam) & 1;                                 // this thread finishes points t with t + par even

    // ---- 1: staging -------------------------------------------------------------
    const double *qsrc = a.q_in + (size_t)c0 * NQ, *msrc = a.met + (size_t)c0 * MS;
    const unsigned cbytes = (unsigned)((S::kPad ? 1 : ncl) * NQ * sizeof(double));
    const bool bulk = (((uintptr_t)qsrc | (uintptr_t)msrc | cbytes) & 15) == 0;
    if (tid < 32) {
        if (tid == 0) {
            sAbort = 0;
            mbar_init(&sBar, 1);
            if (bulk) {
                mbar_expect_tx(&sBar, (unsigned)(ncl * (MS + NQ) * sizeof(double)));
                bulk_g2s(sMet, msrc, (unsigned)(ncl * MS * sizeof(double)), &sBar);
            }
        }
        __syncwarp();
    }
    if (act) {
#pragma unroll 1
        for (int r = 0; r <= N; r += N) {  // the left (partner) cell's normals of the right cell's ends
            const int2 rec = r == 0 ? rec0 : recN;
            if ((rec.y & 0xff) != kFaceRight) continue;
            int pfam, pline, pr;
            face_point<N>((rec.y >> 8) & 0xff, N - (r == 0 ? np0 : npN), pfam, pline, pr);
            const double *pn = a.met + (size_t)rec.x * MS + ML::normal(pfam, pline, pr);
            double *o = reinterpret_cast<double *>(sP + (r == 0 ? 0 : NT) + tid);
            cp_async_pair(o, pn);
            cp_async_pair(o + 1, pn + 1);
        }
    }
    grid_dependency_wait();  // the state, the traces and the maxima come from earlier launches
    if (tid < 32) {
        if (bulk && tid < (S::kPad ? ncl : 1)) bulk_g2s(sQ + tid * QS, qsrc + (size_t)tid * NQ, cbytes, &sBar);
    }
    if (!bulk) {
        for (int k = tid; k < ncl * NQ; k += NT) {
            const int cc = k / NQ;
            sQ[cc * QS + (k - cc * NQ)] = __ldg(qsrc + k);
        }
        for (int k = tid; k < ncl * MS; k += NT) sMet[k] = __ldg(msrc + k);
    }
    // the neighbours' traces: 16 bytes at a time, or value by value where the
    // records are packed (tfs = 9N) to no multiple of that
    const int tfs = a.tfs;
    auto stage_traces = [&](auto piece) {
        using E = decltype(piece);  // what one copy moves
        constexpr int EL = sizeof(E) / sizeof(R), CH = (9 * N + EL - 1) / EL;
        const R *tin = reinterpret_cast<const R *>(a.t_in);
        constexpr int B = 6;  // face records loaded ahead of their copies
        for (int e0 = tid; e0 < ncl * 4 * CH; e0 += B * NT) {
            int2 r[B];
#pragma unroll
            for (int m = 0; m < B; m++) {
                const int f = (e0 + m * NT) / CH;
                r[m] = f < ncl * 4 ? __ldg(a.faces + (size_t)c0 * 4 + f) : make_int2(0, 0);
            }
#pragma unroll
            for (int m = 0; m < B; m++) {
                const int e = e0 + m * NT, f = e / CH, ch = e - f * CH, kd = r[m].y & 0xff;
                if (kd != kFaceLeft && kd != kFaceRight) continue;
                R *dst = sT + (f >> 2) * TS + (f & 3) * trace_stride<N, R>() + ch * EL;
                const R *src = tin + ((size_t)r[m].x * 4 + ((r[m].y >> 8) & 0xff) - 1) * tfs + ch * EL;
                if constexpr (EL > 1) cp_async16(dst, src);
                else cp_async_pair(dst, src);
            }
        }
    };
    if ((tfs * sizeof(R) % 16 | ((uintptr_t)a.t_in & 15)) == 0) stage_traces(double2{});
    else stage_traces(R{});
    for (int k = tid; k < (N - 1) * N; k += NT) {
        sOpH[k] = ops.H[k];
        sOpHL[k] = ops.HL[k];
    }
    const double eig_r = maxima[2 * a.slot_r], um_r = maxima[2 * a.slot_r + 1];
    // compflux.f90:6 -- running maxima of all previous stages
    const R c_h = (R)sqrt(eig_r * (eig_r - um_r));
    cp_async_wait_all();
    if (bulk && tid == 0 && !mbar_wait_bounded(&sBar, 0)) {
        raise_fault(a.err_flags, kErrStagingTimeout);
        sAbort = 1;
        mbar_wait_bounded(&sBar, 0);
    }
    __syncthreads();
    if (sAbort) return;
    if constexpr (!EX) {  // these forms multiply by 1/Jac, rounded once
        for (int k = tid; k < ncl * NN; k += NT) {
            double *J = sMet + k / NN * MS + ML::kJac + k % NN;
            *J = 1.0 / *J;
        }
    }

    // the interpolated state at flux point r, variables v..v+K-1
    auto interpolate = [&](int r, int v, auto &q) {
        constexpr int K = sizeof(q) / sizeof(R);
        int qi = q0;
        asm volatile("" : "+r"(qi));  // read anew at every point: the registers hold sums
#pragma unroll
        for (int k = 0; k < K; k++) q[k] = (R)0;
#pragma unroll
        for (int s = 0; s < N; s++) {
            const R L = opL<R>(ops, r * N + s);
#pragma unroll
            for (int k = 0; k < K; k++) q[k] = q[k] + (R)sQ[qi + qstr * s + v + k] * L;
        }
    };
    auto normal = [&](int r, R &n0, R &n1) {
        const double2 n = *reinterpret_cast<const double2 *>(sMet + c * MS + ML::normal(fam, l, r));
        n0 = (R)n.x;
        n1 = (R)n.y;
    };
    // the other side's trace at the line's end r: 9 values N apart
    auto other_at = [&](int r) {
        return sT + c * TS + ((r == 0 ? lf0 : lfN) - 1) * trace_stride<N, R>() + (N - 1 - (r == 0 ? np0 : npN));
    };
    if (act) {
#pragma unroll 1
        for (int r = 0; r <= N; r += N) {
            const int2 rec = r == 0 ? rec0 : recN;
            const int kind = rec.y & 0xff;
            if (kind == kFaceLeft || kind == kFaceRight) continue;
            R *tp = other_at(r);
            if (kind == kFaceProc) {
                // the received trace, remote point N+1-nfp (procintflux_all.f90:83-99)
                const R *rv = reinterpret_cast<const R *>(a.proc_recv) +
                              ((size_t)rec.x * N + (N - 1 - (r == 0 ? np0 : npN))) * 9;
#pragma unroll
                for (int k = 0; k < 9; k++) tp[k * N] = rv[k];
            } else {
                R own[9], oth[9], n0, n1;
                interpolate(r, 0, own);
                normal(r, n0, n1);
                bc_ghost<R, EX>(kind, own, n0, n1, a.vismode, a.cases ? a.cases[cs].fs : a.fs, oth);
#pragma unroll
                for (int k = 0; k < 9; k++) tp[k * N] = oth[k];
            }
        }
    }

    // ---- 2: gradients (with vismode == 0 the reference never fills nablaQs) --------
    double divB[NH], jz[NH];  // div B and Jz of this thread's points
#pragma unroll
    for (int m = 0; m < NH; m++) divB[m] = jz[m] = 0.0;
    if (a.vismode == 1) {
        constexpr int G = 3;  // variables at a time: their values and sums stay in registers
#pragma unroll 1
        for (int v = 0; v < 9; v += G) {
            R gx[N][G], gy[N][G];
#pragma unroll
            for (int i = 0; i < N; i++)
#pragma unroll
                for (int k = 0; k < G; k++) gx[i][k] = gy[i][k] = (R)0;
            if (act) {
                R qs[N][G];
#pragma unroll
                for (int s = 0; s < N; s++)
#pragma unroll
                    for (int k = 0; k < G; k++) qs[s][k] = (R)sQ[q0 + qstr * s + v + k];
#pragma unroll
                for (int r = 0; r <= N; r++) {
                    R V[G], n0, n1;
                    normal(r, n0, n1);
#pragma unroll
                    for (int k = 0; k < G; k++) V[k] = (R)0;
#pragma unroll
                    for (int s = 0; s < N; s++) {
                        const R L = opL<R>(ops, r * N + s);
#pragma unroll
                        for (int k = 0; k < G; k++) V[k] = V[k] + qs[s][k] * L;
                    }
                    if (r == 0 || r == N) {
                        const R *tp = other_at(r) + v * N;
                        const bool own_right = ((r == 0 ? rec0 : recN).y & 0xff) == kFaceRight;
#pragma unroll
                        for (int k = 0; k < G; k++) {
                            const R o = tp[k * N], ql = own_right ? o : V[k], qr = own_right ? V[k] : o;
                            V[k] = (R)0.5 * ql + (R)0.5 * qr;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < N; i++) {
                        const R M = opM<R>(ops, r * N + i);
#pragma unroll
                        for (int k = 0; k < G; k++) {
                            const R m = V[k] * M;
                            gx[i][k] = gx[i][k] + m * n0;
                            gy[i][k] = gy[i][k] + m * n1;
                        }
                    }
                }
#pragma unroll
                for (int m = 0; m < NH; m++) {
                    const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
                    if (2 * m + 1 < N || par) {
                        double *o = sX + c * XS + (pt0 + pts * (2 * m + 1 - par)) * 2 * G;
#pragma unroll
                        for (int k = 0; k < G; k++) {
                            o[k] = (double)(par ? gx[i0][k] : gx[i1][k]);
                            o[G + k] = (double)(par ? gy[i0][k] : gy[i1][k]);
                        }
                    }
                }
            }
            __syncthreads();
            if (act) {
#pragma unroll
                for (int m = 0; m < NH; m++) {
                    const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
                    if (!(2 * m + 1 < N) && par) continue;
                    const int pt = pt0 + pts * (2 * m + par);
                    double *x = sX + c * XS + pt * 2 * G;
                    const double J = sMet[c * MS + ML::kJac + pt];
                    double g[2 * G];
#pragma unroll
                    for (int k = 0; k < G; k++) {
                        g[k] = (double)((par ? gx[i1][k] : gx[i0][k]) + (R)x[k]);
                        g[G + k] = (double)((par ? gy[i1][k] : gy[i0][k]) + (R)x[G + k]);
                    }
                    if constexpr (EX) {
                        quotients<2 * G>(g, J, g);
                    } else {
#pragma unroll
                        for (int k = 0; k < 2 * G; k++) g[k] = g[k] * J;
                    }
#pragma unroll
                    for (int k = 0; k < 2 * G; k++) x[k] = g[k];
                    // div B = Bx,x + By,y and Jz = By,x - Bx,y
                    if (v == 3) {
                        divB[m] = g[2];
                        jz[m] = g[G + 2];
                    } else if (v == 6) {
                        divB[m] = divB[m] + g[G];
                        jz[m] = g[0] - jz[m];
                    }
                }
            }
            __syncthreads();
            if (a.grad_out) {
                double *go = a.grad_out + (size_t)c0 * 18 * NN + v;
                for (int k = tid; k < ncl * 2 * G * NN; k += NT) {
                    const int cc = k / (2 * G * NN), e = k - cc * (2 * G * NN), p = e / (2 * G), j = e - p * (2 * G);
                    go[(size_t)cc * 18 * NN + p * 18 + (j < G ? j : 9 - G + j)] = sX[cc * XS + e];
                }
            }
            __syncthreads();
        }
    } else if (a.grad_out) {
        for (int k = tid; k < ncl * 18 * NN; k += NT) a.grad_out[(size_t)c0 * 18 * NN + k] = 0.0;
    }
    if (act) {
#pragma unroll
        for (int m = 0; m < NH; m++)
            if (2 * m + 1 < N || !par) sJz[c * NN + pt0 + pts * (2 * m + par)] = jz[m] * jz[m];
    }

    // ---- 3: fluxes and residual -----------------------------------------------------
    R eigmax = (R)0, umax = (R)0;
    unsigned err = 0;
    P2<R> d[N][4];  // derivative sums of the variable pairs 0..7
    R d8[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
#pragma unroll
        for (int k = 0; k < 4; k++) d[i][k] = splat2<R>((R)0);
        d8[i] = (R)0;
    }
    if (act) {
        constexpr bool kHold = resid_hold<N, R, EX>();
        R qs[kHold ? N : 1][9];
        if constexpr (kHold) {
#pragma unroll
            for (int s = 0; s < N; s++)
#pragma unroll
                for (int k = 0; k < 9; k++) qs[s][k] = (R)sQ[q0 + qstr * s + k];
        }
        auto add = [&](int r) {
            R q[9], F[9], n0, n1;
            if constexpr (kHold) {
#pragma unroll
                for (int k = 0; k < 9; k++) q[k] = (R)0;
#pragma unroll
                for (int s = 0; s < N; s++) {
                    const R L = opL<R>(ops, r * N + s);
#pragma unroll
                    for (int k = 0; k < 9; k++) q[k] = q[k] + qs[s][k] * L;
                }
            } else {
                interpolate(r, 0, q);
            }
            normal(r, n0, n1);
            if (r > 0 && r < N) {
                // interior flux point (inviscid_flux_interior)
                if (!(q[0] > (R)0)) err |= kErrNonPositiveDensity;
                if constexpr (EX) {
                    R Fx[9], G[9];
                    iflux<R, EX>(q, c_h, umax, Fx, G);
#pragma unroll
                    for (int k = 0; k < 9; k++) F[k] = Fx[k] * n0 + G[k] * n1;
                } else {
                    iflux_n<R>(q, c_h, n0, n1, umax, F);
                }
            } else {
                // face point (interfaceflux, CYCLOCFLUX, BCFLUX, PROCINTFLUX)
                const int2 rec = r == 0 ? rec0 : recN;
                const int kind = rec.y & 0xff, plf = (rec.y >> 8) & 0xff;
                const bool own_right = kind == kFaceRight, plow = plf == 1 || plf == 4;
                int sign_l = r == 0 ? -1 : 1, sign_r = 1;
                if (kind == kFaceLeft) {
                    sign_r = plow ? 1 : -1;
                } else if (own_right) {
                    const double2 pn = sP[(r == 0 ? 0 : NT) + tid];  // the left (partner) cell's normal
                    n0 = (R)pn.x;
                    n1 = (R)pn.y;
                    sign_l = plow ? -1 : 1;
                    sign_r = r == N ? -1 : 1;
                }
                const R *tp = other_at(r);
                R Ql[9], Qr[9];
#pragma unroll
                for (int k = 0; k < 9; k++) {
                    const R o = tp[k * N];
                    Ql[k] = own_right ? o : q[k];
                    Qr[k] = own_right ? q[k] : o;
                }
                if (!(Ql[0] > (R)0) || !(Qr[0] > (R)0)) err |= kErrNonPositiveDensity;
                R eig_face;
                rusanov<R, EX>(Ql, Qr, F, (R *)nullptr, n0, n1, sign_l, sign_r, c_h, eig_face, umax);
                if (!(Abs(eig_face) < (R)INFINITY)) err |= kErrNonFiniteWaveSpeed;
                if (eig_face > eigmax) eigmax = eig_face;
                // the right cell's slot: the left one's with both signs
                const R so = own_right ? (R)(sign_l * sign_r) : (R)1;
#pragma unroll
                for (int k = 0; k < 9; k++) F[k] = so * F[k];
            }
            // its share of the derivatives (compresid.f90:14-32)
#pragma unroll
            for (int i = 0; i < N; i++) {
                const P2<R> M2 = opM2<R>(ops, r * N + i);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    P2<R> f2;
                    f2.x = F[2 * k];
                    f2.y = F[2 * k + 1];
                    d[i][k] = fma2(f2, M2, d[i][k]);
                }
                d8[i] = d8[i] + F[8] * M2.x;
            }
        };
        add(0);
#pragma unroll 1
        for (int r = 1; r < N; r++) add(r);
        add(N);
    }
    if (act) {
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (2 * m + 1 < N || par) {
                double *o = sX + c * XS + (pt0 + pts * (2 * m + 1 - par)) * 9;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    o[2 * k] = (double)(par ? d[i0][k].x : d[i1][k].x);
                    o[2 * k + 1] = (double)(par ? d[i0][k].y : d[i1][k].y);
                }
                o[8] = (double)(par ? d8[i0] : d8[i1]);
            }
        }
    }
    __syncthreads();
    double part_r = 0.0, part_d = 0.0;
    if (act) {
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (!(2 * m + 1 < N) && par) continue;
            const int pt = pt0 + pts * (2 * m + par);
            double *x = sX + c * XS + pt * 9;
            const double J = sMet[c * MS + ML::kJac + pt], dB = divB[m];
            const double *q = sQ + c * QS + 9 * pt;
            double res[9];
#pragma unroll
            for (int k = 0; k < 9; k++) {
                const R own = k == 8 ? (par ? d8[i1] : d8[i0])
                              : k % 2 ? (par ? d[i1][k / 2].y : d[i0][k / 2].y)
                                      : (par ? d[i1][k / 2].x : d[i0][k / 2].x);
                res[k] = (double)(-(own + (R)x[k]));
                // the viscous chain (compresid.f90:34-49); it adds exactly +0.0
                // when mu == eta0 == 0, which only the exact form reproduces
                if constexpr (EX) {
                    if (a.vismode == 1)
                        res[k] = res[k] + (a.visc ? a.visc[(size_t)(c0 + c) * NQ + 9 * pt + k] : 0.0);
                } else {
                    if (a.vismode == 1 && a.visc) res[k] = res[k] + a.visc[(size_t)(c0 + c) * NQ + 9 * pt + k];
                }
            }
            // compresid.f90:53-78: 1/Jac, Powell 8-wave and GLM sources
            const double Bx = q[5], By = q[6], Bz = q[7], psi = q[8];
            double u[3];
            if constexpr (EX) {
                quotients<9>(res, J, res);
                quotients<3>(q + 1, q[0], u);
            } else {
                const double ri = 1.0 / q[0];
#pragma unroll
                for (int k = 0; k < 9; k++) res[k] = res[k] * J;
                u[0] = q[1] * ri; u[1] = q[2] * ri; u[2] = q[3] * ri;
            }
            res[1] = res[1] - dB * Bx;
            res[2] = res[2] - dB * By;
            res[3] = res[3] - dB * Bz;
            res[4] = res[4] - dB * ((u[0] * Bx + u[1] * By) + u[2] * Bz);
            res[5] = res[5] - dB * u[0];
            res[6] = res[6] - dB * u[1];
            res[7] = res[7] - dB * u[2];
            res[8] = res[8] - a.alpha * psi;
            if (a.mon_part) {
#pragma unroll
                for (int k = 0; k < 9; k++) part_r += res[k] * res[k];
                part_d += dB * dB;
            }
#pragma unroll
            for (int k = 0; k < 9; k++) x[k] = res[k];
        }
    }
    fence_proxy_async();
    __syncthreads();
    if (a.resid_out) {
        double *dst = a.resid_out + (size_t)c0 * NQ;
        if ((((uintptr_t)dst | cbytes) & 15) == 0) {
            if (tid < (S::kPad ? ncl : 1)) bulk_s2g(dst + (size_t)tid * NQ, sX + tid * XS, cbytes);
            if (tid < 32) bulk_wait_read();
        } else {
            for (int k = tid; k < ncl * NQ; k += NT) dst[k] = sX[k / NQ * XS + k % NQ];
        }
        __syncthreads();
    }

    // ---- 4: AV smoothness sensor (comp_artificial_viscosity, AV.f90:14-83) ------
    if (a.artiv == 1 && a.vismode == 1) {
        constexpr int NL = S::NL;
        // the sensed fields, density and Jz^2, side by side in each thread
        auto field = [&](int cc, int is, int js) {
            return make_double2(sQ[cc * QS + 9 * (is + N * js)], sJz[cc * NN + is + N * js]);
        };
        double2 *sLow = reinterpret_cast<double2 *>(sX), *sTmp = sLow + CPB * NL * NL, *sTerm = sTmp + CPB * NL * N;
        if constexpr (EX) {
            // projection to the N-1 points with the reference's double sum
            for (int t = tid; t < ncl * NL * NL; t += NT) {
                const int isl = t % NL, jsl = (t / NL) % NL, cc = t / (NL * NL);
                double2 acc = make_double2(0.0, 0.0);
                for (int js = 0; js < N; js++)
#pragma unroll
                    for (int is = 0; is < N; is++) {
                        const double2 f = field(cc, is, js);
                        const double h = sOpH[isl * N + is], g = sOpH[jsl * N + js];
                        acc.x = acc.x + f.x * h * g;
                        acc.y = acc.y + f.y * h * g;
                    }
                sLow[t] = acc;
            }
        } else {
            // the same projection as two one-dimensional passes
            for (int t = tid; t < ncl * NL * N; t += NT) {
                const int isl = t % NL, js = (t / NL) % N, cc = t / (NL * N);
                double2 acc = make_double2(0.0, 0.0);
#pragma unroll
                for (int is = 0; is < N; is++) {
                    const double2 f = field(cc, is, js);
                    const double h = sOpH[isl * N + is];
                    acc.x += f.x * h;
                    acc.y += f.y * h;
                }
                sTmp[(cc * N + js) * NL + isl] = acc;
            }
            __syncthreads();
            for (int t = tid; t < ncl * NL * NL; t += NT) {
                const int isl = t % NL, jsl = (t / NL) % NL, cc = t / (NL * NL);
                double2 acc = make_double2(0.0, 0.0);
#pragma unroll
                for (int js = 0; js < N; js++) {
                    const double2 f = sTmp[(cc * N + js) * NL + isl];
                    const double h = sOpH[jsl * N + js];
                    acc.x += f.x * h;
                    acc.y += f.y * h;
                }
                sLow[t] = acc;
            }
        }
        __syncthreads();
        // projection back to the solution points and the terms of the sensor
        // sum, one thread per (cell, point)
        if constexpr (!EX) {
            for (int t = tid; t < ncl * N * NL; t += NT) {
                const int is = t % N, jsl = (t / N) % NL, cc = t / (N * NL);
                const double2 *lo = sLow + cc * NL * NL;
                double2 acc = make_double2(0.0, 0.0);
#pragma unroll
                for (int isl = 0; isl < NL; isl++) {
                    const double2 f = lo[isl + NL * jsl];
                    const double h = sOpHL[is * NL + isl];
                    acc.x += f.x * h;
                    acc.y += f.y * h;
                }
                sTmp[(cc * NL + jsl) * N + is] = acc;
            }
            __syncthreads();
        }
        for (int t = tid; t < ncl * NN; t += NT) {
            const int is = t % N, js = (t / N) % N, cc = t / NN;
            double2 hi = make_double2(0.0, 0.0);
            if constexpr (EX) {
                const double2 *lo = sLow + cc * NL * NL;
                for (int jsl = 0; jsl < NL; jsl++)
#pragma unroll
                    for (int isl = 0; isl < NL; isl++) {
                        const double2 f = lo[isl + NL * jsl];
                        const double h = sOpHL[is * NL + isl], g = sOpHL[js * NL + jsl];
                        hi.x = hi.x + f.x * h * g;
                        hi.y = hi.y + f.y * h * g;
                    }
            } else {
#pragma unroll
                for (int jsl = 0; jsl < NL; jsl++) {
                    const double2 f = sTmp[(cc * NL + jsl) * N + is];
                    const double h = sOpHL[js * NL + jsl];
                    hi.x += f.x * h;
                    hi.y += f.y * h;
                }
            }
            const double2 x = field(cc, is, js);
            const double dx = hi.x - x.x, dy = hi.y - x.y;
            sTerm[cc * NN + is + N * js] = make_double2(dx * dx / (x.x * x.x), dy * dy / (x.y * x.y));
        }
        __syncthreads();
        // the sum in the reference's (js, is) order
        for (int t = tid; t < ncl * 2; t += NT) {
            const double *tm = reinterpret_cast<const double *>(sTerm + t / 2 * NN) + t % 2;
            double se = 0.0;
#pragma unroll
            for (int k = 0; k < NN; k++) se = se + tm[2 * k];
            a.sm_ind[2 * (size_t)c0 + t] = log10(se);
        }
    }

    // ---- reductions ----------------------------------------------------------------
    const int lane = tid & 31, wid = tid >> 5;
    constexpr int NW = NT / 32;
    const double em = warp_max((double)eigmax), um = warp_max((double)umax);
    const unsigned eb = __reduce_or_sync(0xffffffffu, err);
    double pr = 0.0, pd = 0.0;
    if (a.mon_part) {
        pr = warp_sum(part_r);
        pd = warp_sum(part_d);
    }
    if (lane == 0) {
        sRed[wid] = em;
        sRed[32 + wid] = um;
        sRed[64 + wid] = pr;
        sRed[96 + wid] = pd;
        if (eb) raise_fault(a.err_flags, eb);
    }
    __syncthreads();
    if (tid == 0) {
        double m0 = 0.0, m1 = 0.0, s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            m0 = sRed[w] > m0 ? sRed[w] : m0;
            m1 = sRed[32 + w] > m1 ? sRed[32 + w] : m1;
            s0 += sRed[64 + w];
            s1 += sRed[96 + w];
        }
        atomic_max_nonneg(&maxima[2 * a.slot_w], m0);
        atomic_max_nonneg(&maxima[2 * a.slot_w + 1], m1);
        if (first_tile) {  // carry the previous stages' maxima forward
            atomic_max_nonneg(&maxima[2 * a.slot_w], maxima[2 * a.slot_r]);
            atomic_max_nonneg(&maxima[2 * a.slot_w + 1], maxima[2 * a.slot_r + 1]);
        }
        if (a.mon_part) {
            a.mon_part[2 * tile] = s0;
            a.mon_part[2 * tile + 1] = s1;
        }
    }
}

// Face traces of a state: T[trace_at(tfs, cell, lf, nfp, k)] = sum_s Q(k, line
// points) * L(r, s) at the flux point of local face lf, face point nfp -- the
// same interpolation, in the same order and type, as the stages form.  One
// thread per line gives the traces at both of its ends; a cell's four faces
// leave by one TMA store (36N values: whole 16-byte units with either stride).
// 90x90 cells, N = 5, FP64, cold: 11.8 us with a thread per value, 8.7 so.
template <int N, typename R> struct TraceSmem {
    static constexpr int CPB = line_tile_cells(N);
    static constexpr int TS = 4 * trace_stride<N, R>() + 16 / (int)sizeof(R);
    static constexpr int QS = ResidSmem<N, R>::QS;
    static constexpr size_t kBytes = (size_t)CPB * (QS * sizeof(double) + TS * sizeof(R));
};
template <int N, typename R, bool EXACT>  // EXACT: compiled with -fmad=false, like the stages
__global__ void __launch_bounds__(line_threads(N, TraceSmem<N, R>::CPB))
    trace_kernel(int ncell, const double *__restrict__ q, R *__restrict__ t, int tfs, const TraceInit init,
                 const Ops ops)
{
    using S = TraceSmem<N, R>;
    constexpr int CPB = S::CPB, NT = line_threads(N, CPB), NQ = 9 * N * N, QS = S::QS, TS = S::TS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *sQ = reinterpret_cast<double *>(smem_raw);
    R *sT = reinterpret_cast<R *>(sQ + CPB * QS);
    const int tid = threadIdx.x, c0 = blockIdx.x * CPB, ncl = min(CPB, ncell - c0);
    const double *qsrc = q + (size_t)c0 * NQ;
    if (init.maxima && blockIdx.x == 0 && tid == 0) {
        for (int k = 0; k < 10; k += 2) {
            init.maxima[k] = init.eig;
            init.maxima[k + 1] = init.um;
        }
    }
    __shared__ __align__(8) unsigned long long sBar;
    __shared__ int sAbort;
    const unsigned cbytes = (unsigned)((QS != NQ ? 1 : ncl) * NQ * sizeof(double));
    const bool bulk = (((uintptr_t)qsrc | cbytes) & 15) == 0;
    if (bulk) {
        if (tid < 32) {
            if (tid == 0) {
                sAbort = 0;
                mbar_init(&sBar, 1);
                mbar_expect_tx(&sBar, (unsigned)(ncl * NQ * sizeof(double)));
            }
            __syncwarp();
            if (tid < (QS != NQ ? ncl : 1)) bulk_g2s(sQ + tid * QS, qsrc + (size_t)tid * NQ, cbytes, &sBar);
            if (tid == 0 && !mbar_wait_bounded(&sBar, 0)) {
                raise_fault(init.flags, kErrStagingTimeout);
                sAbort = 1;
                mbar_wait_bounded(&sBar, 0);
            }
        }
    } else {
        // batches of loads, so that each thread keeps several in flight
        constexpr int kU = 8;
        for (int k0 = tid; k0 < ncl * NQ; k0 += kU * NT) {
            double v[kU];
#pragma unroll
            for (int u = 0; u < kU; u++) v[u] = k0 + u * NT < ncl * NQ ? __ldg(qsrc + k0 + u * NT) : 0.0;
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const int k = k0 + u * NT, cc = k / NQ;
                if (k < ncl * NQ) sQ[cc * QS + (k - cc * NQ)] = v[u];
            }
        }
    }
    __syncthreads();
    if (bulk && sAbort) return;
    const int fam = tid >= N * CPB ? 1 : 0;
    const int lt = tid - fam * N * CPB, c = lt % CPB, l = lt / CPB;
    if (tid < 2 * N * CPB && c < ncl) {
        const double *ql = sQ + c * QS + 9 * (fam == 0 ? N * l : l);
        const int str = fam == 0 ? 9 : 9 * N;
        R e0[9], eN[9];
#pragma unroll
        for (int k = 0; k < 9; k++) e0[k] = eN[k] = (R)0;
#pragma unroll
        for (int s = 0; s < N; s++) {
            const R L0 = opL<R>(ops, s), LN = opL<R>(ops, N * N + s);
#pragma unroll
            for (int k = 0; k < 9; k++) {
                const R x = (R)ql[str * s + k];
                e0[k] = e0[k] + x * L0;
                eN[k] = eN[k] + x * LN;
            }
        }
        R *o0 = sT + c * TS + ((fam == 0 ? 4 : 1) - 1) * tfs + (fam == 0 ? N - 1 - l : l);
        R *oN = sT + c * TS + ((fam == 0 ? 2 : 3) - 1) * tfs + (fam == 0 ? l : N - 1 - l);
#pragma unroll
        for (int k = 0; k < 9; k++) {
            o0[k * N] = e0[k];
            oN[k * N] = eN[k];
        }
    }
    fence_proxy_async();
    __syncthreads();
    if (tid < 32) {
        if (tid < ncl) bulk_s2g(t + (size_t)(c0 + tid) * 4 * tfs, sT + tid * TS, (unsigned)(4 * tfs * sizeof(R)));
        bulk_wait_read();
    }
}

}  // namespace sddc
