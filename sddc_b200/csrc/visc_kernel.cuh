// The viscous / resistive chain of the SDDC residual (vismode = 1 with
// mu or eta0 nonzero): compflux.f90:36-50 and what it calls.
//
// Two launches before each stage launch, both with one thread per line of
// solution points as in line_kernel.cuh (sums in registers, one exchange
// between the lines that cross at a point):
//   visc_grad_kernel  face-averaged states at every flux point (interior:
//                     the interpolated state; faces: (left + right)/2 with
//                     the neighbour's trace or the boundary ghost state, as
//                     interfaceflux/BCFLUX store Qvfi/Qvfj), the gradient of
//                     all nine variables at the solution points (nablaQsp,
//                     compflux.f90:107-157), and its trace at the 4N face
//                     points, published for the neighbours;
//   visc_flux_kernel  the gradient at every flux point (interior:
//                     nablaQ_interior_FP, compflux.f90:159-196; faces: the
//                     average of both cells' traces, interfaceVISflux /
//                     CYCLOCVISFLUX, or the boundary state of BCVISFLUX with
//                     the adiabatic-wall energy gradient, bcflux.f90:380-666,
//                     which needs the internal-energy gradient of
//                     comp_grad_internal_energy, compflux.f90:260-298), the
//                     viscous flux there (getVfluxvectors, getrusanov.f90:
//                     197-294; comp_viscous_flux, compflux.f90:198-258) and
//                     its divergence dFv + dGv (compresid.f90:14-32), which
//                     the stage kernel adds to the inviscid residual.
// The AV viscous flux (getVfluxvectors_AV) has its coefficients hard-coded
// to zero (getrusanov.f90:326,328); it is not formed (it could only change
// the sign of a zero), nor are the first and last viscous flux components,
// which are zero.  Every sum keeps the reference's order; the exact
// instantiation is compiled without FMA.
//
// What bounds them: latency at 1.4 to 1.8 warps per scheduler (up to 255
// registers at N = 4 hold the sums of 18 and 7 values per point of the line;
// the states and gradients are read from shared memory at every flux point,
// which keeps the L1 pipe 59% and 49% busy).  At 128x128 cells, N = 4, FP64,
// they take 37 and 52 us cold; one thread per point and variable, with every
// operand from shared memory and an IEEE division per quotient, took about
// 215 together (a step of the chain: 1253 us then, 678 now).
#pragma once

#include "line_kernel.cuh"

namespace sddc {

constexpr double kLambdaVisc = -2.0 / 3.0;  // LAMBDA, setup2d.f90:69
constexpr double kPrandtl = 0.72;           // PRANDT, setup2d.f90:70

struct ViscArgs {
    int ncell, vismode;
    double mu, eta0;
    Freestream fs;
    const double *q;                  // stage input state
    const void *t_in;                 // its face traces (layout trace_at), in the form's type
    const double *__restrict__ met;   // packed metrics
    const double *__restrict__ met2;  // [cell][lf][nfp][2]: S1(2,1:2) or S2(1,1:2) at the face point
    const int2 *__restrict__ faces;
    double *grad;  // nablaQs (9,2,N,N,NCELL)
    double *gt;    // gradient traces [cell][lf][18][nfp]: (9 x-derivatives, 9 y-derivatives)
    double *rv;    // dFv + dGv (9,N,N,NCELL)
    FaultFlags *err_flags;
};

// o[k-1] = Fv(k) n0 + Gv(k) n1, k = 1..7, of getVfluxvectors
// (getrusanov.f90:197-294) with viscosity mu and resistivity eta0; nQ =
// (9 x-derivatives, 9 y-derivatives)
template <bool EX>
__device__ __forceinline__ void vflux(const double *Qv, const double *nQ, double mu, double eta0, double n0, double n1,
                                      double *o)
{
    const double rho = Qv[0], rhoE = Qv[4];
    const double Bx = Qv[5], By = Qv[6], Bz = Qv[7], psi = Qv[8];
    const double ri = EX ? 0.0 : 1.0 / rho;
    // quotients by rho
    auto over_rho = [&](auto &x) {
        constexpr int n = sizeof(x) / sizeof(double);
        if constexpr (EX) {
            quotients<n>(x, rho, x);
        } else {
#pragma unroll
            for (int k = 0; k < n; k++) x[k] = x[k] * ri;
        }
    };
    double vel[3] = {Qv[1], Qv[2], Qv[3]};
    over_rho(vel);
    const double u = vel[0], v = vel[1], w = vel[2];
    const double NORM_U = (u * u + v * v) + w * w;
    const double NORM_B = (Bx * Bx + By * By) + Bz * Bz;
    // the internal energy and the velocity gradients
    double a[7];
    a[6] = ((rhoE - 0.5 * NORM_U * rho) - 0.5 * NORM_B) - 0.5 * (psi * psi);
#pragma unroll
    for (int d = 0; d < 2; d++) {
        const double *g = nQ + 9 * d;
        a[3 * d] = g[1] - g[0] * u;
        a[3 * d + 1] = g[2] - g[0] * v;
        a[3 * d + 2] = g[3] - g[0] * w;
    }
    over_rho(a);
    const double inte = a[6];
    double e[2];
#pragma unroll
    for (int d = 0; d < 2; d++) {
        const double *g = nQ + 9 * d;
        const double dKE = 0.5 * NORM_U * g[0] + rho * ((u * a[3 * d] + v * a[3 * d + 1]) + w * a[3 * d + 2]);
        const double dpre_B = (Bx * g[5] + By * g[6]) + Bz * g[7];
        const double dpsi2 = psi * g[8];
        e[d] = (((g[4] - dKE) - dpre_B) - g[0] * inte) - dpsi2;
    }
    over_rho(e);
    const double ux = a[0], uy = a[3], vx = a[1], vy = a[4], wx = a[2], wy = a[5];
    const double Bxy = nQ[14], Byx = nQ[6], Bzx = nQ[7], Bzy = nQ[16];
    const double F1 = mu * (2.0 * ux + kLambdaVisc * (ux + vy)), F2 = mu * (vx + uy), F3 = mu * wx;
    const double G2 = mu * (2.0 * vy + kLambdaVisc * (ux + vy)), G3 = mu * wy;
    double h[2] = {mu * kGam * e[0], mu * kGam * e[1]};
    if constexpr (EX) {
        quotients<2>(h, kPrandtl, h);
    } else {
        h[0] = h[0] * (1.0 / kPrandtl);
        h[1] = h[1] * (1.0 / kPrandtl);
    }
    double F4 = ((u * F1 + v * F2) + w * F3) + h[0];
    double G4 = ((F2 * u + G2 * v) + G3 * w) + h[1];
    const double Jx = Bzy - 0.0, Jy = 0.0 - Bzx, Jz = Byx - Bxy;
    const double F6 = eta0 * Jz, F7 = -(eta0 * Jy);
    F4 = (F4 + F6 * By) + F7 * Bz;
    const double G5 = -(eta0 * Jz), G7 = eta0 * Jx;
    G4 = (G4 + G5 * Bx) + G7 * Bz;
    o[0] = F1 * n0 + F2 * n1;
    o[1] = F2 * n0 + G2 * n1;
    o[2] = F3 * n0 + G3 * n1;
    o[3] = F4 * n0 + G4 * n1;
    o[4] = G5 * n1;
    o[5] = F6 * n0;
    o[6] = F7 * n0 + G7 * n1;
}

// internal energy at a face-averaged state (compflux.f90:272-277)
__device__ __forceinline__ double enei_of(const double *q)
{
    const double a = q[1] / q[0], b = q[2] / q[0], c = q[3] / q[0];
    return (((q[4] / q[0] - 0.5 * (a * a)) - 0.5 * (b * b)) - 0.5 * (c * c)) -
           0.5 * (((q[5] * q[5] + q[6] * q[6]) + q[7] * q[7]) + q[8] * q[8]) / q[0];
}

// Shared memory of both kernels, in doubles: the state slice, the packed
// metric records, the neighbours' traces (type T), then in the gradient
// kernel the exchanged sums, which become the gradients, and over the
// earlier regions the gradients' traces; in the flux kernel the gradients,
// the neighbours' gradient traces (then the exchanged sums) and, for cells
// at a wall, the internal-energy gradient.
template <int N, int CPB, typename T> struct ViscSmem {
    static constexpr int NQ = 9 * N * N, NN = N * N;
    static constexpr bool kPad = N % 2 == 0;  // two doubles per cell against bank conflicts
    static constexpr int QS = kPad ? NQ + 2 : NQ;
    static constexpr int MS = MetLayout<N>::kSize;
    static constexpr int TFS = trace_stride<N, T>();
    static constexpr int TS = 4 * TFS + 16 / (int)sizeof(T);  // in T
    static constexpr int GF = 18 * N;                          // a face's gradient trace record
    static constexpr int GTS = 4 * GF + 2;                     // per cell
    static constexpr int GS = 18 * NN + 2;                     // gradients per cell
    static constexpr int NX = 7;                               // flux sums exchanged per point
    static constexpr int kIn = CPB * (QS + MS) + CPB * TS * (int)sizeof(T) / 8;  // doubles of the first three regions
    static constexpr int kGradIn = kIn > CPB * GTS ? kIn : CPB * GTS;
    static constexpr size_t kGradBytes = 8 * (size_t)(kGradIn + CPB * GS);
    static constexpr size_t kFluxBytes = 8 * (size_t)(kIn + CPB * (GS + GTS + 2 * NN));
    static_assert(NX * NN <= GTS, "the exchanged sums fit the gradient traces' region");
};
// cells per CTA: the stage's (at N = 4, 8 cells leave 6 warps per SM and 4
// cells 7, but with twice the bank conflicts: 38 and 41 us, 58 and 60 with the
// ends peeled)
__host__ __device__ constexpr int visc_cells(int n) { return line_tile_cells(n); }
template <int N, int CPB, size_t SMEM> constexpr int visc_min_blocks()
{
    // 8 warps of 255 registers per SM, 12 of 168 where those hold a line (at N = 2
    // 16 of 128 left 92 bytes of spills: us per stage of the chain, exact, 64 cells
    // 20.8 and 20.3 so, 14400 cells 50.3 and 49.1)
    const int w = (N >= 4 ? 8 : 12) / (line_threads(N, CPB) / 32), m = (int)(228 * 1024 / (SMEM + 1280));
    const int b = w < m ? w : m;
    return b < 1 ? 1 : b;
}

// the 18 gradient components of a point in shared memory (16-byte aligned),
// two at a time
__device__ __forceinline__ void load18(const double *p, double *g)
{
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const double2 v = reinterpret_cast<const double2 *>(p)[k];
        g[2 * k] = v.x;
        g[2 * k + 1] = v.y;
    }
}
__device__ __forceinline__ void store18(double *p, const double *g)
{
#pragma unroll
    for (int k = 0; k < 9; k++) reinterpret_cast<double2 *>(p)[k] = make_double2(g[2 * k], g[2 * k + 1]);
}

// what both kernels share: a thread's line, the staging, and the
// face-averaged state at a flux point of the line
template <int N, int CPB, typename T> struct ViscTile {
    using S = ViscSmem<N, CPB, T>;
    using ML = MetLayout<N>;
    static constexpr int NT = line_threads(N, CPB);
    const ViscArgs &a;
    const Ops &ops;
    double *sQ, *sMet;
    T *sT;
    int c0, ncl, fam, c, l, lf0, lfN, np0, npN;
    bool act;
    int2 rec0, recN;
    unsigned cbytes;

    __device__ __forceinline__ ViscTile(const ViscArgs &a_, const Ops &o_, double *base)
        : a(a_), ops(o_), sQ(base), sMet(base + CPB * S::QS), sT(reinterpret_cast<T *>(base + CPB * (S::QS + S::MS)))
    {
        const int tid = threadIdx.x;
        c0 = blockIdx.x * CPB;
        ncl = min(CPB, a.ncell - c0);
        fam = tid >= N * CPB ? 1 : 0;
        const int lt = tid - fam * N * CPB, lc = lt % CPB;
        act = tid < 2 * N * CPB && lc < ncl;
        c = act ? lc : 0;
        l = act ? lt / CPB : 0;
        lf0 = fam == 0 ? 4 : 1;
        lfN = fam == 0 ? 2 : 3;
        np0 = fam == 0 ? N - 1 - l : l;
        npN = fam == 0 ? l : N - 1 - l;
        rec0 = recN = make_int2(0, 0);
        if (act) {
            rec0 = __ldg(a.faces + (size_t)(c0 + c) * 4 + lf0 - 1);
            recN = __ldg(a.faces + (size_t)(c0 + c) * 4 + lfN - 1);
        }
        cbytes = (unsigned)((S::kPad ? 1 : ncl) * S::NQ * sizeof(double));
    }
    // bytes of each pair face's record of PER values of type V from src to dst
    // (cell stride DS), by asynchronous copies
    template <typename V, int PER, int DS> __device__ __forceinline__ void fetch_faces(V *dst, const V *src)
    {
        constexpr int CH = PER * (int)sizeof(V) / 16, E = 16 / (int)sizeof(V), IT = (CPB * 4 * CH + NT - 1) / NT;
        static_assert(PER * sizeof(V) % 16 == 0, "whole 16-byte units");
        constexpr int B = IT < 9 ? IT : 9;  // records loaded ahead of their copies
#pragma unroll 1
        for (int m0 = 0; m0 < IT; m0 += B) {
            int2 r[B];
#pragma unroll
            for (int m = 0; m < B; m++) {
                const int f = ((int)threadIdx.x + (m0 + m) * NT) / CH;
                r[m] = f < ncl * 4 ? __ldg(a.faces + (size_t)c0 * 4 + f) : make_int2(0, 0);
            }
#pragma unroll
            for (int m = 0; m < B; m++) {
                const int e = (int)threadIdx.x + (m0 + m) * NT, f = e / CH, ch = e - f * CH, kd = r[m].y & 0xff;
                if (kd == kFaceLeft || kd == kFaceRight)
                    cp_async16(dst + (f >> 2) * DS + (f & 3) * PER + ch * E,
                               src + ((size_t)r[m].x * 4 + ((r[m].y >> 8) & 0xff) - 1) * PER + ch * E);
            }
        }
    }
    // stages the state, the metrics, the traces and (g null: not) the
    // gradients and their neighbours' traces; false if the copies timed out
    __device__ __forceinline__ bool stage(const double *g, double *sG, const double *gt, double *sGT)
    {
        __shared__ __align__(8) unsigned long long sBar;
        __shared__ int sAbort;
        const int tid = threadIdx.x;
        const double *qsrc = a.q + (size_t)c0 * S::NQ;
        const bool bulk = (((uintptr_t)qsrc | cbytes) & 15) == 0;
        if (tid < 32) {
            if (tid == 0) {
                sAbort = 0;
                mbar_init(&sBar, 1);
                mbar_expect_tx(&sBar, (unsigned)(ncl * (S::MS + (bulk ? S::NQ : 0) + (g ? 18 * S::NN : 0)) * sizeof(double)));
                bulk_g2s(sMet, a.met + (size_t)c0 * S::MS, (unsigned)(ncl * S::MS * sizeof(double)), &sBar);
            }
            __syncwarp();
            grid_dependency_wait();
            if (bulk && tid < (S::kPad ? ncl : 1)) bulk_g2s(sQ + tid * S::QS, qsrc + (size_t)tid * S::NQ, cbytes, &sBar);
            if (g && tid < ncl)
                bulk_g2s(sG + tid * S::GS, g + (size_t)(c0 + tid) * 18 * S::NN, 18 * S::NN * sizeof(double), &sBar);
        }
        grid_dependency_wait();
        grid_launch_dependents();
        fetch_faces<T, S::TFS, S::TS>(sT, reinterpret_cast<const T *>(a.t_in));
        if (g) fetch_faces<double, S::GF, S::GTS>(sGT, gt);
        if (!bulk)
            for (int k = tid; k < ncl * S::NQ; k += NT) {
                const int cc = k / S::NQ;
                sQ[cc * S::QS + (k - cc * S::NQ)] = qsrc[k];
            }
        cp_async_wait_all();
        if (tid == 0 && !mbar_wait_bounded(&sBar, 0)) {
            raise_fault(a.err_flags, kErrStagingTimeout);
            sAbort = 1;
            mbar_wait_bounded(&sBar, 0);
        }
        __syncthreads();
        return !sAbort;
    }
    __device__ __forceinline__ void normal(int r, double &n0, double &n1) const
    {
        const double2 n = *reinterpret_cast<const double2 *>(sMet + c * S::MS + ML::normal(fam, l, r));
        n0 = n.x;
        n1 = n.y;
    }
    // the interpolated state at flux point r
    __device__ __forceinline__ void own_state(int r, double *q) const
    {
        int q0 = c * S::QS + (fam == 0 ? 9 * N * l : 9 * l);
        asm volatile("" : "+r"(q0));  // read anew at every point: the registers hold sums
        const int str = fam == 0 ? 9 : 9 * N;
#pragma unroll
        for (int k = 0; k < 9; k++) q[k] = 0.0;
#pragma unroll
        for (int s = 0; s < N; s++) {
            const double L = ops.L[r * N + s];
#pragma unroll
            for (int k = 0; k < 9; k++) q[k] = q[k] + sQ[q0 + str * s + k] * L;
        }
    }
    // the face-averaged state from the own trace, at the line's end r (0 or N)
    __device__ __forceinline__ void face_average(int r, double *q) const
    {
        const int2 rec = r == 0 ? rec0 : recN;
        const int lf = r == 0 ? lf0 : lfN, np = r == 0 ? np0 : npN, kind = rec.y & 0xff;
        double oth[9];
        if (kind == kFaceLeft || kind == kFaceRight) {
            const T *tp = sT + c * S::TS + (lf - 1) * S::TFS + (N - 1 - np);
#pragma unroll
            for (int k = 0; k < 9; k++) oth[k] = (double)tp[k * N];
        } else {
            double n0, n1;
            normal(r, n0, n1);
            bc_ghost<double, true>(kind, q, n0, n1, a.vismode, a.fs, oth);
        }
#pragma unroll
        for (int k = 0; k < 9; k++) q[k] = 0.5 * q[k] + 0.5 * oth[k];
    }
    // point t of the line, and the parity of the points this thread finishes
    __device__ __forceinline__ int point(int t) const { return (fam == 0 ? N * l : l) + (fam == 0 ? 1 : N) * t; }
    __device__ __forceinline__ int parity() const { return (l ^ fam) & 1; }
};

// f(r) at every flux point of the line.  ROLLED: one body for the ends and the
// points between them.  The chain's three kernels with the ends peeled do not fit
// the instruction cache together, and each launch fetches its own again: us per
// stage of the chain, peeled and rolled, exact, 8100 cells, N = 4 103 and 83, N = 5
// 168 and 152; FP64, 14400 cells, N = 4 127 and 121.  Where the sums fit the
// registers of three warps anyway (N = 2 and 3 outside the exact form) that
// shows on meshes of one wave only (64 cells, N = 3 24 and 22; 8100 cells 46 and 47),
// and at N = 6 the peeled ends give more than they cost (FP64, 14400 cells 315 and
// 331).
template <int N, bool ROLLED, typename F> __device__ __forceinline__ void along_line(F f)
{
    if constexpr (!ROLLED) {
        f(0);
#pragma unroll 1
        for (int r = 1; r < N; r++) f(r);
        f(N);
    } else {
#pragma unroll 1
        for (int r = 0; r <= N; r++) f(r);
    }
}

// ---- gradients at the solution points and their face traces ------------------------
// T: the trace type of the form (EX and T keep the instantiations of the
// translation units apart)
template <int N, bool EX, typename T, int CPB, bool ROLLED>
__global__ void __launch_bounds__(line_threads(N, CPB), (visc_min_blocks<N, CPB, ViscSmem<N, CPB, T>::kGradBytes>()))
    visc_grad_kernel(const ViscArgs a, const Ops ops)
{
    using S = ViscSmem<N, CPB, T>;
    using ML = MetLayout<N>;
    constexpr int NH = (N + 1) / 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *base = reinterpret_cast<double *>(smem_raw);
    double *sX = base + S::kGradIn;  // [CPB][GS]
    ViscTile<N, CPB, T> t(a, ops, base);
    if (!t.stage(nullptr, nullptr, nullptr, nullptr)) return;

    // nablaQsp (compflux.f90:107-157): this line's sums
    double gx[N][9], gy[N][9];
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int k = 0; k < 9; k++) gx[i][k] = gy[i][k] = 0.0;
    if (t.act) {
        auto add = [&](int r) {
            double V[9], n0, n1;
            t.own_state(r, V);
            t.normal(r, n0, n1);
            if (r == 0 || r == N) t.face_average(r, V);
#pragma unroll
            for (int i = 0; i < N; i++) {
                const double M = ops.M[r * N + i];
#pragma unroll
                for (int k = 0; k < 9; k++) {
                    const double m = V[k] * M;
                    gx[i][k] = gx[i][k] + m * n0;
                    gy[i][k] = gy[i][k] + m * n1;
                }
            }
        };
        along_line<N, ROLLED>(add);
    }
    const int par = t.parity();
    if (t.act) {
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (2 * m + 1 < N || par) {
                double o[18];
#pragma unroll
                for (int k = 0; k < 9; k++) {
                    o[k] = par ? gx[i0][k] : gx[i1][k];
                    o[9 + k] = par ? gy[i0][k] : gy[i1][k];
                }
                store18(sX + t.c * S::GS + t.point(2 * m + 1 - par) * 18, o);
            }
        }
    }
    __syncthreads();
    if (t.act) {
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (!(2 * m + 1 < N) && par) continue;
            const int pt = t.point(2 * m + par);
            double *x = sX + t.c * S::GS + pt * 18;
            const double J = t.sMet[t.c * S::MS + ML::kJac + pt];
            double g[18];
            load18(x, g);
#pragma unroll
            for (int k = 0; k < 9; k++) {
                g[k] = (par ? gx[i1][k] : gx[i0][k]) + g[k];
                g[9 + k] = (par ? gy[i1][k] : gy[i0][k]) + g[9 + k];
            }
            if constexpr (EX) {
                quotients<18>(g, J, g);
            } else {
                const double rJ = 1.0 / J;
#pragma unroll
                for (int k = 0; k < 18; k++) g[k] = g[k] * rJ;
            }
            store18(x, g);
        }
    }
    fence_proxy_async();
    __syncthreads();
    if ((int)threadIdx.x < t.ncl)
        bulk_s2g(a.grad + (size_t)(t.c0 + threadIdx.x) * 18 * S::NN, sX + threadIdx.x * S::GS, 18 * S::NN * sizeof(double));
    // the gradients' traces at the line's ends (the same interpolation)
    if (t.act) {
        double e0[18], eN[18];
#pragma unroll
        for (int k = 0; k < 18; k++) e0[k] = eN[k] = 0.0;
#pragma unroll
        for (int s = 0; s < N; s++) {
            double g[18];
            load18(sX + t.c * S::GS + t.point(s) * 18, g);
            const double L0 = ops.L[s], LN = ops.L[N * N + s];
#pragma unroll
            for (int k = 0; k < 18; k++) {
                e0[k] = e0[k] + g[k] * L0;
                eN[k] = eN[k] + g[k] * LN;
            }
        }
        double *o0 = base + t.c * S::GTS + (t.lf0 - 1) * S::GF + t.np0, *oN = base + t.c * S::GTS + (t.lfN - 1) * S::GF + t.npN;
#pragma unroll
        for (int k = 0; k < 18; k++) {
            o0[k * N] = e0[k];
            oN[k * N] = eN[k];
        }
    }
    fence_proxy_async();
    __syncthreads();
    if (threadIdx.x < 32) {
        if ((int)threadIdx.x < t.ncl)
            bulk_s2g(a.gt + (size_t)(t.c0 + threadIdx.x) * 4 * S::GF, base + threadIdx.x * S::GTS, 4 * S::GF * sizeof(double));
        bulk_wait_read();
    }
}

// ---- the viscous flux and its divergence ---------------------------------------------
template <int N, bool EX, typename T, int CPB, bool ROLLED>
__global__ void __launch_bounds__(line_threads(N, CPB), (visc_min_blocks<N, CPB, ViscSmem<N, CPB, T>::kFluxBytes>()))
    visc_flux_kernel(const ViscArgs a, const Ops ops)
{
    using S = ViscSmem<N, CPB, T>;
    constexpr int NN = S::NN, NH = (N + 1) / 2, NX = S::NX;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *base = reinterpret_cast<double *>(smem_raw);
    double *sG = base + S::kIn;         // [CPB][GS] gradients
    double *sGT = sG + CPB * S::GS;     // [CPB][GTS] neighbours' gradient traces, then exchanged sums
    double *sDE = sGT + CPB * S::GTS;   // [CPB][NN][2] internal-energy gradient of cells at a wall
    ViscTile<N, CPB, T> t(a, ops, base);
    if (!t.stage(a.grad, sG, a.gt, sGT)) return;

    // comp_grad_internal_energy (compflux.f90:260-298) for cells with a wall
    // face (the only ones whose values are read)
    bool wall = false;
    if (t.act)
        for (int f = 0; f < 4; f++) wall |= (__ldg(a.faces + (size_t)(t.c0 + t.c) * 4 + f).y & 0xff) == kFaceWall;
    if (__syncthreads_or(wall)) {
        if (wall) {
            double de[N];
#pragma unroll
            for (int i = 0; i < N; i++) de[i] = 0.0;
#pragma unroll 1
            for (int r = 0; r <= N; r++) {
                double V[9];
                t.own_state(r, V);
                if (r == 0 || r == N) t.face_average(r, V);
                const double e = enei_of(V);
#pragma unroll
                for (int i = 0; i < N; i++) de[i] = de[i] + e * ops.M[r * N + i];
            }
#pragma unroll
            for (int i = 0; i < N; i++) sDE[(t.c * NN + t.point(i)) * 2 + t.fam] = de[i];
        }
        __syncthreads();
    }

    double d[N][NX];
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int k = 0; k < NX; k++) d[i][k] = 0.0;
    if (t.act) {
        auto add = [&](int r) {
            double V[9], g[18], n0, n1;
            t.own_state(r, V);
            t.normal(r, n0, n1);
            {
                int g0 = t.c * S::GS + t.point(0) * 18;
                asm volatile("" : "+r"(g0));  // read anew at every point
                const int str = t.fam == 0 ? 18 : 18 * N;
#pragma unroll
                for (int k = 0; k < 18; k++) g[k] = 0.0;
#pragma unroll
                for (int s = 0; s < N; s++) {
                    const double L = ops.L[r * N + s];
                    double x[18];
                    load18(sG + g0 + str * s, x);
#pragma unroll
                    for (int k = 0; k < 18; k++) g[k] = g[k] + x[k] * L;
                }
            }
            if (r == 0 || r == N) {
                // the average of both sides' gradients (interfaceVISflux,
                // CYCLOCVISFLUX), or of the own and the boundary's (BCVISFLUX)
                const int2 rec = r == 0 ? t.rec0 : t.recN;
                const int lf = r == 0 ? t.lf0 : t.lfN, np = r == 0 ? t.np0 : t.npN, kind = rec.y & 0xff;
                if (kind == kFaceLeft || kind == kFaceRight) {
                    const double *tp = sGT + t.c * S::GTS + (lf - 1) * S::GF + (N - 1 - np);
#pragma unroll
                    for (int k = 0; k < 18; k++) g[k] = 0.5 * g[k] + 0.5 * tp[k * N];
                } else {
                    double o4[2] = {g[4], g[13]};
                    if (kind == kFaceWall) {
                        // adiabatic wall: the boundary energy gradient
                        // (bcflux.f90:469-583); V is still the own trace
                        double dxi = 0.0, deta = 0.0;
#pragma unroll
                        for (int s = 0; s < N; s++) {
                            const double *de = sDE + (t.c * NN + t.point(s)) * 2;
                            dxi = dxi + de[0] * ops.L[r * N + s];
                            deta = deta + de[1] * ops.L[r * N + s];
                        }
                        const double *m2 = a.met2 + (((size_t)(t.c0 + t.c) * 4 + (lf - 1)) * N + np) * 2;
                        const double ur = V[1] / V[0], vr = V[2] / V[0], wr = V[3] / V[0];
                        const double inte = (V[4] / V[0] - 0.5 * ((ur * ur + vr * vr) + wr * wr)) -
                                            0.5 * (((V[5] * V[5] + V[6] * V[6]) + V[7] * V[7]) + V[8] * V[8]) / V[0];
                        // dBp of both directions is the first direction's (bcflux.f90:563)
                        const double dBp = ((V[5] * g[5] + V[6] * g[6]) + V[7] * g[7]) + V[8] * g[8];
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const double *gd = g + 9 * e;
                            const double dur = (gd[1] - ur * gd[0]) / V[0];
                            const double dvr = (gd[2] - vr * gd[0]) / V[0];
                            const double dwr = (gd[3] - wr * gd[0]) / V[0];
                            const double dKE =
                                0.5 * ((ur * ur + vr * vr) + wr * wr) * gd[0] + V[0] * ((ur * dur + vr * dvr) + wr * dwr);
                            // the ghost family's other normal row: S1(2,e) on xi
                            // faces, S2(1,e) on eta faces; the energy gradient along it
                            const double tw = t.fam == 0 ? 2.0 * deta * m2[e] * V[0] : 2.0 * dxi * m2[e] * V[0];
                            o4[e] = (((-gd[4] + 2.0 * inte * gd[0]) + 2.0 * dKE) + dBp) + tw;
                        }
                    }
                    // the other components' boundary gradients are the own ones
                    const double g4 = g[4], g13 = g[13];
#pragma unroll
                    for (int k = 0; k < 18; k++) g[k] = 0.5 * g[k] + 0.5 * g[k];
                    g[4] = 0.5 * g4 + 0.5 * o4[0];
                    g[13] = 0.5 * g13 + 0.5 * o4[1];
                }
                t.face_average(r, V);
            }
            double o[NX];
            vflux<EX>(V, g, a.mu, a.eta0, n0, n1, o);
#pragma unroll
            for (int i = 0; i < N; i++) {
                const double M = ops.M[r * N + i];
#pragma unroll
                for (int k = 0; k < NX; k++) d[i][k] = d[i][k] + o[k] * M;
            }
        };
        along_line<N, ROLLED>(add);
    }
    __syncthreads();  // the gradient traces and the states are read
    const int par = t.parity();
    double *sX = sGT;
    if (t.act) {
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (2 * m + 1 < N || par) {
                double *o = sX + t.c * S::GTS + t.point(2 * m + 1 - par) * NX;
#pragma unroll
                for (int k = 0; k < NX; k++) o[k] = par ? d[i0][k] : d[i1][k];
            }
        }
    }
    __syncthreads();
    if (t.act) {
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (!(2 * m + 1 < N) && par) continue;
            const int pt = t.point(2 * m + par);
            const double *x = sX + t.c * S::GTS + pt * NX;
            double *o = t.sQ + t.c * S::QS + 9 * pt;
            o[0] = 0.0;
#pragma unroll
            for (int k = 0; k < NX; k++) o[1 + k] = (par ? d[i1][k] : d[i0][k]) + x[k];
            o[8] = 0.0;
        }
    }
    fence_proxy_async();
    __syncthreads();
    double *dst = a.rv + (size_t)t.c0 * S::NQ;
    if ((((uintptr_t)dst | t.cbytes) & 15) == 0) {
        if (threadIdx.x < 32) {
            if ((int)threadIdx.x < (S::kPad ? t.ncl : 1))
                bulk_s2g(dst + (size_t)threadIdx.x * S::NQ, t.sQ + threadIdx.x * S::QS, t.cbytes);
            bulk_wait_read();
        }
    } else {
        for (int k = threadIdx.x; k < t.ncl * S::NQ; k += line_threads(N, CPB)) {
            const int cc = k / S::NQ;
            dst[k] = t.sQ[cc * S::QS + (k - cc * S::NQ)];
        }
    }
}

}  // namespace sddc
