// Kernels of the discrete adjoint (VJP) of the SDDC residual and RK stage.
//
// For one RK stage out = ... + c R(q) the reverse stage needs
// qbar = (dR/dq)^T lambda with lambda = c * xbar (xbar: adjoint of the stage
// output).  R is the compresid chain (compresid.f90:1-80, compflux.f90,
// interfaceflux_all.f90, cyclocflux_all.f90, bcflux.f90); its linear parts
// (interpolation, flux derivative, metric gradient of B, sources) are
// transposed here by hand, its point functions go through
// adjoint_point.cuh.  The AV sensor enters no residual (its coefficients are
// zero, getrusanov.f90:326,328) and so has no adjoint.
//
// Per reverse stage:
//   adjoint traces    per (cell, face point): the adjoint of the flux value
//                     and of the face-averaged Bx, By that this cell's
//                     residual sees at the face point (its neighbour needs
//                     them: a shared face's flux and average enter both
//                     cells' residuals).  They depend on the cell's own
//                     output adjoint only, which is the previous reverse
//                     stage's out: that stage's vjp_kernel forms them in its
//                     epilogue when it knows this stage's input state, else
//                     adj_trace_kernel does;
//   vjp_kernel        per tile of cells, staged in shared memory: primal
//                     recomputation (traces, divB), the transposed
//                     divergence and gradient, the point adjoints, the
//                     transposed interpolation, the RK reverse update as an
//                     element-wise epilogue, and the next stage's adjoint
//                     traces.
// c_h = sqrt(L (L - U)) is a function of the running maxima L, U of the wave
// speed and velocity over all earlier stages; its adjoint is carried by
// adj_reduce_kernel to the stage and points where the maximum was attained
// (argmax records written by vjp_kernel).
#pragma once

#include "adjoint_point.cuh"
#include "line_kernel.cuh"

namespace sddc {

enum : unsigned { kErrAdjointMaxLost = 4u, kErrAdjointRecords = 8u };

// a point where a running maximum was attained: the gradient of the wave
// speed (kind 0) or velocity maximum (kind 1) there with respect to the
// cell's own flux-point state (slot: (fam*N + line)*(N+1) + r) and to the
// free stream (boundary faces)
struct AdjRec {
    int cell, slot, kind, counted;
    double d[9];
    double p[6];
};

// device-side scalars carried across reverse stages
struct AdjScalars {
    double lam_eig, lam_um;  // adjoints of the running maxima not yet given to their argmax
    double pbar[6];          // adjoint of (rinf, pinf, uinf, vinf, bxinf, byinf)
    double cbar;             // sum over stages of lambda . dR/dc_h
    double ties;             // stages whose raised maximum several points attained
};

struct VjpArgs {
    int ncell, vismode;
    double alpha, c_h;
    Freestream fs;
    const double *__restrict__ q;     // stage input state (9,N,N,NCELL)
    const double *__restrict__ t_in;  // its face traces, layout trace_at
    const double *xbar;               // adjoint of the stage output; null: objective seeds only
    double lam_scale;                 // lambda = lam_scale * xbar
    const double *__restrict__ at;    // adjoint traces, layout adj_trace_at
    const double *__restrict__ met;
    const int2 *__restrict__ faces;
    // epilogue: out = (wa*ra + wb*rb) + qbar;  out2 = wc*rc + wd*xbar
    const double *ra, *rb;
    double wa, wb;
    double *out;
    const double *rc;
    double wc, wd;
    double *out2;
    // objective: adjoint of the wall force (Fx, Fy) at this state
    double sx, sy;
    double wq[kMaxN];
    double *part;  // [8][CTAs]: cbar, pbar[6], 0
    FaultFlags *err;
    // the next reverse stage's adjoint traces, formed from out (the adjoint of
    // that stage's output) in the epilogue: its input state and lam_scale, and
    // the trace buffer (null: its own trace launch forms them)
    const double *q_next;
    double scale_next;
    double *at_next;
};

// ---- adjoint traces ----------------------------------------------------------
// at(cell, lf, nfp) = (Fbar(9), Vbar_Bx, Vbar_By, 0): the adjoint of this
// cell's flux value at the face point (from the divergence, compresid.f90:
// 12-51) and of the face-averaged Bx, By (from divB in the Powell source,
// compresid.f90:58, through nablaQsp compflux.f90:107-157).
constexpr int kTraceCpb = 8;  // cells per CTA of adj_trace_kernel

// adjoint trace layout, [cell][local face][value][face point] like trace_at:
// the N points of a face, which consecutive lanes write and read, are
// adjacent (lf 1-based, nfp0 0-based, 12 values, the last one 0)
template <int N> __host__ __device__ __forceinline__ size_t adj_trace_at(size_t cell, int lf, int nfp0, int k)
{
    return ((cell * 4 + (size_t)(lf - 1)) * 12 + (size_t)k) * N + (size_t)nfp0;
}

template <int N>
__global__ void __launch_bounds__(128) adj_trace_kernel(int ncell, int vismode, const double *__restrict__ xbar,
                                                        double lam_scale, const double *__restrict__ q,
                                                        const double *__restrict__ met, const Ops ops,
                                                        double *__restrict__ at)
{
    using ML = MetLayout<N>;
    constexpr int NQ = 9 * N * N, NN = N * N, CPB = kTraceCpb;
    __shared__ __align__(16) double sMu[CPB * NQ];  // lambda source, then -lambda/J
    __shared__ __align__(16) double sQs[CPB * NQ];  // the state
    __shared__ double sB[CPB * NN];                 // Jac, 1/Jac, then the divB adjoint over Jac
    __shared__ __align__(8) unsigned long long sBar;
    __shared__ int sAbort;
    const int tid = threadIdx.x, c0 = blockIdx.x * CPB, ncl = min(CPB, ncell - c0);
    // the lambda source and state slices by TMA bulk copies when aligned
    const double *xsrc = xbar + (size_t)c0 * NQ, *qsrc = q + (size_t)c0 * NQ;
    const size_t bytes = (size_t)ncl * NQ * sizeof(double);
    const bool bulk = (((uintptr_t)xsrc | (uintptr_t)qsrc | bytes) & 15) == 0;
    if (tid == 0) {
        sAbort = 0;
        if (bulk) {
            mbar_init(&sBar, 1);
            mbar_expect_tx(&sBar, (unsigned)(2 * bytes));
            bulk_g2s(sMu, xsrc, (unsigned)bytes, &sBar);
            bulk_g2s(sQs, qsrc, (unsigned)bytes, &sBar);
        }
    }
    for (int k = tid; k < ncl * NN; k += 128) {
        const int c = k / NN;
        sB[k] = met[(size_t)(c0 + c) * ML::kSize + ML::kJac + (k - c * NN)];
    }
    if (!bulk)
        for (int k = tid; k < ncl * NQ; k += 128) {
            sMu[k] = xsrc[k];
            sQs[k] = qsrc[k];
        }
    if (bulk && tid == 0 && !mbar_wait_bounded(&sBar, 0)) {
        sAbort = 1;  // the copies did not complete; the caller sees stale traces
        mbar_wait_bounded(&sBar, 0);
    }
    __syncthreads();
    if (sAbort) return;
    // per solution point: the divB adjoint from the Powell source
    // (compresid.f90:60-76), over Jac
    double beta[(CPB * NN + 127) / 128];
    for (int k = tid, it = 0; k < ncl * NN; k += 128, it++) {
        const double *x = sMu + 9 * k;
        double db = 0.0;
        if (vismode == 1) {
            const double *qq = sQs + 9 * k;
            const double ri = 1.0 / qq[0], ux = qq[1] * ri, uy = qq[2] * ri, uz = qq[3] * ri;
            db = -lam_scale * (x[1] * qq[5] + x[2] * qq[6] + x[3] * qq[7] +
                               x[4] * ((ux * qq[5] + uy * qq[6]) + uz * qq[7]) + x[5] * ux + x[6] * uy + x[7] * uz);
        }
        const double rJ = 1.0 / sB[k];
        beta[it] = db * rJ;
        sB[k] = rJ;
    }
    __syncthreads();
    for (int k = tid; k < ncl * NQ; k += 128) sMu[k] = -(lam_scale * sMu[k]) * sB[k / 9];
    __syncthreads();
    for (int k = tid, it = 0; k < ncl * NN; k += 128, it++) sB[k] = beta[it];
    __syncthreads();
    // per face point: the transposed flux derivative and B gradient
    for (int t = tid; t < ncl * 4 * N; t += 128) {
        const int c = t / (4 * N), f = t - c * 4 * N;
        const int nfp = 1 + f % N, lf = 1 + f / N;
        int fam, line, r;
        face_point<N>(lf, nfp, fam, line, r);
        double fb[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, bs = 0.0;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int sp = fam == 0 ? i + N * line : line + N * i;
            const double m = ops.M[r * N + i];
            const double *mu = sMu + c * NQ + 9 * sp;
#pragma unroll
            for (int k = 0; k < 9; k++) fb[k] += m * mu[k];
            bs += m * sB[c * NN + sp];
        }
        const double *nr = met + (size_t)(c0 + c) * ML::kSize + ML::normal(fam, line, r);
#pragma unroll
        for (int k = 0; k < 9; k++) at[adj_trace_at<N>(c0 + c, lf, nfp - 1, k)] = fb[k];
        at[adj_trace_at<N>(c0 + c, lf, nfp - 1, 9)] = bs * nr[0];
        at[adj_trace_at<N>(c0 + c, lf, nfp - 1, 10)] = bs * nr[1];
        at[adj_trace_at<N>(c0 + c, lf, nfp - 1, 11)] = 0.0;
    }
}

// The adjoint trace at face point f (0..4N-1) of one cell from global memory,
// in adj_trace_kernel's arithmetic: the reduction uses it to form again the
// next stage's traces of the cells that its records changed.
template <int N>
__device__ void adj_trace_point(size_t cell, int f, const double *xbar, const double *q, double scale,
                                const double *met, int vismode, const Ops &ops, double *at)
{
    using ML = MetLayout<N>;
    constexpr int NQ = 9 * N * N;
    const int nfp = 1 + f % N, lf = 1 + f / N;
    int fam, line, r;
    face_point<N>(lf, nfp, fam, line, r);
    const double *mc = met + cell * ML::kSize;
    double fb[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, bs = 0.0;
    for (int i = 0; i < N; i++) {
        const int sp = fam == 0 ? i + N * line : line + N * i;
        const double *x = xbar + cell * NQ + 9 * sp;
        double db = 0.0;
        if (vismode == 1) {
            const double *qq = q + cell * NQ + 9 * sp;
            const double ri = 1.0 / qq[0], ux = qq[1] * ri, uy = qq[2] * ri, uz = qq[3] * ri;
            db = -scale * (x[1] * qq[5] + x[2] * qq[6] + x[3] * qq[7] + x[4] * ((ux * qq[5] + uy * qq[6]) + uz * qq[7]) +
                           x[5] * ux + x[6] * uy + x[7] * uz);
        }
        const double rJ = 1.0 / mc[ML::kJac + sp];
        const double m = ops.M[r * N + i];
        for (int k = 0; k < 9; k++) fb[k] += m * (-(scale * x[k]) * rJ);
        bs += m * (db * rJ);
    }
    const double *nr = mc + ML::normal(fam, line, r);
    for (int k = 0; k < 9; k++) at[adj_trace_at<N>(cell, lf, nfp - 1, k)] = fb[k];
    at[adj_trace_at<N>(cell, lf, nfp - 1, 9)] = bs * nr[0];
    at[adj_trace_at<N>(cell, lf, nfp - 1, 10)] = bs * nr[1];
    at[adj_trace_at<N>(cell, lf, nfp - 1, 11)] = 0.0;
}

// ---- running-max argmax records ----------------------------------------------------
// where the records go (passed by value: the out-of-line record path must
// not copy the kernel's argument block)
struct RecSink {
    AdjRec *recs;
    int cap;
    int *n;
    int *cnt;
    FaultFlags *err;
};

static __device__ __noinline__ void adj_record(RecSink rs, int cell, int slot, int kind, int counted, const double *d,
                                        const double *p)
{
    const int k = atomicAdd(rs.n, 1);
    if (k < rs.cap) {
        AdjRec &R = rs.recs[k];
        R.cell = cell;
        R.slot = slot;
        R.kind = kind;
        R.counted = counted;
        for (int m = 0; m < 9; m++) R.d[m] = d[m];
        for (int m = 0; m < 6; m++) R.p[m] = p ? p[m] : 0.0;
    } else {
        raise_fault(rs.err, kErrAdjointRecords);
    }
    if (counted) atomicAdd(rs.cnt + kind, 1);
}

// a face point whose wave speed (hit_eig) or velocity maximum (hit_um)
// equals the stage's new running max: the gradient of that value with
// respect to this cell's trace (and the free stream, through a ghost
// state); a shared face is counted by its left cell only
static __device__ __noinline__ void adj_record_face(RecSink rs, Freestream fs, int vismode, double c_h, bool hit_eig,
                                             bool hit_um, int cell, int slot, int kind, bool own_right,
                                             const double *own, const double *oth, double n0, double n1, int sign_l)
{
    const bool pair = kind == kFaceLeft || kind == kFaceRight;
    const double *ql = own_right ? oth : own, *qr = own_right ? own : oth;
    const double z[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int kk = 0; kk < 2; kk++) {
        if (!(kk == 0 ? hit_eig : hit_um)) continue;
        double d[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, dg[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, p[6] = {0, 0, 0, 0, 0, 0};
        double e2, u2;
        if (pair) {
            rusanov_vjp(ql, qr, n0, n1, sign_l, c_h, z, kk == 0 ? 1.0 : 0.0, kk == 1 ? 1.0 : 0.0,
                        own_right ? nullptr : d, own_right ? d : nullptr, e2, u2);
        } else {
            rusanov_vjp(own, oth, n0, n1, sign_l, c_h, z, kk == 0 ? 1.0 : 0.0, kk == 1 ? 1.0 : 0.0, d, dg, e2, u2);
            bc_ghost_vjp(kind, own, n0, n1, vismode, fs, dg, d, p);
        }
        adj_record(rs, cell, slot, kk, own_right ? 0 : 1, d, p);
    }
}

// ---- the stage VJP -------------------------------------------------------------
// One thread per line of solution points, as the forward stage works
// (line_kernel.cuh).  At every flux point of its line, one after the other,
// the thread forms the primal state and the flux adjoint (the transposed flux
// derivative) from the states and -lambda/J of the line, applies the point
// adjoint and adds its share of the transposed interpolation to N*9 sums in
// registers; the two lines through a point exchange their sums once.
//
// What bounds it: latency, at 2 warps of up to 255 registers per scheduler
// (a line's sums, a point's state, flux adjoint and state adjoint, and the
// Rusanov adjoint's own values); the states are read from shared memory at
// every flux point.  One thread per point and variable, every operand through
// shared memory, 4 CTAs of 4 warps per SM: 64 us at 64x128 cells, N = 4, and
// 144 ms for the reverse sweep of 100 steps at 128x256; by lines 53 us and
// 122 ms.
template <int N> struct VjpSmem {
    static constexpr int CPB = line_tile_cells(N);
    static constexpr int NQ = 9 * N * N, NN = N * N;
    static constexpr bool kPad = N % 2 == 0;  // two doubles per cell against bank conflicts
    static constexpr int QS = kPad ? NQ + 2 : NQ;
    static constexpr int MS = MetLayout<N>::kSize;
    static constexpr int TFS = trace_stride<N, double>();
    static constexpr int TS = 4 * TFS + 2;
    static constexpr int AF = 12 * N;          // a face's adjoint trace record
    static constexpr int AS = 4 * AF + 2;      // per cell
    static constexpr int XS = 9 * NN + 1;      // exchanged sums per cell, over the traces
    static_assert(XS <= TS + AS, "the exchanged sums fit the traces' region");
    static constexpr size_t kBytes =
        8 * ((size_t)CPB * (2 * QS + MS + TS + AS + NN) + 2 * 2 * line_threads(N, CPB) + 8 * 32);
};
template <int N> constexpr int vjp_min_blocks()
{
    const int w = (N >= 4 ? 8 : N == 3 ? 9 : 12) / (line_threads(N, VjpSmem<N>::CPB) / 32);
    const int m = (int)(228 * 1024 / (VjpSmem<N>::kBytes + 1280));
    const int b = w < m ? w : m;
    return b < 1 ? 1 : b;
}

// a boundary face point (rare): the own trace's adjoint of its flux and
// average, through the ghost state, and the free stream's; out of line
static __device__ __noinline__ double vjp_boundary(int kind, const double *own, const double *oth, double n0, double n1,
                                                   int sign_l, int vismode, Freestream fs, double c_h, const double *fbar,
                                                   const double *fown, double vbx, double vby, double *qown, double *pb)
{
    double qgb[9] = {0, 0, 0, 0, 0, 0.5 * vbx, 0.5 * vby, 0, 0}, eig, um;
    const double wdc =
        rusanov_vjp(own, oth, n0, n1, sign_l, c_h, fbar, 0.0, 0.0, qown, qgb, eig, um, nullptr, fown);
    bc_ghost_vjp(kind, own, n0, n1, vismode, fs, qgb, qown, pb);
    return wdc;
}
static __device__ __noinline__ void vjp_ghost(int kind, const double *own, double n0, double n1, int vismode, Freestream fs,
                                              double *oth)
{
    bc_ghost<double, true>(kind, own, n0, n1, vismode, fs, oth);
}

template <int N>
__global__ void __launch_bounds__(line_threads(N, VjpSmem<N>::CPB), (vjp_min_blocks<N>()))
    vjp_kernel(const VjpArgs a, const Ops ops)
{
    using S = VjpSmem<N>;
    using ML = MetLayout<N>;
    constexpr int CPB = S::CPB, NT = line_threads(N, CPB), NQ = S::NQ, NN = S::NN, QS = S::QS, NH = (N + 1) / 2;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *sQ = reinterpret_cast<double *>(smem_raw);  // [CPB][QS] q, then qbar, then out
    double *sA = sQ + CPB * QS;                         // [CPB][QS] lambda, then -lambda/J, then the next stage's q
    double *sMet = sA + CPB * QS;                       // [CPB][MS] normals, Jac
    double *sT = sMet + CPB * S::MS;                    // [CPB][TS] neighbours' (or ghost) traces
    double *sAT = sT + CPB * S::TS;                     // [CPB][AS] neighbours' adjoint traces
    double *sX = sT;                                    // [CPB][XS] exchanged sums, over both
    double *sBeta = sAT + CPB * S::AS;                  // [CPB][NN] div B sums, then the adjoint of div B over J
    double2 *sP = reinterpret_cast<double2 *>(sBeta + CPB * NN);  // [2][NT] partners' normals at the line's ends
    double *sRed = reinterpret_cast<double *>(sP + 2 * NT);       // [8][32]
    __shared__ __align__(8) unsigned long long sBar, sBarN;
    __shared__ int sAbort;

    const int tid = threadIdx.x, c0 = blockIdx.x * CPB, ncl = min(CPB, a.ncell - c0);
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
    const int par = (l ^ fam) & 1;                                 // this thread finishes points t with t + par even

    // ---- staging --------------------------------------------------------------------
    const double *qsrc = a.q + (size_t)c0 * NQ, *xsrc = a.xbar ? a.xbar + (size_t)c0 * NQ : nullptr;
    const unsigned cbytes = (unsigned)((S::kPad ? 1 : ncl) * NQ * sizeof(double));
    const bool bulk = (((uintptr_t)qsrc | (uintptr_t)xsrc | cbytes) & 15) == 0;
    if (tid < 32) {
        if (tid == 0) {
            sAbort = 0;
            mbar_init(&sBar, 1);
            mbar_init(&sBarN, 1);
            mbar_expect_tx(&sBar, (unsigned)((ncl * S::MS + (bulk ? ncl * NQ * (xsrc ? 2 : 1) : 0)) * sizeof(double)));
            bulk_g2s(sMet, a.met + (size_t)c0 * S::MS, (unsigned)(ncl * S::MS * sizeof(double)), &sBar);
        }
        __syncwarp();
        if (bulk && tid < (S::kPad ? ncl : 1)) {
            bulk_g2s(sQ + tid * QS, qsrc + (size_t)tid * NQ, cbytes, &sBar);
            if (xsrc) bulk_g2s(sA + tid * QS, xsrc + (size_t)tid * NQ, cbytes, &sBar);
        }
        // L2 prefetches of the RK registers the epilogue reads
        if (tid < 3) {
            const double *r = tid == 0 ? a.ra : tid == 1 ? a.rb : a.out2 ? a.rc : nullptr;
            const unsigned n = (unsigned)((size_t)ncl * NQ * sizeof(double));
            if (r && (((uintptr_t)(r + (size_t)c0 * NQ) | n) & 15) == 0) bulk_prefetch_l2(r + (size_t)c0 * NQ, n);
        }
    }
    // the neighbours' traces and adjoint traces, 16 bytes of a face at a time
    {
        constexpr int CT = S::TFS / 2, CA = S::AF / 2, IT = (CPB * 4 * (CT + CA) + NT - 1) / NT, B = IT < 8 ? IT : 8;
#pragma unroll 1
        for (int m0 = 0; m0 < IT; m0 += B) {
            int2 r[B];
#pragma unroll
            for (int m = 0; m < B; m++) {
                const int f = (tid + (m0 + m) * NT) / (CT + CA);
                r[m] = f < ncl * 4 ? __ldg(a.faces + (size_t)c0 * 4 + f) : make_int2(0, 0);
            }
#pragma unroll
            for (int m = 0; m < B; m++) {
                const int e = tid + (m0 + m) * NT, f = e / (CT + CA), ch = e - f * (CT + CA), kd = r[m].y & 0xff;
                if (kd != kFaceLeft && kd != kFaceRight) continue;
                const size_t pf = (size_t)r[m].x * 4 + ((r[m].y >> 8) & 0xff) - 1;
                if (ch < CT)
                    cp_async16(sT + (f >> 2) * S::TS + (f & 3) * S::TFS + 2 * ch, a.t_in + pf * S::TFS + 2 * ch);
                else if (a.xbar)
                    cp_async16(sAT + (f >> 2) * S::AS + (f & 3) * S::AF + 2 * (ch - CT), a.at + pf * S::AF + 2 * (ch - CT));
            }
        }
    }
    auto fetch_pn = [&](const int2 rec, int np, double2 *dst) {
        if ((rec.y & 0xff) != kFaceRight) return;
        int pfam, pline, pr;
        face_point<N>((rec.y >> 8) & 0xff, N - np, pfam, pline, pr);
        cp_async_pair(dst, reinterpret_cast<const double2 *>(a.met + (size_t)rec.x * S::MS + ML::normal(pfam, pline, pr)));
    };
    if (act) {
        fetch_pn(rec0, np0, sP + tid);
        fetch_pn(recN, npN, sP + NT + tid);
    }
    if (!bulk)
        for (int k = tid; k < ncl * NQ; k += NT) {
            const int cc = k / NQ, o = cc * QS + (k - cc * NQ);
            sQ[o] = qsrc[k];
            if (xsrc) sA[o] = xsrc[k];
        }
    cp_async_wait_all();
    if (tid == 0 && !mbar_wait_bounded(&sBar, 0)) {
        raise_fault(a.err, kErrStagingTimeout);  // the copies did not complete
        sAbort = 1;
        mbar_wait_bounded(&sBar, 0);
    }
    __syncthreads();
    if (sAbort) return;

    const int q0 = c * QS + 9 * pt0, qstr = 9 * pts;  // the line's values in sQ and sA
    // the interpolated state at flux point r
    auto own_state = [&](int r, double (&q)[9]) {
        int qi = q0;
        asm volatile("" : "+r"(qi));  // read anew at every point
#pragma unroll
        for (int k = 0; k < 9; k++) q[k] = 0.0;
#pragma unroll
        for (int s = 0; s < N; s++) {
            const double L = ops.L[r * N + s];
#pragma unroll
            for (int k = 0; k < 9; k++) q[k] = q[k] + sQ[qi + qstr * s + k] * L;
        }
    };
    auto normal = [&](int r) { return *reinterpret_cast<const double2 *>(sMet + c * S::MS + ML::normal(fam, l, r)); };
    // the other side's trace at the line's end r: 9 values N apart
    auto other_at = [&](int r) { return sT + c * S::TS + ((r == 0 ? lf0 : lfN) - 1) * S::TFS + (N - 1 - (r == 0 ? np0 : npN)); };
    auto is_pair = [](int kind) { return kind == kFaceLeft || kind == kFaceRight; };

    // ---- primal: ghost traces, and the line's share of div B ---------------------------
    if (act) {
#pragma unroll 1
        for (int r = 0; r <= N; r += N) {
            const int kind = (r == 0 ? rec0 : recN).y & 0xff;
            if (is_pair(kind)) continue;
            double own[9], oth[9];
            own_state(r, own);
            const double2 n = normal(r);
            vjp_ghost(kind, own, n.x, n.y, a.vismode, a.fs, oth);
            double *tp = other_at(r);
            for (int k = 0; k < 9; k++) tp[k * N] = oth[k];
        }
    }
    double dvb[N];  // div B sums (nablaQsp of Bx in x and By in y)
#pragma unroll
    for (int i = 0; i < N; i++) dvb[i] = 0.0;
    if (act && a.vismode == 1) {
#pragma unroll
        for (int r = 0; r <= N; r++) {
            double bx = 0.0, by = 0.0;
#pragma unroll
            for (int s = 0; s < N; s++) {
                bx += sQ[q0 + qstr * s + 5] * ops.L[r * N + s];
                by += sQ[q0 + qstr * s + 6] * ops.L[r * N + s];
            }
            if (r == 0 || r == N) {
                const double *tp = other_at(r);
                bx = 0.5 * bx + 0.5 * tp[5 * N];
                by = 0.5 * by + 0.5 * tp[6 * N];
            }
            const double2 n = normal(r);
            const double bn = bx * n.x + by * n.y;
#pragma unroll
            for (int i = 0; i < N; i++) dvb[i] += bn * ops.M[r * N + i];
        }
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (2 * m + 1 < N || par) sBeta[c * NN + pt0 + pts * (2 * m + 1 - par)] = par ? dvb[i0] : dvb[i1];
        }
    }
    __syncthreads();

    // ---- per solution point: the source adjoint, -lambda/J, divB adjoint ----------------
    double acc[N][9];  // the line's sums of the state adjoint; a finished point's start from its source adjoint
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int k = 0; k < 9; k++) acc[i][k] = 0.0;
    if (act) {
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (!(2 * m + 1 < N) && par) continue;
            const int pt = pt0 + pts * (2 * m + par);
            const double rJ = 1.0 / sMet[c * S::MS + ML::kJac + pt];
            const double divB = a.vismode == 1 ? (sBeta[c * NN + pt] + (par ? dvb[i1] : dvb[i0])) * rJ : 0.0;
            const double *qs = sQ + c * QS + 9 * pt;
            double *lp = sA + c * QS + 9 * pt;
            double lam[9];
#pragma unroll
            for (int k = 0; k < 9; k++) lam[k] = a.xbar ? a.lam_scale * lp[k] : 0.0;
            const double ri = 1.0 / qs[0], ux = qs[1] * ri, uy = qs[2] * ri, uz = qs[3] * ri;
            const double Bx = qs[5], By = qs[6], Bz = qs[7];
            double db = 0.0;
            if (a.vismode == 1)
                db = -(lam[1] * Bx + lam[2] * By + lam[3] * Bz + lam[4] * ((ux * Bx + uy * By) + uz * Bz) +
                       lam[5] * ux + lam[6] * uy + lam[7] * uz);
            // Powell and GLM sources (compresid.f90:60-78)
            const double ub = -divB * (lam[4] * Bx + lam[5]);
            const double vb = -divB * (lam[4] * By + lam[6]);
            const double wb = -divB * (lam[4] * Bz + lam[7]);
            double src[9];
            src[0] = -(ub * ux + vb * uy + wb * uz) * ri;
            src[1] = ub * ri;
            src[2] = vb * ri;
            src[3] = wb * ri;
            src[4] = 0.0;
            src[5] = -divB * (lam[1] + lam[4] * ux);
            src[6] = -divB * (lam[2] + lam[4] * uy);
            src[7] = -divB * (lam[3] + lam[4] * uz);
            src[8] = -a.alpha * lam[8];
#pragma unroll
            for (int k = 0; k < 9; k++) {
                lp[k] = -lam[k] * rJ;
                if (i1 != i0) {
                    acc[i0][k] = par ? 0.0 : src[k];
                    acc[i1][k] = par ? src[k] : 0.0;
                } else {
                    acc[i0][k] = src[k];
                }
            }
            sBeta[c * NN + pt] = db * rJ;
        }
    }
    __syncthreads();

    // ---- per flux point of the line: the point adjoint and its interpolation's share -----
    double cbar = 0.0, pb[6] = {0, 0, 0, 0, 0, 0};
    if (act) {
        auto point = [&](int r) {
            double q[9], fb[9], qb[9], bt = 0.0;
            own_state(r, q);
            {
                int qi = q0, bi = c * NN + pt0;
                asm volatile("" : "+r"(qi), "+r"(bi));  // read anew at every point
#pragma unroll
                for (int k = 0; k < 9; k++) fb[k] = 0.0;
#pragma unroll
                for (int s = 0; s < N; s++) {
                    const double M = ops.M[r * N + s];
#pragma unroll
                    for (int k = 0; k < 9; k++) fb[k] += M * sA[qi + qstr * s + k];
                    bt += M * sBeta[bi + pts * s];
                }
            }
            const double2 nn = normal(r);
            double vbx = bt * nn.x, vby = bt * nn.y;  // adjoint of Bx, By there (zero unless vismode = 1)
#pragma unroll
            for (int k = 0; k < 9; k++) qb[k] = 0.0;
            if (r > 0 && r < N) {
                double um;
                cbar += iflux_vjp(q, a.c_h, nn.x, nn.y, fb, qb, um, nullptr);
                qb[5] += vbx;
                qb[6] += vby;
            } else {
                const int2 rec = r == 0 ? rec0 : recN;
                const int lf = r == 0 ? lf0 : lfN, np = r == 0 ? np0 : npN, kind = rec.y & 0xff;
                const double *tp = other_at(r);
                double oth[9], fbar[9];
#pragma unroll
                for (int k = 0; k < 9; k++) oth[k] = tp[k * N];
                if (is_pair(kind)) {
                    const int plf = (rec.y >> 8) & 0xff;
                    const bool own_right = kind == kFaceRight, plow = plf == 1 || plf == 4;
                    const double2 pn = own_right ? sP[(r == 0 ? 0 : NT) + tid] : nn;
                    const int sign_l = own_right ? (plow ? -1 : 1) : (r == 0 ? -1 : 1);
                    const int sign_r = own_right ? (r == N ? -1 : 1) : (plow ? 1 : -1);
                    const double slr = (double)(sign_l * sign_r);
                    // own slot's and the partner's share; a right cell's slot is
                    // the left one's with both signs
                    const double ms = own_right ? slr : 1.0, ps = own_right ? 1.0 : slr;
                    const double *ap = sAT + c * S::AS + (lf - 1) * S::AF + (N - 1 - np);
#pragma unroll
                    for (int k = 0; k < 9; k++) fbar[k] = ms * fb[k] + (a.xbar ? ps * ap[k * N] : 0.0);
                    if (a.xbar && a.vismode == 1) {
                        vbx += ap[9 * N];
                        vby += ap[10 * N];
                    }
                    // the face-averaged Bx, By feed the gradients of both cells
                    qb[5] = 0.5 * vbx;
                    qb[6] = 0.5 * vby;
                    // the flux is the same with the roles swapped and the normal
                    // reversed, so this cell is the left one here
                    cbar += ms * rusanov_vjp_own(q, oth, pn.x, pn.y, own_right ? -sign_l : sign_l, a.c_h, fbar, fb, qb);
                } else {
                    const int sign_l = r == 0 ? -1 : 1;
#pragma unroll
                    for (int k = 0; k < 9; k++) fbar[k] = fb[k];
                    if (kind == kFaceWall) {  // the objective: force on the wall faces
                        const double w = a.wq[l] * (double)sign_l;
                        fbar[1] += a.sx * w;
                        fbar[2] += a.sy * w;
                    }
                    double qo[9], fo[9], ql[9], og[9], ff[9];  // the call's own copies
                    for (int k = 0; k < 9; k++) {
                        qo[k] = 0.0;
                        fo[k] = fbar[k];
                        ff[k] = fb[k];
                        ql[k] = q[k];
                        og[k] = oth[k];
                    }
                    qo[5] = 0.5 * vbx;
                    qo[6] = 0.5 * vby;
                    cbar += vjp_boundary(kind, ql, og, nn.x, nn.y, sign_l, a.vismode, a.fs, a.c_h, fo, ff, vbx, vby, qo, pb);
                    for (int k = 0; k < 9; k++) qb[k] = qo[k];
                }
            }
#pragma unroll
            for (int i = 0; i < N; i++) {
                const double L = ops.L[r * N + i];
#pragma unroll
                for (int k = 0; k < 9; k++) acc[i][k] += L * qb[k];
            }
        };
        point(0);
#pragma unroll 1
        for (int r = 1; r < N; r++) point(r);
        point(N);
    }
    __syncthreads();  // the traces, the states and -lambda/J are read

    // the next stage's input state, for its adjoint traces, over -lambda/J
    const bool fuse = a.at_next != nullptr;  // uniform
    const double *qn = fuse ? a.q_next + (size_t)c0 * NQ : nullptr;
    const bool qn_bulk = fuse && (((uintptr_t)qn | cbytes) & 15) == 0;
    if (qn_bulk && tid < 32) {
        if (tid == 0) {
            fence_proxy_async();
            mbar_expect_tx(&sBarN, (unsigned)(ncl * NQ * sizeof(double)));
        }
        __syncwarp();
        if (tid < (S::kPad ? ncl : 1)) bulk_g2s(sA + tid * QS, qn + (size_t)tid * NQ, cbytes, &sBarN);
    }

    // ---- the exchange: state adjoint at the solution points -----------------------------
    if (act) {
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (2 * m + 1 < N || par) {
                double *o = sX + c * S::XS + (pt0 + pts * (2 * m + 1 - par)) * 9;
#pragma unroll
                for (int k = 0; k < 9; k++) o[k] = par ? acc[i0][k] : acc[i1][k];
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
            const double *x = sX + c * S::XS + pt * 9;
            double *o = sQ + c * QS + 9 * pt;
#pragma unroll
            for (int k = 0; k < 9; k++) o[k] = (par ? acc[i1][k] : acc[i0][k]) + x[k];
        }
    }
    __syncthreads();

    // ---- RK reverse update, element-wise ----------------------------------------------
    // the register reads of kU elements are issued before their use, so that
    // each thread keeps several loads in flight
    {
        constexpr int kU = 6;
        const size_t g0 = (size_t)c0 * NQ;
        const int n = ncl * NQ;
        for (int e0 = tid; e0 < n; e0 += kU * NT) {
            double va[kU], vb[kU], vc[kU], vx[kU];
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const int e = e0 + u * NT;
                const size_t g = g0 + (e < n ? e : 0);
                va[u] = a.ra ? a.ra[g] : 0.0;
                vb[u] = a.rb ? a.rb[g] : 0.0;
                vc[u] = a.out2 && a.rc ? a.rc[g] : 0.0;
                vx[u] = a.out2 ? a.xbar[g] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const int e = e0 + u * NT;
                if (e >= n) break;
                const size_t g = g0 + e;
                const int cc = e / NQ;
                double *x = sQ + cc * QS + (e - cc * NQ);
                double o = 0.0;
                if (a.ra) o = a.wa * va[u];
                if (a.rb) o = o + a.wb * vb[u];
                const double ov = o + *x;
                a.out[g] = ov;
                if (fuse) *x = ov;
                if (a.out2) a.out2[g] = (a.rc ? a.wc * vc[u] : 0.0) + a.wd * vx[u];
            }
        }
    }

    // ---- the next reverse stage's adjoint traces from out (adj_trace_kernel's ----------
    // ---- arithmetic): -lambda/J and the divB adjoint per point, then per line end -------
    if (fuse) {
        if (!qn_bulk)
            for (int k = tid; k < ncl * NQ; k += NT) {
                const int cc = k / NQ;
                sA[cc * QS + (k - cc * NQ)] = qn[k];
            }
        else if (tid == 0 && !mbar_wait_bounded(&sBarN, 0)) {
            raise_fault(a.err, kErrStagingTimeout);  // the copy did not complete
            sAbort = 1;
            mbar_wait_bounded(&sBarN, 0);
        }
        __syncthreads();
        if (sAbort) return;
        for (int k = tid; k < ncl * NN; k += NT) {
            const int cc = k / NN, pt = k - cc * NN;
            double *x = sQ + cc * QS + 9 * pt;
            double db = 0.0;
            if (a.vismode == 1) {
                const double *qq = sA + cc * QS + 9 * pt;
                const double ri = 1.0 / qq[0], ux = qq[1] * ri, uy = qq[2] * ri, uz = qq[3] * ri;
                db = -a.scale_next * (x[1] * qq[5] + x[2] * qq[6] + x[3] * qq[7] +
                                      x[4] * ((ux * qq[5] + uy * qq[6]) + uz * qq[7]) + x[5] * ux + x[6] * uy +
                                      x[7] * uz);
            }
            const double rJ = 1.0 / sMet[cc * S::MS + ML::kJac + pt];
            sBeta[k] = db * rJ;
#pragma unroll
            for (int m = 0; m < 9; m++) x[m] = -(a.scale_next * x[m]) * rJ;
        }
        __syncthreads();
        if (act) {
            double f0[9], fN[9], b0 = 0.0, bN = 0.0;
#pragma unroll
            for (int k = 0; k < 9; k++) f0[k] = fN[k] = 0.0;
#pragma unroll
            for (int i = 0; i < N; i++) {
                const double m0 = ops.M[i], mN = ops.M[N * N + i];
                const double *mu = sQ + q0 + qstr * i;
#pragma unroll
                for (int k = 0; k < 9; k++) {
                    f0[k] += m0 * mu[k];
                    fN[k] += mN * mu[k];
                }
                const double b = sBeta[c * NN + pt0 + pts * i];
                b0 += m0 * b;
                bN += mN * b;
            }
            const double2 n0 = normal(0), nN = normal(N);
            // collected over the neighbours' traces: sX's readers are done
            double *o0 = sT + c * S::AS + (lf0 - 1) * S::AF + np0, *oN = sT + c * S::AS + (lfN - 1) * S::AF + npN;
#pragma unroll
            for (int k = 0; k < 9; k++) {
                o0[k * N] = f0[k];
                oN[k * N] = fN[k];
            }
            o0[9 * N] = b0 * n0.x;
            o0[10 * N] = b0 * n0.y;
            o0[11 * N] = 0.0;
            oN[9 * N] = bN * nN.x;
            oN[10 * N] = bN * nN.y;
            oN[11 * N] = 0.0;
        }
        fence_proxy_async();
        __syncthreads();
        if (tid < ncl)
            bulk_s2g(a.at_next + (size_t)(c0 + tid) * 4 * S::AF, sT + tid * S::AS, 4 * S::AF * sizeof(double));
    }

    // ---- per-CTA sums of the c_h and free-stream adjoints ------------------------------
    {
        const int lane = tid & 31, wid = tid >> 5;
        constexpr int NW = NT / 32;
        double v[7] = {cbar, pb[0], pb[1], pb[2], pb[3], pb[4], pb[5]};
        // the free-stream adjoints are zero away from boundary faces: a warp
        // whose lanes all hold zero skips that sum
#pragma unroll
        for (int m = 0; m < 7; m++) {
            if (m == 0 || __any_sync(0xffffffffu, v[m] != 0.0)) v[m] = warp_sum(v[m]);
            if (lane == 0) sRed[m * 32 + wid] = v[m];
        }
        __syncthreads();
        if (tid < 7) {
            double s = 0.0;
            for (int w = 0; w < NW; w++) s += sRed[tid * 32 + w];
            a.part[(size_t)tid * gridDim.x + blockIdx.x] = s;
        }
    }
    if (tid < 32) bulk_wait_read();
}

// ---- per-stage reduction and the running-max adjoint --------------------------------
// Sums the per-CTA partials in a fixed order; gives the adjoint accumulated
// for the running maxima to the points recorded for this stage (split
// equally among the points attaining the maximum, a shared face counted
// once); then restarts the accumulation at this stage's owner and adds this
// stage's c_h adjoint (dc/dL, dc/dU from the maxima it read).
// Where the VJP formed the next stage's adjoint traces from out, the cells
// that the records change get theirs formed again (next.at non-null).
constexpr int kRedThreads = 1024;
struct NextTraces {
    double *at;       // the next stage's adjoint traces (null: none formed yet)
    const double *q;  // its input state
    double scale;     // its lam_scale
    const double *met;
    int vismode;
};
template <int N>
static __global__ void __launch_bounds__(kRedThreads) adj_reduce_kernel(int nblk, const double *__restrict__ part,
                                                                 AdjScalars *acc, int owner_eig, int owner_um,
                                                                 double dc_dl, double dc_du,
                                                                 const AdjRec *__restrict__ recs, int *rec_n,
                                                                 int *rec_cnt, int rec_cap, double *out,
                                                                 const Ops ops, FaultFlags *err, NextTraces next)
{
    __shared__ double s[7][kRedThreads / 32];
    __shared__ double w[2];
    __shared__ double ps[6];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    // unrolled so that the loads of several partials are in flight at once
#pragma unroll 8
    for (int b = tid; b < nblk; b += kRedThreads)
#pragma unroll
        for (int m = 0; m < 7; m++) v[m] += part[(size_t)m * nblk + b];
#pragma unroll
    for (int m = 0; m < 7; m++) {
        v[m] = warp_sum(v[m]);
        if (lane == 0) s[m][wid] = v[m];
    }
    if (tid < 6) ps[tid] = 0.0;
    if (tid == 0) {
        const int ce = rec_cnt[0], cu = rec_cnt[1];
        w[0] = (owner_eig && ce > 0) ? acc->lam_eig / ce : 0.0;
        w[1] = (owner_um && cu > 0) ? acc->lam_um / cu : 0.0;
        if ((owner_eig && ce == 0) || (owner_um && cu == 0)) raise_fault(err, kErrAdjointMaxLost);
    }
    __syncthreads();
    const int nrec = min(*rec_n, rec_cap);
    const int NP = N + 1, NQ = 9 * N * N;
    for (int k = tid; k < nrec; k += kRedThreads) {
        const AdjRec &R = recs[k];
        const double wt = w[R.kind];
        if (wt == 0.0) continue;
        const int r = R.slot % NP, fl = R.slot / NP, line = fl % N, fam = fl / N;
        for (int sidx = 0; sidx < N; sidx++) {
            const int sp = fam == 0 ? sidx + N * line : line + N * sidx;
            const double l = wt * ops.L[r * N + sidx];
            double *o = out + (size_t)R.cell * NQ + 9 * sp;
            for (int m = 0; m < 9; m++) atomicAdd(o + m, l * R.d[m]);
        }
        for (int m = 0; m < 6; m++)
            if (R.p[m] != 0.0) atomicAdd(&ps[m], wt * R.p[m]);
    }
    __syncthreads();
    if (next.at)  // one warp per record, a lane per face point of its cell
        for (int k = wid; k < nrec; k += kRedThreads / 32) {
            const AdjRec &R = recs[k];
            if (w[R.kind] == 0.0) continue;
            for (int f = lane; f < 4 * N; f += 32)
                adj_trace_point<N>((size_t)R.cell, f, out, next.q, next.scale, next.met, next.vismode, ops, next.at);
        }
    if (tid == 0) {
        double t[7] = {0, 0, 0, 0, 0, 0, 0};
        for (int x = 0; x < kRedThreads / 32; x++)
            for (int m = 0; m < 7; m++) t[m] += s[m][x];
        const double cb = t[0];
        for (int m = 0; m < 6; m++) acc->pbar[m] += t[1 + m] + ps[m];
        acc->cbar += cb;
        if ((owner_eig && rec_cnt[0] > 1) || (owner_um && rec_cnt[1] > 1)) acc->ties += 1.0;
        acc->lam_eig = (owner_eig ? 0.0 : acc->lam_eig) + cb * dc_dl;
        acc->lam_um = (owner_um ? 0.0 : acc->lam_um) + cb * dc_du;
        *rec_n = 0;
        rec_cnt[0] = 0;
        rec_cnt[1] = 0;
    }
}

// ---- where a running maximum was raised --------------------------------------------
// Each thread checks the recorded maxima of one CTA of the forward stage
// (cpb cells each; a block covers 128 of them).  For every CTA whose
// recorded maximum equals the stage's new running max, in ascending order,
// the block recomputes, in the exact form (its translation unit is compiled
// with -fmad=false, like the forward stage kernel), the wave speed and
// velocity maximum of its points and records the gradient of each one equal
// to the new maximum.
struct LocateArgs {
    int ncell, vismode, cpb;
    double c_h;
    Freestream fs;
    const double *q, *t_in, *met;
    const int2 *faces;
    const double *cta_max;  // per forward CTA (max eigv, max umax)
    int hit_eig, hit_um;    // which running maximum the stage raised
    double eig_max, um_max;
    RecSink rs;
};

constexpr int kLocateThreads = 128;

// the points of forward CTA `tile` (cpb cells) that attain the new maximum
template <int N>
__device__ void locate_tile(const LocateArgs &a, const Ops &ops, int tile, bool e, bool u)
{
    using ML = MetLayout<N>;
    constexpr int NQ = 9 * N * N, NP = N + 1;
    const int c0 = tile * a.cpb, ncl = min(a.cpb, a.ncell - c0);
    // flux-point state of line (fam, line) at point r, as the forward form computes it
    auto interp = [&](int cell, int fam, int line, int r, double *qf) {
        const double *qc = a.q + (size_t)cell * NQ;
        for (int v = 0; v < 9; v++) {
            double acc = 0.0;
            for (int s = 0; s < N; s++) {
                const double x = fam == 0 ? qc[v + 9 * (s + N * line)] : qc[v + 9 * (line + N * s)];
                acc = acc + x * ops.L[r * N + s];
            }
            qf[v] = acc;
        }
    };
    const int nface = ncl * 4 * N, nint = ncl * 2 * N * (N - 1);
    for (int t = threadIdx.x; t < nface + nint; t += blockDim.x) {
        if (t < nface) {
            const int nfp = 1 + t % N, lf = 1 + (t / N) % 4, c = t / (4 * N);
            const int cell = c0 + c;
            int fam, line, r;
            face_point<N>(lf, nfp, fam, line, r);
            double own[9], oth[9];
            interp(cell, fam, line, r, own);
            const int2 rec = a.faces[(size_t)cell * 4 + (lf - 1)];
            const int kind = rec.y & 0xff;
            const bool pair = kind == kFaceLeft || kind == kFaceRight, own_right = kind == kFaceRight;
            const double *onrm = a.met + (size_t)cell * ML::kSize + ML::normal(fam, line, r);
            double n0 = onrm[0], n1 = onrm[1];
            int sign_l = r == 0 ? -1 : 1, sign_r = 1;
            if (pair) {
                const int pc = rec.x, plf = (rec.y >> 8) & 0xff;
                int pfam, pline, pr;
                face_point<N>(plf, N - nfp + 1, pfam, pline, pr);
                for (int k = 0; k < 9; k++) oth[k] = a.t_in[trace_at<N>(trace_stride<N, double>(), pc, plf, N - nfp, k)];
                if (!own_right) {
                    sign_r = pr == N ? -1 : 1;
                } else {
                    const double *pn = a.met + (size_t)pc * ML::kSize + ML::normal(pfam, pline, pr);
                    n0 = pn[0];
                    n1 = pn[1];
                    sign_l = pr == 0 ? -1 : 1;
                    sign_r = r == N ? -1 : 1;
                }
            } else {
                bc_ghost<double, true>(kind, own, n0, n1, a.vismode, a.fs, oth);
            }
            double Ql[9], Qr[9], Fl[9], Fr[9], eig, um = 0.0;
            for (int k = 0; k < 9; k++) {
                Ql[k] = own_right ? oth[k] : own[k];
                Qr[k] = own_right ? own[k] : oth[k];
            }
            rusanov<double, true>(Ql, Qr, Fl, Fr, n0, n1, sign_l, sign_r, a.c_h, eig, um);
            const bool he = e && eig == a.eig_max, hu = u && um == a.um_max;
            if (he || hu)
                adj_record_face(a.rs, a.fs, a.vismode, a.c_h, he, hu, cell, (fam * N + line) * NP + r, kind, own_right,
                                own, oth, n0, n1, sign_l);
        } else if (u) {
            const int k = t - nface;
            const int r = 1 + k % (N - 1), l = (k / (N - 1)) % N, f = (k / ((N - 1) * N)) % 2, c = k / (2 * N * (N - 1));
            double qf[9];
            interp(c0 + c, f, l, r, qf);
            // the velocity maximum as the forward's iflux forms it
            const double uu = qf[1] / qf[0], vv = qf[2] / qf[0], ww = qf[3] / qf[0];
            if (Max(Max(Abs(uu), Abs(vv)), Abs(ww)) == a.um_max) {
                double umd[9], qb[9], fz[9], um;
                for (int m = 0; m < 9; m++) fz[m] = qb[m] = 0.0;
                iflux_vjp(qf, a.c_h, 0.0, 0.0, fz, qb, um, umd);
                adj_record(a.rs, c0 + c, (f * N + l) * NP + r, 1, 1, umd, nullptr);
            }
        }
    }
}

template <int N>
__global__ void __launch_bounds__(kLocateThreads) adj_locate_kernel(const LocateArgs a, const Ops ops, int ntiles)
{
    __shared__ unsigned sE[kLocateThreads / 32], sU[kLocateThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    {
        const int bt = blockIdx.x * kLocateThreads + threadIdx.x;
        const bool e = bt < ntiles && a.hit_eig && a.cta_max[2 * bt] == a.eig_max;
        const bool u = bt < ntiles && a.hit_um && a.cta_max[2 * bt + 1] == a.um_max;
        const unsigned me = __ballot_sync(0xffffffffu, e), mu = __ballot_sync(0xffffffffu, u);
        if (lane == 0) {
            sE[wid] = me;
            sU[wid] = mu;
        }
    }
    __syncthreads();
    for (int w = 0; w < kLocateThreads / 32; w++)
        for (unsigned m = sE[w] | sU[w]; m; m &= m - 1) {
            const int bit = __ffs(m) - 1;
            const int tile = blockIdx.x * kLocateThreads + 32 * w + bit;
            const bool e = (sE[w] >> bit) & 1u, u = (sU[w] >> bit) & 1u;
            locate_tile<N>(a, ops, tile, e, u);
        }
}

// ---- the objective: force on the wall faces -------------------------------------------
// out[0..1] = sum over wall face points of w(line) * sign_l * f(1..2), f the
// wall face's Rusanov flux (BCFLUX wall state) at the state whose traces are
// t; one block, fixed summation order.
template <int N>
__global__ void __launch_bounds__(256) wall_force_kernel(int nw, const int2 *__restrict__ wall,
                                                         const double *__restrict__ t, const double *__restrict__ met,
                                                         int vismode, Freestream fs, const double *__restrict__ wq,
                                                         double *out)
{
    using ML = MetLayout<N>;
    __shared__ double s0[256], s1[256];
    const int tid = threadIdx.x;
    double fx = 0.0, fy = 0.0;
    for (int e = tid; e < nw * N; e += 256) {
        const int2 wf = wall[e / N];
        const int nfp = 1 + e % N, lf = wf.y;
        int fam, line, r;
        face_point<N>(lf, nfp, fam, line, r);
        const size_t own = trace_at<N>(trace_stride<N, double>(), wf.x, lf, nfp - 1, 0);  // variable k at own + k*N
        const double *nr = met + (size_t)wf.x * ML::kSize + ML::normal(fam, line, r);
        const int sign_l = r == 0 ? -1 : 1;
        double ql[9], gh[9], Fl[9], Fr[9], eig, um = 0.0;
        for (int k = 0; k < 9; k++) ql[k] = t[own + (size_t)k * N];
        bc_ghost<double, true>(kFaceWall, ql, nr[0], nr[1], vismode, fs, gh);
        rusanov<double, true>(ql, gh, Fl, Fr, nr[0], nr[1], sign_l, 1, 0.0, eig, um);
        const double w = wq[line] * (double)sign_l;
        fx += w * Fl[1];
        fy += w * Fl[2];
    }
    s0[tid] = fx;
    s1[tid] = fy;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if (tid < h) {
            s0[tid] += s0[tid + h];
            s1[tid] += s1[tid + h];
        }
        __syncthreads();
    }
    if (tid == 0) {
        out[0] = s0[0];
        out[1] = s1[0];
    }
}

// launches compiled in the exact translation unit (adjoint_exact.cu)
cudaError_t launch_adj_locate(int N, int nblk, const LocateArgs &a, const Ops &ops, cudaStream_t st);
cudaError_t launch_wall_force(int N, int nw, const int2 *wall, const double *t, const double *met, int vismode,
                              const Freestream &fs, const double *wq, double *out, cudaStream_t st);

}  // namespace sddc
