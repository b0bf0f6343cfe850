// The RK stage of a time step with one thread per line of solution points.
//
// One launch evaluates compresid (compresid.f90:1-80 and what it calls, as
// stage_kernel.cuh lists it) for every cell and applies one RK stage update
// (iterations.f90:88-213), so a stage reads the state once and writes it
// once.  A cell has N xi lines and N eta lines, and one thread takes a whole
// line.  It forms the state at one flux point after the other, its flux
// (Rusanov at the two ends, which are the cell's face points) and adds that
// flux's share of the line derivative to sums in registers.  The flux-point
// states, the fluxes and their derivatives, which the tile kernel passes
// through shared memory between its phases, never leave the registers; only
// the derivative of the line that crosses a point is exchanged, once.
//
// Steps of a CTA (a tile of CPB cells):
//   1  what no earlier launch writes: face records, normals, Jac (TMA) and
//      the partners' normals; then, after the end of the previous launch,
//      the state slice and, in a stage that reads one, the RK register's by
//      TMA, the neighbours' face traces by 16-byte asynchronous copies;
//   2  per line: interpolation, fluxes, derivative sums, div B sums (of the
//      contravariant Bn = Bx n0 + By n1, outside the exact form);
//   3  the exchange: of the two lines through a solution point the one of
//      matching parity finishes the point, the other hands over its sums,
//      so every thread finishes half of its points;
//   4  sources and the RK update of the point, the output in place over the
//      RK register's slice, from where one bulk store takes it to memory;
//   5  per line: the output's traces at its two ends, collected in shared
//      memory and stored by TMA.
// All sums run in the tile kernel's order, so the results are the same bits.
// Running maxima go through atomicMax on rotating slots, as there.
//
// What bounds it: latency.  At N = 5 in the mixed form (6 cells, 64 threads,
// 128 registers) a scheduler holds 3.3 warps and issues in 48% of its cycles,
// with 40% of DRAM bandwidth and the L1 pipe 62% busy (the tile kernel: 87%); in
// the FP64 form (252 registers) it holds 1.9 warps and issues in 37%.  Why this
// split: a stage moves 10 KB per cell through shared memory instead of 26 KB.
// us per RK_S5P3 step, tile kernel and this one: 256x512 cells, N = 5, mixed 1373
// and 1070, FP64 2267 and 1685; 512x512 cells, N = 4, mixed 1810 and 1290.
#pragma once

#include "stage_kernel.cuh"

namespace sddc {

__host__ __device__ constexpr int line_threads(int n, int cpb) { return (2 * n * cpb + 31) / 32 * 32; }

template <int N, typename R, bool EX> struct LineSmem {
    static constexpr int NQ = 9 * N * N, NN = N * N;
    // cell stride of the state slices in doubles: an odd number of doubles
    // per line (odd N) already spreads the lines over the banks; for even N
    // two more per cell halve the conflicts (and keep 16-byte alignment)
    static constexpr bool kPad = N % 2 == 0;
    static constexpr int QS = kPad ? NQ + 2 : NQ;
    // sums handed over per point: 9 derivatives and div B's (float: even, so
    // that pairs move together; double: odd, against bank conflicts)
    static constexpr int ND = sizeof(R) == 4 ? 10 : 11;
    static constexpr int XS = NN * ND + (N == 4 ? (sizeof(R) == 4 ? 4 : 2) : 0);  // per cell
    // face traces per cell: the global record, and its padded stride here
    static constexpr int TFS = trace_stride<N, R>();
    static constexpr int TS = 4 * TFS + (sizeof(R) == 4 ? (N == 5 ? 8 : 4) : 2);
    // the float form's output copy lies in the exchange slots and its traces
    // over the state, which holds them except at N = 2
    static constexpr bool kTOwn = sizeof(R) == 4 && TS * sizeof(R) > QS * sizeof(double);
    static constexpr int NM = 2 * MetLayout<N>::kFam, NJ = MetLayout<N>::kJacPad;
};

template <int N, int CPB, typename R, bool EX> __host__ __device__ constexpr size_t line_smem_bytes()
{
    using S = LineSmem<N, R, EX>;
    // the region that holds the neighbours' traces and normals, then the
    // exchanged sums, then the output's traces
    const size_t t = (size_t)CPB * S::TS * sizeof(R) + 2 * line_threads(N, CPB) * sizeof(P2<R>);
    const size_t x = (size_t)CPB * S::XS * sizeof(R);
    // state and RK register slices, Jac, normals, and that region
    return (size_t)CPB * ((2 * S::QS + S::NJ) * sizeof(double) + S::NM * sizeof(R)) + ((t > x ? t : x) + 15) / 16 * 16 +
           (S::kTOwn ? (size_t)CPB * S::TS * sizeof(R) : 0);
}

// Whether a thread holds its line's states in registers beside the sums.  In
// double at N = 6 they do not fit (121x87 cells in exact operations: 638 us a step
// with spills, 465 read from shared memory), in the exact form not at N = 5 either
// (300x300 cells 428 us a stage with spills, 402), and at N = 4 there is a second
// kernel without them (WIDE): 168 registers instead of 240 let a scheduler
// hold 3 warps instead of 2.  (At N = 5 the sums alone leave no third warp: 363
// us a stage held, 423 read.)
template <int N, typename R, bool EX, bool WIDE> __host__ __device__ constexpr bool line_hold()
{
    return sizeof(R) == sizeof(float) || (N <= (EX ? 4 : 5) && !WIDE);
}
__host__ __device__ constexpr bool line_has_wide(int n, int elem) { return n == 4 && elem == 8; }
// Which of the two takes a stage of the given tiles, by the waves it needs
// (CTAs resident at once: 592 held, 888 wide) and what a wave costs: one wave
// of a small mesh takes 9.4 us held and 12.2 wide.  us per step, held and
// wide: FP64, 64x64 cells (1 wave each) 47 and 61, 96x96 (2 and 2) 96 and 109,
// 128x128 (4 and 3) 178 and 172, 256x256 (14 and 10) 630 and 573; exact,
// 256x256 cells 922 and 852.
__host__ __device__ constexpr bool line_use_wide(int tiles, int resident_held, int resident_wide)
{
    return (tiles + resident_wide - 1) / resident_wide * 13 < (tiles + resident_held - 1) / resident_held * 10;
}

// CTAs per SM the kernel is compiled for: as many as shared memory holds, up
// to the warps whose registers hold a line (a scheduler's 512 registers per
// lane go to whole warps: 4 warps of 128 registers, 3 of 168, 2 of 255)
template <int N, typename R, bool WIDE> constexpr int line_warps()
{
    if (sizeof(R) == 4) return N >= 6 ? 12 : N >= 4 ? 16 : N == 3 ? 20 : 24;
    return N >= 4 && !WIDE ? 8 : 12;
}
template <int N, int CPB, typename R, bool EX, bool WIDE> constexpr int line_min_blocks()
{
    int b = (int)((228 * 1024) / (line_smem_bytes<N, CPB, R, EX>() + 1024 + 256));
    const int br = line_warps<N, R, WIDE>() / (line_threads(N, CPB) / 32);
    b = b < br ? b : br;
    return b < 1 ? 1 : b;
}

// 16 bytes from global to shared memory, asynchronously
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
// the pair of a normal (8 or 16 bytes)
template <typename T> __device__ __forceinline__ void cp_async_pair(T *dst, const T *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src), "n"(sizeof(T)) : "memory");
}
// programmatic dependent launch: wait for the launches this one depends on
// (complete, their writes visible); let the dependent launch's CTAs start
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int N, int CPB, typename R, bool EXACT, int KIND, bool WIDE>
__device__ __forceinline__ bool line_tile(const StageArgs &a, const Ops &ops, const int tile)
{
    constexpr bool EX = EXACT && sizeof(R) == sizeof(double);
    constexpr bool kBn = !EX;
    using S = LineSmem<N, R, EX>;
    using ML = MetLayout<N>;
    constexpr int NT = line_threads(N, CPB), NQ = S::NQ, NN = S::NN, NP = N + 1, QS = S::QS, ND = S::ND, XS = S::XS,
                  TFS = S::TFS, TS = S::TS, NM = S::NM, NJ = S::NJ;
    constexpr int NH = (N + 1) / 2;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *sQ = reinterpret_cast<double *>(smem_raw);  // [CPB][QS] state
    double *sA = sQ + CPB * QS;                          // [CPB][QS] RK register, then the output
    double *sJac = sA + CPB * QS;                        // [CPB][NJ]
    R *sN = reinterpret_cast<R *>(sJac + CPB * S::NJ);   // [CPB][NM] normals
    R *sX = sN + CPB * NM;                               // neighbours' traces, exchanged sums, output traces
    // the partners' normals at the ends r = 0 and r = N of each thread's line
    P2<R> *sP = reinterpret_cast<P2<R> *>(sX + CPB * TS);  // [2][NT]
    __shared__ __align__(8) unsigned long long sBar;
    __shared__ int sAbort;
    __shared__ double sRed[4 * (NT / 32)], sCarry[2];

    const int tid = threadIdx.x;
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

    // this thread's line: family f (0: xi, 1: eta), line l, of cell c;
    // neighbouring lanes take the same line of neighbouring cells (15-25%
    // fewer shared-memory wavefronts than the lines of one cell side by side)
    const int fam = tid >= N * CPB ? 1 : 0;
    const int lt = tid - fam * N * CPB, lc = lt % CPB;
    const bool act = tid < 2 * N * CPB && lc < ncl;
    const int c = act ? lc : 0, l = act ? lt / CPB : 0;
    // its end faces: (r = 0) local face 4 or 1, (r = N) local face 2 or 3
    // (face2fpconnec, initsetup.f90:347-383), and its face points there
    const int lf0 = fam == 0 ? 4 : 1, lfN = fam == 0 ? 2 : 3;
    const int np0 = fam == 0 ? N - 1 - l : l, npN = fam == 0 ? l : N - 1 - l;  // 0-based
    int2 rec0 = make_int2(0, 0), recN = make_int2(0, 0);
    if (act) {
        rec0 = __ldg(a.faces + (size_t)(c0 + c) * 4 + lf0 - 1);
        recN = __ldg(a.faces + (size_t)(c0 + c) * 4 + lfN - 1);
    }
    // the face records of this thread's pieces of the neighbours' traces (16
    // bytes of face f of the tile each); all loads are issued before the first
    // asynchronous copy, which orders what follows it
    constexpr int CH = TFS * (int)sizeof(R) / 16, CE = 16 / (int)sizeof(R);
    constexpr int IT = (CPB * 4 * CH + NT - 1) / NT;
    int2 frec[IT];
#pragma unroll
    for (int m = 0; m < IT; m++) {
        const int f = (tid + m * NT) / CH;
        frec[m] = f < ncl * 4 ? __ldg(a.faces + (size_t)c0 * 4 + f) : make_int2(0, 0);
    }

    // ---- 1: staging -------------------------------------------------------------
    // first what no earlier launch writes: normals and Jac (the split arrays,
    // or the packed records, in double)
    const int kind = KIND >= 0 ? KIND : a.rk_kind;
    const bool want_ra = kind == kRkTwoReg || kind == kRkTwoRegT;
    const double *qsrc = a.q_in + (size_t)c0 * NQ;
    const double *rsrc = want_ra ? a.reg_a + (size_t)c0 * NQ : nullptr;
    const bool split = sizeof(R) == sizeof(float) || a.nrm != nullptr;  // uniform
    const R *nbase = split ? reinterpret_cast<const R *>(a.nrm) : reinterpret_cast<const R *>(a.met);
    const int nstride = split ? NM : ML::kSize;
    // state slices: one copy of the tile, or one per cell where the cells are padded
    const unsigned cbytes = (unsigned)((S::kPad ? 1 : ncl) * NQ * sizeof(double));
    const bool bulk = (((uintptr_t)qsrc | (uintptr_t)rsrc | cbytes) & 15) == 0;  // uniform
    if (tid < 32) {
        if (tid == 0) {
            sAbort = 0;
            mbar_init(&sBar, 1);
            mbar_expect_tx(&sBar, (unsigned)(ncl * (NM * sizeof(R) + NJ * sizeof(double)) +
                                             (bulk ? ncl * NQ * sizeof(double) * (want_ra ? 2 : 1) : 0)));
        }
        __syncwarp();
        if (tid < (split ? 1 : ncl)) {  // (always whole 16-byte units)
            const unsigned n = split ? ncl : 1;
            bulk_g2s(sN + tid * NM, nbase + (size_t)(c0 + tid) * nstride, (unsigned)(n * NM * sizeof(R)), &sBar);
            bulk_g2s(sJac + tid * NJ,
                     split ? a.jac + (size_t)c0 * NJ : a.met + (size_t)(c0 + tid) * ML::kSize + ML::kJac,
                     (unsigned)(n * NJ * sizeof(double)), &sBar);
        }
    }
    auto fetch_pn = [&](const int2 rec, int np, P2<R> *dst) {
        if ((rec.y & 0xff) != kFaceRight) return;
        int pfam, pline, pr;
        face_point<N>((rec.y >> 8) & 0xff, N - np, pfam, pline, pr);
        cp_async_pair(dst, reinterpret_cast<const P2<R> *>(nbase + (size_t)rec.x * nstride + ML::normal(pfam, pline, pr)));
    };
    // what the previous launch wrote: the states, the neighbours' traces and
    // the running maxima.  Its end is awaited here; the next launch's CTAs may
    // start as soon as every CTA of this one has.
    grid_dependency_wait();
    grid_launch_dependents();
    const double eig_r = maxima[2 * a.slot_r], um_r = maxima[2 * a.slot_r + 1];
    if (bulk && tid < (S::kPad ? ncl : 1)) {
        bulk_g2s(sQ + tid * QS, qsrc + (size_t)tid * NQ, cbytes, &sBar);
        if (want_ra) bulk_g2s(sA + tid * QS, rsrc + (size_t)tid * NQ, cbytes, &sBar);
    }
    const R *tin = reinterpret_cast<const R *>(a.t_in);
#pragma unroll
    for (int m = 0; m < IT; m++) {
        const int e = tid + m * NT, f = e / CH, ch = e - f * CH, kd = frec[m].y & 0xff;
        if (kd == kFaceLeft || kd == kFaceRight)
            cp_async16(sX + (f >> 2) * TS + (f & 3) * TFS + ch * CE,
                       tin + ((size_t)frec[m].x * 4 + ((frec[m].y >> 8) & 0xff) - 1) * TFS + ch * CE);
    }
    // the left (partner) cell's normal where this cell is the right one
    if (act) {
        fetch_pn(rec0, np0, sP + tid);
        fetch_pn(recN, npN, sP + NT + tid);
    }
    if (!bulk)
        for (int k = tid; k < ncl * NQ; k += NT) {
            const int cc = k / NQ, o = cc * QS + (k - cc * NQ);
            sQ[o] = qsrc[k];
            if (want_ra) sA[o] = rsrc[k];
        }

    // FiveStageRk's last stage adds four registers and its input to the residual:
    // their sum goes to the register's slice here, while the copies above travel,
    // in whole lines of memory (point by point in step 4, with 36 loads 72 bytes
    // apart, a stage of FiveStageRk took on average 97.7 us instead of 81.3 at
    // 32400 cells, N = 5, mixed, 125 instead of 116 in FP64)
    // (the persistent kernel, KIND -2, does so: the pass beside its loop costs
    // every stage 6%)
    if (KIND != -2 && kind == kRkFive) {
        // a thread's share in two batches, three where it has the float form's
        // registers
        constexpr int per = (CPB * NQ + NT - 1) / NT, kU = sizeof(R) == 8 ? (per + 1) / 2 : (per + 2) / 3;
        const double dt5 = a.cases ? a.cases[cs].dt : a.dt;
        auto cf = [&](int i) -> double { return ((a.dt_mask >> i) & 1u) ? a.cb[i] * dt5 : a.cb[i]; };
        const double w1 = cf(1), w2 = cf(2), w3 = cf(3), w4 = cf(4), w5 = cf(5);
        const size_t g0 = (size_t)c0 * NQ;
        for (int e0 = tid; e0 < ncl * NQ; e0 += kU * NT) {
            double va[kU], vb[kU], vc[kU], vq[kU], vd[kU];
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const size_t g = g0 + min(e0 + u * NT, ncl * NQ - 1);
                va[u] = a.reg_a[g];
                vb[u] = a.reg_b[g];
                vc[u] = a.reg_c[g];
                vq[u] = a.q_in[g];
                vd[u] = a.reg_d[g];
            }
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const int e = e0 + u * NT, cc = e / NQ;
                if (e < ncl * NQ)
                    sA[cc * QS + (e - cc * NQ)] = (((w1 * va[u] + w2 * vb[u]) + w3 * vc[u]) + w4 * vq[u]) + w5 * vd[u];
            }
        }
    }

    if (tid == 0) {
        sCarry[0] = eig_r;
        sCarry[1] = um_r;
    }
    // compflux.f90:6 -- running maxima of all previous stages
    const R c_h = (R)sqrt(eig_r * (eig_r - um_r));
    cp_async_wait_all();
    if (tid == 0 && !mbar_wait_bounded(&sBar, 0)) {
        raise_fault(a.err_flags, kErrStagingTimeout);
        sAbort = 1;
        mbar_wait_bounded(&sBar, 0);
    }
    __syncthreads();
    if (sAbort) return false;
    // into L2: the face records and traces of the tile that takes this CTA's
    // place, the two loads in a row that its start waits for (with its state,
    // register and metrics too it was no faster; us per stage at 256x512 cells,
    // N = 5: FP64 362 before, 345 after; mixed 227 and 226; N = 4, 512x512 cells
    // 274 and 270)
    if (tid == NT - 1) {
        const int nc0 = c0 + a.ahead * CPB;
        if (nc0 + CPB <= a.ncell && (N % 2 == 0 || !(nc0 & 1))) {
            bulk_prefetch_l2(a.faces + (size_t)nc0 * 4, CPB * 4 * sizeof(int2));
            bulk_prefetch_l2(tin + (size_t)nc0 * 4 * TFS, CPB * 4 * TFS * sizeof(R));
        }
    }

    // ---- 2: the line ------------------------------------------------------------
    R eigmax = (R)0, umax = (R)0;
    unsigned err = 0;
    constexpr int K2 = 4;     // variable pairs 0..7
    P2<R> d[N][K2 + 1];       // derivative sums; the last pair holds variable 8 and the div B sum
    R dy[N];                  // exact form: the second div B sum
#pragma unroll
    for (int i = 0; i < N; i++) {
#pragma unroll
        for (int k = 0; k <= K2; k++) d[i][k] = splat2<R>((R)0);
        dy[i] = (R)0;
    }
    if (act) {
        // the line's states: in registers, or read from shared memory at every
        // flux point (line_hold); then both ends' fluxes are formed first, while
        // the sums' registers are still free
        constexpr bool kHold = line_hold<N, R, EX, WIDE>();
        P2<R> q2[kHold ? N : 1][K2];
        R q8[kHold ? N : 1];
        const int q0 = c * QS + (fam == 0 ? 9 * N * l : 9 * l);
        const int qstr = fam == 0 ? 9 : 9 * N;
        if constexpr (kHold) {
#pragma unroll
            for (int s = 0; s < N; s++) {
#pragma unroll
                for (int k = 0; k < K2; k++) {
                    q2[s][k].x = (R)sQ[q0 + qstr * s + 2 * k];
                    q2[s][k].y = (R)sQ[q0 + qstr * s + 2 * k + 1];
                }
                q8[s] = (R)sQ[q0 + qstr * s + 8];
            }
        }
        const P2<R> *nl = reinterpret_cast<const P2<R> *>(sN + c * NM + ML::normal(fam, l, 0));
        // the flux along the normal at flux point r (F), the normal (n), and
        // what div B sums there (V): Bn, or in the exact form Bx and By
        auto flux_at = [&](const int r, R (&F)[9], R (&V)[2], P2<R> &n) {
            n = nl[r];
            const R n0 = n.x, n1 = n.y;
            // the state at flux point r
            R q[9];
            int qi = q0;
            if constexpr (!kHold) asm volatile("" : "+r"(qi));  // not kept from point to point
            {
                P2<R> acc[K2];
                R acc8 = (R)0;
#pragma unroll
                for (int k = 0; k < K2; k++) acc[k] = splat2<R>((R)0);
#pragma unroll
                for (int s = 0; s < N; s++) {
                    const P2<R> L2 = opL2<R>(ops, r * N + s);
#pragma unroll
                    for (int k = 0; k < K2; k++) {
                        P2<R> v;
                        if constexpr (kHold) {
                            v = q2[s][k];
                        } else {
                            v.x = (R)sQ[qi + qstr * s + 2 * k];
                            v.y = (R)sQ[qi + qstr * s + 2 * k + 1];
                        }
                        acc[k] = fma2(v, L2, acc[k]);
                    }
                    const R v8 = kHold ? q8[kHold ? s : 0] : (R)sQ[qi + qstr * s + 8];
                    acc8 = acc8 + v8 * L2.x;
                }
#pragma unroll
                for (int k = 0; k < K2; k++) {
                    q[2 * k] = acc[k].x;
                    q[2 * k + 1] = acc[k].y;
                }
                q[8] = acc8;
            }
            if (r > 0 && r < N) {
                // interior flux point (inviscid_flux_interior)
                if (!(q[0] > (R)0)) err |= kErrNonPositiveDensity;
                if constexpr (EX) {
                    R Fx[9], G[9];
                    iflux<R, EX>(q, c_h, umax, Fx, G);
#pragma unroll
                    for (int k = 0; k < 9; k++) F[k] = Fx[k] * n0 + G[k] * n1;
                    V[0] = q[5];
                    V[1] = q[6];
                } else {
                    iflux_n<R>(q, c_h, n0, n1, umax, F);
                    V[0] = q[5] * n0 + q[6] * n1;
                }
            } else {
                // face point (interfaceflux, CYCLOCFLUX, BCFLUX, PROCINTFLUX)
                const int2 rec = r == 0 ? rec0 : recN;
                const int lf = r == 0 ? lf0 : lfN, np = r == 0 ? np0 : npN;
                const int kind = rec.y & 0xff, plf = (rec.y >> 8) & 0xff;
                const bool own_right = kind == kFaceRight;
                R other[9], m0 = n0, m1 = n1;
                int sign_l = r == 0 ? -1 : 1, sign_r = 1;
                if (kind == kFaceLeft || own_right) {
                    const R *tp = sX + c * TS + (lf - 1) * TFS + (N - 1 - np);
#pragma unroll
                    for (int k = 0; k < 9; k++) other[k] = tp[k * N];
                    const bool plow = plf == 1 || plf == 4;  // the partner's line starts at this face
                    if (!own_right) {
                        sign_r = plow ? 1 : -1;
                    } else {
                        const P2<R> pn = sP[(r == 0 ? 0 : NT) + tid];  // the left (partner) cell's normal
                        m0 = pn.x;
                        m1 = pn.y;
                        sign_l = plow ? -1 : 1;
                        sign_r = r == N ? -1 : 1;
                    }
                } else if (kind == kFaceProc) {
                    // the received trace, remote point N+1-nfp (procintflux_all.f90:83-99)
                    const R *rv = reinterpret_cast<const R *>(a.proc_recv) + ((size_t)rec.x * N + (N - 1 - np)) * 9;
#pragma unroll
                    for (int k = 0; k < 9; k++) other[k] = rv[k];
                } else {
                    bc_ghost<R, EX>(kind, q, n0, n1, a.vismode, a.cases ? a.cases[cs].fs : a.fs, other);
                }
                R Ql[9], Qr[9];
#pragma unroll
                for (int k = 0; k < 9; k++) {
                    Ql[k] = own_right ? other[k] : q[k];
                    Qr[k] = own_right ? q[k] : other[k];
                }
                if (!(Ql[0] > (R)0) || !(Qr[0] > (R)0)) err |= kErrNonPositiveDensity;
                R eig_face;
                rusanov<R, EX>(Ql, Qr, F, (R *)nullptr, m0, m1, sign_l, sign_r, c_h, eig_face, umax);
                if (!(Abs(eig_face) < (R)INFINITY)) err |= kErrNonFiniteWaveSpeed;
                if (eig_face > eigmax) eigmax = eig_face;
                // the right cell's slot: the left one's with both signs
                const R so = own_right ? (R)(sign_l * sign_r) : (R)1;
#pragma unroll
                for (int k = 0; k < 9; k++) F[k] = so * F[k];
                const R bxa = (R)0.5 * Ql[5] + (R)0.5 * Qr[5], bya = (R)0.5 * Ql[6] + (R)0.5 * Qr[6];
                if constexpr (kBn) {
                    V[0] = bxa * n0 + bya * n1;  // this cell's normal
                } else {
                    V[0] = bxa;
                    V[1] = bya;
                }
            }
        };
        // its share of the derivatives (compresid.f90:14-32) and of div B
        auto accumulate = [&](const int r, const R (&F)[9], const R (&V)[2], const P2<R> &n) {
#pragma unroll
            for (int i = 0; i < N; i++) {
                const P2<R> M2 = opM2<R>(ops, r * N + i);
#pragma unroll
                for (int k = 0; k < K2; k++) {
                    P2<R> f2;
                    f2.x = F[2 * k];
                    f2.y = F[2 * k + 1];
                    d[i][k] = fma2(f2, M2, d[i][k]);
                }
                if constexpr (kBn) {
                    P2<R> f2;
                    f2.x = F[8];
                    f2.y = V[0];
                    d[i][K2] = fma2(f2, M2, d[i][K2]);
                } else {
                    d[i][K2].x = d[i][K2].x + F[8] * M2.x;
                    d[i][K2].y = d[i][K2].y + V[0] * M2.x * n.x;
                    dy[i] = dy[i] + V[1] * M2.x * n.y;
                }
            }
        };
        R F[9], V[2], G[9], W[2];
        P2<R> n, m;
        flux_at(0, F, V, n);
        if constexpr (!kHold) flux_at(N, G, W, m);
        accumulate(0, F, V, n);
#pragma unroll 1
        for (int r = 1; r < N; r++) {
            flux_at(r, F, V, n);
            accumulate(r, F, V, n);
        }
        if constexpr (kHold) flux_at(N, G, W, m);
        accumulate(N, G, W, m);
    }
    // the tile's maxima, sent while its points are finished (every one of them
    // is non-negative, so they order as their bit patterns)
    const int lane = tid & 31, wid = tid >> 5;
    constexpr int NW = NT / 32;
    double em, um;
    if constexpr (sizeof(R) == sizeof(float)) {
        em = (double)__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(eigmax)));
        um = (double)__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(umax)));
    } else {
        em = warp_max_nonneg((double)eigmax);
        um = warp_max_nonneg((double)umax);
    }
    const unsigned eb = __reduce_or_sync(0xffffffffu, err);
    if (lane == 0) {
        sRed[wid] = em;
        sRed[NW + wid] = um;
        if (eb) raise_fault(a.err_flags, eb);
    }
    __syncthreads();  // the neighbours' traces are read: sX is free
    if (tid == 0) {
        double m0 = 0.0, m1 = 0.0;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            m0 = sRed[w] > m0 ? sRed[w] : m0;
            m1 = sRed[NW + w] > m1 ? sRed[NW + w] : m1;
        }
        if (a.cta_max) {
            a.cta_max[2 * tile] = m0;
            a.cta_max[2 * tile + 1] = m1;
        }
        if (first_tile) {  // carry the previous stages' maxima forward
            m0 = sCarry[0] > m0 ? sCarry[0] : m0;
            m1 = sCarry[1] > m1 ? sCarry[1] : m1;
        }
        atomic_max_nonneg(&maxima[2 * a.slot_w], m0);
        atomic_max_nonneg(&maxima[2 * a.slot_w + 1], m1);
    }

    // ---- 3: hand over the sums of the points the crossing line finishes ------------
    // point t of the line is finished by this thread if (t + l + fam) is even
    const int par = (l ^ fam) & 1;
    const int pt0 = fam == 0 ? N * l : l, pts = fam == 0 ? 1 : N;  // point t of the line: pt0 + pts*t
    if (act) {
        R *x = sX + c * XS;
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (2 * m + 1 < N || par) {
                R *o = x + (pt0 + pts * (2 * m + 1 - par)) * ND;
#pragma unroll
                for (int k = 0; k <= K2; k++) {
                    P2<R> v;
                    v.x = par ? d[i0][k].x : d[i1][k].x;
                    v.y = par ? d[i0][k].y : d[i1][k].y;
                    if constexpr (sizeof(R) == sizeof(float)) {
                        reinterpret_cast<P2<R> *>(o)[k] = v;
                    } else {
                        o[2 * k] = v.x;
                        o[2 * k + 1] = v.y;
                    }
                }
                if constexpr (EX) o[10] = par ? dy[i0] : dy[i1];
            }
        }
    }
    __syncthreads();

    // ---- 4: sources, residual and RK update of this thread's points -----------------
    const double cdt = a.cases ? a.cases[cs].dt : a.dt;
    auto cf = [&](int i) -> double { return ((a.dt_mask >> i) & 1u) ? a.cb[i] * cdt : a.cb[i]; };
    const double k0 = cf(0), k1 = cf(1), k2 = cf(2);
    double part_r = 0.0, part_d = 0.0;
    if (act) {
#pragma unroll
        for (int m = 0; m < NH; m++) {
            const int i0 = 2 * m, i1 = 2 * m + 1 < N ? 2 * m + 1 : 2 * m;
            if (!(2 * m + 1 < N) && par) continue;
            const int pt = pt0 + pts * (2 * m + par);
            const R *x = sX + c * XS + pt * ND;
            // the sums of both lines through the point
            R e[10], ey = (R)0;
#pragma unroll
            for (int k = 0; k <= K2; k++) {
                P2<R> v;
                if constexpr (sizeof(R) == sizeof(float)) {
                    v = reinterpret_cast<const P2<R> *>(x)[k];
                } else {
                    v.x = x[2 * k];
                    v.y = x[2 * k + 1];
                }
                e[2 * k] = (par ? d[i1][k].x : d[i0][k].x) + v.x;
                e[2 * k + 1] = (par ? d[i1][k].y : d[i0][k].y) + v.y;
            }
            if constexpr (EX) ey = (par ? dy[i1] : dy[i0]) + x[10];
            // Jac, or its reciprocal where the array holds reciprocals
            const double Jv = sJac[c * NJ + pt];
            double J = Jv, rJ = Jv;
            if constexpr (!EX) {
                if (!a.jac_inv) rJ = 1.0 / Jv;
            }
            double divB = 0.0;
            if constexpr (!EX) {
                if (a.vismode == 1) divB = (double)e[9] * rJ;
            }
            const size_t g = (size_t)(c0 + c) * NQ + 9 * pt;
            double res[9];
#pragma unroll
            for (int k = 0; k < 9; k++) {
                res[k] = (double)(-e[k]);
                // the viscous chain (compresid.f90:34-49); it adds exactly +0.0
                // when mu == eta0 == 0, which only the exact form reproduces
                if constexpr (EX) {
                    if (a.vismode == 1) res[k] = res[k] + (a.visc ? a.visc[g + k] : 0.0);
                } else {
                    if (a.vismode == 1 && a.visc) res[k] = res[k] + a.visc[g + k];
                }
            }
            const double *q = sQ + c * QS + 9 * pt;
            double *ap = sA + c * QS + 9 * pt;
            if constexpr (EX) {
                // the residual and the two terms of div B over J
                double num[11];
#pragma unroll
                for (int k = 0; k < 9; k++) num[k] = res[k];
                num[9] = (double)e[9];
                num[10] = (double)ey;
                quotients<11>(num, J, num);
#pragma unroll
                for (int k = 0; k < 9; k++) res[k] = num[k];
                if (a.vismode == 1) divB = num[9] + num[10];
            } else {
#pragma unroll
                for (int k = 0; k < 9; k++) res[k] = res[k] * rJ;
            }
            double qv[9];
#pragma unroll
            for (int k = 0; k < 9; k++) qv[k] = q[k];
            // compresid.f90:53-78: Powell 8-wave and GLM sources
            const double Bx = qv[5], By = qv[6], Bz = qv[7], psi = qv[8];
            double ux, uy, uz;
            if constexpr (EX) {
                double uu[3];
                quotients<3>(qv + 1, qv[0], uu);
                ux = uu[0]; uy = uu[1]; uz = uu[2];
            } else {
                const double ri = 1.0 / qv[0];
                ux = qv[1] * ri; uy = qv[2] * ri; uz = qv[3] * ri;
            }
            res[1] = res[1] - divB * Bx;
            res[2] = res[2] - divB * By;
            res[3] = res[3] - divB * Bz;
            res[4] = res[4] - divB * ((ux * Bx + uy * By) + uz * Bz);
            res[5] = res[5] - divB * ux;
            res[6] = res[6] - divB * uy;
            res[7] = res[7] - divB * uz;
            res[8] = res[8] - a.alpha * psi;
            if (a.mon_part) {
#pragma unroll
                for (int k = 0; k < 9; k++) part_r += res[k] * res[k];
                part_d += divB * divB;
            }
            // the RK stage update (iterations.f90:88-213); the point's slots are
            // this thread's alone
            double o[9];
            if (kind == kRkAxpy) {
#pragma unroll
                for (int k = 0; k < 9; k++) o[k] = qv[k] + k0 * res[k];
            } else if (kind == kRkTwoReg) {
#pragma unroll
                for (int k = 0; k < 9; k++) o[k] = (k1 * ap[k] + k2 * qv[k]) + k0 * res[k];
            } else if (kind == kRkTwoRegT) {
#pragma unroll
                for (int k = 0; k < 9; k++) o[k] = (k1 * ap[k] + k2 * qv[k]) + (k0 * res[k]) * cf(3);
            } else if constexpr (KIND != -2) {  // kRkFive: its other terms lie in ap
#pragma unroll
                for (int k = 0; k < 9; k++) o[k] = ap[k] + k0 * res[k];
            } else {
#pragma unroll
                for (int k = 0; k < 9; k++)
                    o[k] = ((((k1 * a.reg_a[g + k] + k2 * a.reg_b[g + k]) + cf(3) * a.reg_c[g + k]) + cf(4) * qv[k]) +
                            cf(5) * a.reg_d[g + k]) +
                           k0 * res[k];
            }
#pragma unroll
            for (int k = 0; k < 9; k++) ap[k] = o[k];
            if (a.resid_w) {
#pragma unroll
                for (int k = 0; k < 9; k++) a.resid_w[g + k] = res[k];
            }
            // the float form's copy for step 5, in the point's exchange slot
            // (read above, by this thread alone)
            if constexpr (sizeof(R) != sizeof(double)) {
                R *qf = sX + c * XS + pt * ND;
#pragma unroll
                for (int k = 0; k < K2; k++) {
                    P2<R> v;
                    v.x = (R)o[2 * k];
                    v.y = (R)o[2 * k + 1];
                    reinterpret_cast<P2<R> *>(qf)[k] = v;
                }
                qf[8] = (R)o[8];
            }
        }
    }
    fence_proxy_async();  // sA is the source of the bulk store below
    __syncthreads();

    // ---- the output store ---------------------------------------------------------
    const size_t g0 = (size_t)c0 * NQ;
    double *dst = a.q_out + g0;
    const bool out_bulk = (((uintptr_t)dst | cbytes) & 15) == 0;
    if (out_bulk) {
        if (tid < (S::kPad ? ncl : 1)) bulk_s2g(dst + (size_t)tid * NQ, sA + tid * QS, cbytes);
    } else {
        for (int k = tid; k < ncl * NQ; k += NT) {
            const int cc = k / NQ;
            dst[k] = sA[cc * QS + (k - cc * NQ)];
        }
    }

    // where the output's traces are collected (see LineSmem)
    R *sT = sizeof(R) == sizeof(double) ? sX
            : S::kTOwn ? reinterpret_cast<R *>(smem_raw + line_smem_bytes<N, CPB, R, EX>()) - CPB * TS
                       : reinterpret_cast<R *>(sQ);

    // ---- 5: the output's face traces for the next stage's neighbours ------------------
    if (act) {
        constexpr int PS = sizeof(R) == sizeof(double) ? 9 : ND;  // R per point
        const R *qo = sizeof(R) == sizeof(double) ? reinterpret_cast<const R *>(sA) + c * QS : sX + c * XS;
        qo += fam == 0 ? PS * N * l : PS * l;
        const int stride = fam == 0 ? PS : PS * N;
        R *t0 = sT + c * TS + (lf0 - 1) * TFS + np0, *tN = sT + c * TS + (lfN - 1) * TFS + npN;
        P2<R> s0[K2], sN[K2];
        R s08 = (R)0, sN8 = (R)0;
#pragma unroll
        for (int k = 0; k < K2; k++) s0[k] = sN[k] = splat2<R>((R)0);
#pragma unroll
        for (int s = 0; s < N; s++) {
            const R *o = qo + stride * s;
            const P2<R> L0 = opL2<R>(ops, s), LN = opL2<R>(ops, N * N + s);
#pragma unroll
            for (int k = 0; k < K2; k++) {
                P2<R> v;
                if constexpr (sizeof(R) == sizeof(float)) {
                    v = reinterpret_cast<const P2<R> *>(o)[k];
                } else {
                    v.x = o[2 * k];
                    v.y = o[2 * k + 1];
                }
                s0[k] = fma2(v, L0, s0[k]);
                sN[k] = fma2(v, LN, sN[k]);
            }
            s08 = s08 + o[8] * L0.x;
            sN8 = sN8 + o[8] * LN.x;
        }
#pragma unroll
        for (int k = 0; k < K2; k++) {
            t0[(2 * k) * N] = s0[k].x;
            t0[(2 * k + 1) * N] = s0[k].y;
            tN[(2 * k) * N] = sN[k].x;
            tN[(2 * k + 1) * N] = sN[k].y;
        }
        t0[8 * N] = s08;
        tN[8 * N] = sN8;
    }
    fence_proxy_async();

    // ---- the monitors' sums, the traces' store ----------------------------------------
    double pr = 0.0, pd = 0.0;
    if (a.mon_part) {
        pr = warp_sum(part_r);
        pd = warp_sum(part_d);
    }
    if (a.mon_part && lane == 0) {
        sRed[2 * NW + wid] = pr;
        sRed[3 * NW + wid] = pd;
    }
    __syncthreads();
    if (tid < 32) {
        // the traces, per cell (their buffer's records are whole 16-byte units)
        if (a.t_out && tid < ncl)
            bulk_s2g(reinterpret_cast<R *>(a.t_out) + (size_t)(c0 + tid) * 4 * TFS, sT + tid * TS,
                     (unsigned)(4 * TFS * sizeof(R)));
        if (tid == 0) {
            if (a.mon_part) {
                double s0 = 0.0, s1 = 0.0;
#pragma unroll
                for (int w = 0; w < NW; w++) {
                    s0 += sRed[2 * NW + w];
                    s1 += sRed[3 * NW + w];
                }
                a.mon_part[2 * tile] = s0;
                a.mon_part[2 * tile + 1] = s1;
            }
            mbar_inval(&sBar);
        }
        // every lane's bulk stores have read shared memory before it goes
        bulk_wait_read();
    }
    return true;
}

// KIND: the stage's RkKind, or -1 for any (read from the arguments; -2 in the
// persistent kernel)
template <int N, int CPB, typename R, bool EXACT, int KIND, bool WIDE>
__global__ void __launch_bounds__(line_threads(N, CPB), (line_min_blocks<N, CPB, R, EXACT, WIDE>()))
    line_kernel(const StageArgs a, const Ops ops)
{
    line_tile<N, CPB, R, EXACT, KIND, WIDE>(a, ops, blockIdx.x);
}

// a batch's stage as a persistent launch: each CTA walks the tile table with
// a grid stride
template <int N, int CPB, typename R, bool EXACT, bool WIDE>
__global__ void __launch_bounds__(line_threads(N, CPB), (line_min_blocks<N, CPB, R, EXACT, WIDE>()))
    line_kernel_persistent(const StageArgs a, const Ops ops)
{
    for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
        if (!line_tile<N, CPB, R, EXACT, -2, WIDE>(a, ops, t)) return;
        __syncthreads();  // tile t's last shared-memory reads before tile t+grid stages
    }
}

}  // namespace sddc
