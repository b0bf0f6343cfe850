// What the stage kernels share (their arguments, operators, TMA copies, face
// traces), and the RK stage of the exact form by tiles, for the meshes and
// batches on which that is faster (exact_by_tiles).  Every other stage runs in line_kernel
// (line_kernel.cuh), a residual evaluation in resid_kernel
// (resid_kernel.cuh), both with a thread per line of solution points.
//
// One launch evaluates compresid (compresid.f90:1-80, compflux.f90:1-104,
// interfaceflux_all.f90:1-112, cyclocflux_all.f90:1-112, bcflux.f90:1-377,
// nablaQsp compflux.f90:107-157) for every cell and applies the RK stage
// update (iterations.f90:88-213).
//
// Work split: one CTA owns CPB consecutive cells (tile_cells) and stages them in
// shared memory.  Phases, separated by __syncthreads:
//   A  Lagrange interpolation of every line of solution points to its N+1
//      flux points (one thread per cell x line index x variable: the xi-
//      and eta-line of one index share the operator row);
//   B1 physical flux at the interior flux points (thread per point);
//   B2 Rusanov flux at the 4N face points of each cell (thread per point).
//      The neighbour's trace at the face point comes from the trace buffer
//      (trace_at) that the stage producing the input published.  Each
//      shared face is evaluated by both of its cells, each with the
//      reference's left/right assignment, so both get the value the
//      reference scatters to them;
//   C  divergence of the flux, B gradients from the face-averaged flux-point
//      states, Powell and GLM sources and the RK update (thread per solution
//      point): the RK register slice was staged by TMA with the state, the
//      output is formed in shared memory and stored by one TMA bulk copy
//      while phase F runs;
//   F  the face traces of the output state, published for the next stage.
// Running maxima of the wave speed and of the velocity (the c_h input of
// the next stage) go through atomicMax on five rotating slots, so that
// launches need no host synchronisation.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "physics.cuh"

namespace sddc {

constexpr int kMaxN = 6;

// threads of a CTA of the kernel by tiles: one per face point (4N a cell), in
// the 6-cell tile of N >= 5 one per solution point; whole warps
__host__ __device__ constexpr int stage_threads(int n, int cpb)
{
    return ((cpb == 6 && n >= 5 ? n * n : 4 * n) * cpb + 31) / 32 * 32;
}

// Cells per CTA of the kernels by lines (2N threads per cell): one or two
// warps with few idle lanes.
__host__ __device__ constexpr int line_tile_cells(int n)
{
    return n == 2 ? 8 : n == 3 ? 10 : n == 4 ? 8 : n == 5 ? 6 : 2;
}

// Cells per CTA of the kernel by tiles.  us per stage with 4, 6 and 8: N = 2, 8100 cells 12.0, 16.8,
// 11.5; N = 3, 4096 11.9, 13.2, 13.2; N = 4, 14400 45.7, 47.3, 43.7; N = 5, 576 11.3,
// 9.7, 12.8, 14400 80, 71, 92; N = 6, 576 12.6, 11.4, 14.4, 8100 71, 65, 62
__host__ __device__ constexpr int tile_cells(int n, int ncell)
{
    return n == 3 ? 4 : n == 5 || (n == 6 && ncell < 148 * 8) ? 6 : 8;
}

// operators in kernel parameter space (row-major)
struct Ops {
    double L[(kMaxN + 1) * kMaxN];   // L[r*N + s]  = Lmat(r+1, s+1)
    double M[(kMaxN + 1) * kMaxN];   // M[r*N + s]  = Mmat(r+1, s+1)
    double H[(kMaxN - 1) * kMaxN];   // H[l*N + s]  = hhval(s+1, Xs_low(l+1))
    double HL[kMaxN * (kMaxN - 1)];  // HL[s*(N-1) + l] = hhval_low(l+1, Xs(s+1))
    float Lf[(kMaxN + 1) * kMaxN];
    float Mf[(kMaxN + 1) * kMaxN];
    // (L, L) and (M, M): operands of paired FMAs as they are read
    float2 Lp[(kMaxN + 1) * kMaxN];
    float2 Mp[(kMaxN + 1) * kMaxN];
    // element k = r*N + s of both operators, in every type
    __host__ __device__ void set(int k, double l, double m)
    {
        L[k] = l;
        M[k] = m;
        Lf[k] = (float)l;
        Mf[k] = (float)m;
        Lp[k] = make_float2(Lf[k], Lf[k]);
        Mp[k] = make_float2(Mf[k], Mf[k]);
    }
};

// how the stage output is formed from the residual r of the stage input q
enum RkKind : int {
    kRkNone = 0,     // residual evaluation only (compresid)
    kRkAxpy = 1,     // out = q + c0*r                                     RK_S5P3 stages 1-2, FiveStageRk stage 1
    kRkTwoReg = 2,   // out = (c1*a + c2*q) + c0*r                         RK_S5P3 stages 3-5, FiveStageRk stages 3-4
    kRkTwoRegT = 3,  // out = (c1*a + c2*q) + (c0*r)*c3                    FiveStageRk stage 2
    kRkFive = 4      // out = ((((c1*a + c2*b) + c3*c) + c4*q) + c5*d) + c0*r   FiveStageRk stage 5
};

// Where kernels leave fault bits, in device memory: OR-ed into its word and, by the
// warp that first finds a bit missing there, into the host's (pinned; null
// where the caller copies the device word), which is read after a
// synchronisation without a copy.  A diverged mesh faults in every warp of every
// stage: with all of them OR-ed across the host link a stage of 131072 cells
// (N = 5, FP64) took 41.7 ms, so 0.39 (0.34 without a fault).
struct FaultFlags {
    unsigned bits, pad;
    unsigned *host;
};
__device__ __forceinline__ void raise_fault(FaultFlags *f, unsigned bits)
{
    const unsigned seen = atomicOr(&f->bits, bits);
    if ((bits & ~seen) && f->host) atomicOr(f->host, bits);
}

// per-case data of a batch of independent cases sharing one launch
struct CaseParams {
    Freestream fs;
    double dt;
    double pad;
};

struct StageArgs {
    int ncell;
    int vismode;
    int artiv;
    int rk_kind;
    int slot_r, slot_w;
    double alpha;
    // RK coefficients of the stage: c[i] = cb[i] * dt when bit i of dt_mask
    // is set, else cb[i] (the products round as the host's would)
    double cb[8];
    unsigned dt_mask;
    int kinds;                         // how many different RkKinds a step's stages have
    double dt;                         // single case
    Freestream fs;                     // single case
    // batch: one tile per CTA (first cell, cells, case, 1 if the case's
    // first tile), per-case data and running maxima [case][5][2]; null for
    // a single case
    const int4 *tiles;
    int ntiles;
    // batch launched persistently: each CTA walks the tile table with a grid
    // stride (the table is ordered largest case first); 0: one CTA per tile
    int persistent;
    int ahead;  // tiles resident at once (set by the launch)
    const CaseParams *cases;
    const double *__restrict__ q_in;   // (9,N,N,NCELL), never written during the stage
    double *q_out;                     // RK output (may be reg_a: FiveStageRk stage 5)
    const void *__restrict__ t_in;     // face traces of q_in, R[NCELL][4][tfs] (trace_at)
    void *t_out;                       // face traces of q_out (null: not produced)
    int tfs;                           // stride of a face's record in both
    const double *reg_a;               // RK registers read by this stage
    const double *reg_b;
    const double *reg_c;
    const double *reg_d;
    double *resid_w;                   // residual copy (FiveStageRk stage 4 resid0)
    const double *__restrict__ met;    // packed metrics, per cell (residual evaluations)
    // the same metrics split for the stages: normals in the arithmetic type
    // [NCELL][4N(N+1)] and Jac [NCELL][MetLayout::kJacPad]
    const void *__restrict__ nrm;
    const double *__restrict__ jac;
    int jac_inv;                       // jac holds 1/Jac (the forms other than the exact one)
    const int2 *__restrict__ faces;    // (cell, local face) records
    // remote traces of the processor faces of a decomposed run, [slot][nfp][9]
    // in the sending rank's point order (procintflux_all.f90:83-99)
    const void *__restrict__ proc_recv;
    double *maxima;                    // [5][2]: running max of eigv, umax
    double *__restrict__ sm_ind;       // (2,NCELL) AV sensor
    double *__restrict__ resid_out;    // (9,N,N,NCELL), residual evaluation only (null: not kept)
    double *__restrict__ grad_out;     // (9,2,N,N,NCELL), residual evaluation only (null: not kept)
    double *__restrict__ mon_part;     // per-CTA (sum resid^2, sum divB^2), or null
    double *__restrict__ cta_max;      // per-CTA (max eigv, max umax) of this stage, or null
    const double *__restrict__ visc;   // dFv + dGv (9,N,N,NCELL) of the viscous chain, or null (mu = eta0 = 0)
    FaultFlags *err_flags;
};

// beside the state and the traces, what a launch of the face traces takes: the
// fault flags and, where not null, the running-max slots it sets to a seed
struct TraceInit {
    FaultFlags *flags;
    double *maxima = nullptr;
    double eig = 0.0, um = 0.0;
};

// packed per-cell metric record: normals of both flux-point families, then Jac
template <int N> struct MetLayout {
    static constexpr int kFam = 2 * N * (N + 1);       // doubles per family
    static constexpr int kJac = 2 * kFam;              // offset of Jac(i,j) at kJac + i + N*j
    static constexpr int kSize = (2 * kFam + N * N + 1) & ~1;
    static constexpr int kJacPad = (N * N + 1) & ~1;  // Jac per cell in the split layout (16-byte rows)
    // normal (S1(1,1:2) or S2(2,1:2)) of family f, line l, flux point r
    __host__ __device__ static constexpr int normal(int f, int l, int r) { return f * kFam + 2 * (l * (N + 1) + r); }
};

// error flag bits
enum : unsigned { kErrNonPositiveDensity = 1u, kErrNonFiniteWaveSpeed = 2u, kErrStagingTimeout = 16u };

// ---- one-dimensional TMA bulk copies into shared memory, completed on an
// mbarrier (PTX mbarrier.*, cp.async.bulk) -------------------------------------
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_inval(unsigned long long *bar)
{
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
// dst and src 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait (each try_wait may suspend the thread briefly); false if it
// gave up
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long *bar, unsigned parity)
{
    for (int it = 0; it < (1 << 22); it++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// shared-memory writes of this thread made visible to the bulk-copy (async)
// proxy, before a barrier after which one thread issues a bulk store
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// shared -> global bulk store; src and dst 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_s2g(void *dst, const void *src, unsigned bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_addr(src)),
                 "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// the issuing thread's bulk stores have read their shared-memory source
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// a hint that brings [src, src + bytes) into L2; src 16-byte aligned, bytes a
// multiple of 16, the range inside one allocation
__device__ __forceinline__ void bulk_prefetch_l2(const void *src, unsigned bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

template <int N> struct Smem {
    static constexpr int NQ = 9 * N * N;
    static constexpr int NP = N + 1;
    static constexpr int kF = 2 * N * NP * 9;  // per cell: state then flux at every flux point
    static constexpr int kV = 2 * N * NP * 2;  // per cell: face-averaged Bx, By at every flux point
};

// Lagrange coefficient access in the arithmetic type
template <typename R> __device__ __forceinline__ R opL(const Ops &o, int i);
template <> __device__ __forceinline__ double opL<double>(const Ops &o, int i) { return o.L[i]; }
template <> __device__ __forceinline__ float opL<float>(const Ops &o, int i) { return o.Lf[i]; }
template <typename R> __device__ __forceinline__ R opM(const Ops &o, int i);
template <> __device__ __forceinline__ double opM<double>(const Ops &o, int i) { return o.M[i]; }
template <> __device__ __forceinline__ float opM<float>(const Ops &o, int i) { return o.Mf[i]; }


// two lanes of the arithmetic type through one paired FMA (FFMA2 for float,
// each component rounded as fmaf; for double two scalar multiply-adds, in
// the order a + x*y of the scalar code)
template <typename R> struct Pair2;
template <> struct Pair2<float> { using T = float2; };
template <> struct Pair2<double> { using T = double2; };
template <typename R> using P2 = typename Pair2<R>::T;
__device__ __forceinline__ float2 fma2(float2 x, float2 y, float2 z) { return __ffma2_rn(x, y, z); }
__device__ __forceinline__ double2 fma2(double2 x, double2 y, double2 z)
{
    return make_double2(z.x + x.x * y.x, z.y + x.y * y.y);
}
template <typename R> __device__ __forceinline__ P2<R> splat2(R v)
{
    P2<R> p;
    p.x = v;
    p.y = v;
    return p;
}

template <typename R> __device__ __forceinline__ P2<R> opL2(const Ops &o, int i);
template <> __device__ __forceinline__ P2<double> opL2<double>(const Ops &o, int i) { return splat2<double>(o.L[i]); }
template <> __device__ __forceinline__ P2<float> opL2<float>(const Ops &o, int i) { return o.Lp[i]; }
template <typename R> __device__ __forceinline__ P2<R> opM2(const Ops &o, int i);
template <> __device__ __forceinline__ P2<double> opM2<double>(const Ops &o, int i) { return splat2<double>(o.M[i]); }
template <> __device__ __forceinline__ P2<float> opM2<float>(const Ops &o, int i) { return o.Mp[i]; }

// local face lf (1..4), face point nfp (1..N) -> flux point (family, line, point)
// (face2fpconnec, initsetup.f90:347-383)
template <int N>
__device__ __forceinline__ void face_point(int lf, int nfp, int &fam, int &line, int &r)
{
    switch (lf) {
    case 1: fam = 1; line = nfp - 1; r = 0; break;       // (nfp, 1)
    case 2: fam = 0; line = nfp - 1; r = N; break;       // (N+1, nfp)
    case 3: fam = 1; line = N - nfp; r = N; break;       // (N-nfp+1, N+1)
    default: fam = 0; line = N - nfp; r = 0; break;      // (1, N-nfp+1)
    }
}

// face traces of a state, [cell][local face][variable][face point]: the N
// points of one face, which consecutive lanes read and write, are adjacent.
// tfs is the face record's stride; lf is 1-based, nfp0 0-based.
template <int N>
__host__ __device__ __forceinline__ size_t trace_at(int tfs, size_t cell, int lf, int nfp0, int k)
{
    return (cell * 4 + (size_t)(lf - 1)) * tfs + (size_t)(k * N + nfp0);
}
// the stride of a context's records in values of elem bytes: 9N rounded up to
// whole 16-byte units, so that asynchronous copies move a face at a time
// (6.7% more at N = 5 in the mixed form, none at N = 4).  The allocation-free
// entry packs its records (stride 9N) where its fixed scratch array holds no more.
__host__ __device__ constexpr int trace_stride(int n, int elem) { return (9 * n * elem + 15) / 16 * 16 / elem; }
template <int N, typename R> __host__ __device__ constexpr int trace_stride() { return trace_stride(N, sizeof(R)); }

template <typename T> __device__ __forceinline__ T warp_max(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        T w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    return v;
}

// the same of non-negative doubles, which order as their bit patterns
__device__ __forceinline__ double warp_max_nonneg(double v)
{
    const unsigned hi = (unsigned)__double2hiint(v), top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = __reduce_max_sync(0xffffffffu, hi == top ? (unsigned)__double2loint(v) : 0u);
    return __hiloint2double((int)top, (int)lo);
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int N, int CPB> constexpr size_t stage_smem_bytes()
{
    using S = Smem<N>;
    return sizeof(double) * ((size_t)CPB * (2 * S::NQ + MetLayout<N>::kJacPad + S::kF + S::kV + 2 * MetLayout<N>::kFam) +
                             4 * 32 + 2 * (N + 1) * N);
}

// CTAs per SM the kernel is compiled for: as many as the 228 KB of shared
// memory per SM hold (1 KB per CTA is the driver's), but no fewer than 96
// registers per thread, and at most 8
template <int N, int CPB> constexpr int stage_min_blocks()
{
    int b = (int)((228 * 1024) / (stage_smem_bytes<N, CPB>() + 1024));
    b = b < 1 ? 1 : (b > 8 ? 8 : b);
    while (b > 1 && 65536 / (stage_threads(N, CPB) * b) < 96) b--;
    return b;
}

// Compiled without FMA contraction (-fmad=false): the reference's operations
// in its order.  GEN: also the tiles of a batch, with their cases' data, and
// metrics from the packed records (a.nrm null: contexts of another form); a
// kernel of its own, so that a plain case does not carry them.  False if the
// staging copies did not arrive.
template <int N, int CPB, bool GEN>
__device__ __forceinline__ bool stage_tile(const StageArgs &a, const Ops &ops, const int tile)
{
    using R = double;
    using S = Smem<N>;
    using ML = MetLayout<N>;
    constexpr int NT = stage_threads(N, CPB);  // whole warps: the reductions use full-warp masks
    constexpr int NQ = S::NQ, NP = S::NP, NG = 2;
    constexpr int NN = N * N;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int NM = 2 * ML::kFam;  // normals per cell
    constexpr int NJ = ML::kJacPad;
    double *sQ = reinterpret_cast<double *>(smem_raw);          // [CPB][NQ]
    double *sJac = sQ + CPB * NQ;                                // [CPB][NJ]
    constexpr int NWR = 32;
    double *sRed = sJac + CPB * NJ;                              // [4][NWR] block reductions
    double *sA = sRed + 4 * NWR;                                 // [CPB][NQ] the RK register, then the output
    R *sNrm = sA + CPB * NQ;                                     // [CPB][NM] flux-point normals
    R *sF = sNrm + CPB * NM;                // [CPB][2][N][NP][9]
    R *sV = sF + CPB * S::kF;                                    // [CPB][2][N][NP][NG]
    // operators read with lane-dependent indices live in shared memory
    // (divergent reads of kernel parameters serialise per address)
    R *sOpL = sV + CPB * S::kV;                                  // [NP][N]
    R *sOpM = sOpL + NP * N;                                     // [NP][N]

    const int tid = threadIdx.x;
    int c0 = tile * CPB, ncl = min(CPB, a.ncell - c0), cs = 0;  // cells of this tile, their case
    bool first_tile = tile == 0;
    if (GEN && a.tiles) {
        const int4 tl = a.tiles[tile];
        c0 = tl.x;
        ncl = tl.y;
        cs = tl.z;
        first_tile = tl.w != 0;
    }
    double *maxima = a.maxima + 10 * cs;
    // a thread has one face point at most (a cell has 4N of them)
    const bool has_fp = tid < ncl * 4 * N;

    // ---- stage the state, the metrics and the operators ------------------------
    // The tile's state slice goes to sQ, its normals to sNrm and Jac to sJac
    // and, in a stage that reads one RK register, that register's slice to sA,
    // by TMA bulk copies that one thread issues.  Where the state slices are no
    // whole 16-byte units (odd N, an odd first cell or count) they come by
    // batches of loads.
    __shared__ __align__(8) unsigned long long sBar;
    __shared__ int sAbort;
    const bool want_ra = a.rk_kind == kRkTwoReg || a.rk_kind == kRkTwoRegT;
    const size_t qbytes = (size_t)ncl * NQ * sizeof(double);
    // normals and Jac from their own arrays, or both from the packed records
    // (where they lie one behind the other, as they do here per cell)
    const bool split = !GEN || a.nrm != nullptr;  // uniform
    static_assert(ML::kJac == NM && ML::kSize == NM + NJ && NM % 2 == 0 && NJ % 2 == 0,
                  "a record is a cell's normals, then its Jac, both whole 16-byte units");
    const R *nbase = split ? reinterpret_cast<const R *>(a.nrm) : a.met;
    const int nstride = split ? NM : ML::kSize;
    const double *qsrc = a.q_in + (size_t)c0 * NQ;
    const double *rsrc = want_ra ? a.reg_a + (size_t)c0 * NQ : nullptr;
    const bool bulk = (((uintptr_t)qsrc | (uintptr_t)rsrc | qbytes) & 15) == 0;  // uniform in the CTA
    if (tid == 0) {
        sAbort = 0;
        mbar_init(&sBar, 1);
        mbar_expect_tx(&sBar, (unsigned)(ncl * (NM + NJ) * sizeof(double) + (bulk ? qbytes * (want_ra ? 2 : 1) : 0)));
        if (bulk) bulk_g2s(sQ, qsrc, (unsigned)qbytes, &sBar);
        if (split) {
            bulk_g2s(sNrm, nbase + (size_t)c0 * NM, (unsigned)(ncl * NM * sizeof(R)), &sBar);
            bulk_g2s(sJac, a.jac + (size_t)c0 * NJ, (unsigned)(ncl * NJ * sizeof(double)), &sBar);
        } else {
            for (int c = 0; c < ncl; c++) {
                const double *rec = a.met + (size_t)(c0 + c) * ML::kSize;
                bulk_g2s(sNrm + c * NM, rec, NM * sizeof(R), &sBar);
                bulk_g2s(sJac + c * NJ, rec + ML::kJac, NJ * sizeof(double), &sBar);
            }
        }
        if (bulk && want_ra) bulk_g2s(sA, rsrc, (unsigned)qbytes, &sBar);
    }
    for (int k = tid; k < NP * N; k += NT) {
        sOpL[k] = opL<R>(ops, k);
        sOpM[k] = opM<R>(ops, k);
    }
    if (!bulk) {
        // batches of kU independent loads per thread before their stores, so
        // that each thread keeps several loads in flight
        auto stage_copy = [&](double *dst, const double *src) {
            constexpr int kU = 8;
            const int n = ncl * NQ;
            for (int k0 = tid; k0 < n; k0 += kU * NT) {
                double v[kU];
#pragma unroll
                for (int u = 0; u < kU; u++) v[u] = k0 + u * NT < n ? __ldg(src + k0 + u * NT) : 0.0;
#pragma unroll
                for (int u = 0; u < kU; u++)
                    if (k0 + u * NT < n) dst[k0 + u * NT] = v[u];
            }
        };
        stage_copy(sQ, qsrc);
        if (want_ra) stage_copy(sA, rsrc);
    }
    const double eig_r = maxima[2 * a.slot_r], um_r = maxima[2 * a.slot_r + 1];
    // compflux.f90:6 -- running maxima of all previous stages
    const R c_h = (R)sqrt(eig_r * (eig_r - um_r));
    if (tid == 0 && !mbar_wait_bounded(&sBar, 0)) {
        // the copies did not complete: flag it, give them time to land in
        // this CTA's shared memory, and leave (every thread, below)
        raise_fault(a.err_flags, kErrStagingTimeout);
        sAbort = 1;
        mbar_wait_bounded(&sBar, 0);
    }
    __syncthreads();
    if (sAbort) return false;
    // ---- A: interpolate every line to its flux points ---------------------------
    // one thread per (cell, line index l, variable): xi-line l and eta-line l
    // together, their sums paired (both use the same operator row)
    for (int t = tid; t < ncl * N * 9; t += NT) {
        const int v = t % 9, l = (t / 9) % N, c = t / (9 * N);
        const double *q = sQ + c * NQ + v;
        P2<R> qs[N];
#pragma unroll
        for (int s = 0; s < N; s++) {
            qs[s].x = (R)q[9 * (s + N * l)];
            qs[s].y = (R)q[9 * (l + N * s)];
        }
        R *ox = sF + c * S::kF + l * NP * 9 + v;  // xi-line l (family 0)
        R *oy = ox + N * NP * 9;                   // eta-line l (family 1)
#pragma unroll
        for (int r = 0; r < NP; r++) {
            P2<R> acc = splat2<R>((R)0);
#pragma unroll
            for (int s = 0; s < N; s++) acc = fma2(qs[s], opL2<R>(ops, r * N + s), acc);
            ox[r * 9] = acc.x;
            oy[r * 9] = acc.y;
        }
    }
    __syncthreads();

    R eigmax = (R)0, umax = (R)0;
    unsigned err = 0;

    // ---- B1: interior flux points (inviscid_flux_interior) ---------------------
    for (int t = tid; t < ncl * 2 * N * (N - 1); t += NT) {
        const int r = 1 + t % (N - 1), l = (t / (N - 1)) % N, f = (t / ((N - 1) * N)) % 2,
                  c = t / (2 * N * (N - 1));
        R *slot = sF + c * S::kF + ((f * N + l) * NP + r) * 9;
        R q[9];
#pragma unroll
        for (int k = 0; k < 9; k++) q[k] = slot[k];
        if (!(q[0] > (R)0)) err |= kErrNonPositiveDensity;
        const R *nrm = sNrm + c * NM + ML::normal(f, l, r);
        const R n0 = nrm[0], n1 = nrm[1];
        // the reference's F and G, projected
        R F[9], G[9];
        iflux<R, true>(q, c_h, umax, F, G);
#pragma unroll
        for (int k = 0; k < 9; k++) slot[k] = F[k] * n0 + G[k] * n1;
        R *vs = sV + c * S::kV + ((f * N + l) * NP + r) * NG;
        vs[0] = q[5];
        vs[1] = q[6];
    }

    // ---- B2: face points (interfaceflux, CYCLOCFLUX, BCFLUX) -------------------
    if (has_fp) {
        const int nfp = 1 + tid % N, lf = 1 + (tid / N) % 4, c = tid / (4 * N);
        int fam, line, r;
        face_point<N>(lf, nfp, fam, line, r);
        R *slot = sF + c * S::kF + ((fam * N + line) * NP + r) * 9;
        R own[9], Fl[9], Fr[9];
#pragma unroll
        for (int k = 0; k < 9; k++) own[k] = slot[k];
        const int2 frec = __ldg(a.faces + (size_t)c0 * 4 + tid / N);
        const int kind = frec.y & 0xff;
        const bool pair = kind == kFaceLeft || kind == kFaceRight;
        const bool own_right = kind == kFaceRight;
        const R *nrm = sNrm + c * NM + ML::normal(fam, line, r);
        R n0 = nrm[0], n1 = nrm[1], other[9];
        int sign_l = r == 0 ? -1 : 1, sign_r = 1;
        if (kind == kFaceProc) {
            // PROCINTFLUX / CYCREMFLUX (procintflux_all.f90:83-151): this cell
            // is the left cell; the received trace, remote point N+1-nfp
            const R *rv = reinterpret_cast<const R *>(a.proc_recv) + ((size_t)frec.x * N + (N - nfp)) * 9;
#pragma unroll
            for (int k = 0; k < 9; k++) other[k] = rv[k];
        } else if (pair) {
            // partner point N-nfp+1 on the partner's local face; its trace was
            // published by the stage that produced q_in
            const int pc = frec.x, plf = (frec.y >> 8) & 0xff;
            const R *tp = reinterpret_cast<const R *>(a.t_in);
#pragma unroll
            for (int k = 0; k < 9; k++) other[k] = tp[trace_at<N>(a.tfs, pc, plf, N - nfp, k)];
            int pfam, pline, pr;
            face_point<N>(plf, N - nfp + 1, pfam, pline, pr);
            if (own_right) {
                // the left (partner) cell's normal
                const R *pn = nbase + (size_t)pc * nstride + ML::normal(pfam, pline, pr);
                n0 = __ldg(pn);
                n1 = __ldg(pn + 1);
                sign_l = pr == 0 ? -1 : 1;
                sign_r = r == N ? -1 : 1;
            } else {
                sign_r = pr == N ? -1 : 1;
            }
        } else {
            bc_ghost<R, true>(kind, own, n0, n1, a.vismode, GEN && a.cases ? a.cases[cs].fs : a.fs, other);
        }
        // left and right states by element-wise selects (arrays picked
        // through a pointer would live in local memory)
        R Ql[9], Qr[9];
#pragma unroll
        for (int k = 0; k < 9; k++) {
            Ql[k] = own_right ? other[k] : own[k];
            Qr[k] = own_right ? own[k] : other[k];
        }
        if (!(Ql[0] > (R)0) || !(Qr[0] > (R)0)) err |= kErrNonPositiveDensity;
        R eig_face;
        rusanov<R, true>(Ql, Qr, Fl, Fr, n0, n1, sign_l, sign_r, c_h, eig_face, umax);
        if (!(Abs(eig_face) < (R)INFINITY)) err |= kErrNonFiniteWaveSpeed;
        if (eig_face > eigmax) eigmax = eig_face;
#pragma unroll
        for (int k = 0; k < 9; k++) slot[k] = own_right ? Fr[k] : Fl[k];
        R *vs = sV + c * S::kV + ((fam * N + line) * NP + r) * NG;
        vs[0] = (R)0.5 * Ql[5] + (R)0.5 * Qr[5];
        vs[1] = (R)0.5 * Ql[6] + (R)0.5 * Qr[6];
    }
    __syncthreads();

    // ---- C1: flux derivative along every line, in place ------------------------
    // one thread per (cell, line index, variable), the xi- and eta-line of
    // the index paired: the N+1 flux values of each line, d(i) = sum over r
    // of F(r) * M(r, i) in the reference's order (compresid.f90:14-32),
    // written over point slots 0..N-1 of the line
    for (int t = tid; t < ncl * N * 9; t += NT) {
        const int k = t % 9, l = (t / 9) % N, c = t / (9 * N);
        R *cx = sF + c * S::kF + l * NP * 9 + k;  // xi-line l
        R *cy = cx + N * NP * 9;                   // eta-line l
        P2<R> fv[NP];
#pragma unroll
        for (int r = 0; r < NP; r++) {
            fv[r].x = cx[r * 9];
            fv[r].y = cy[r * 9];
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            P2<R> d = splat2<R>((R)0);
#pragma unroll
            for (int r = 0; r < NP; r++) d = fma2(fv[r], opM2<R>(ops, r * N + i), d);
            cx[i * 9] = d.x;
            cy[i * 9] = d.y;
        }
    }
    __syncthreads();

    // ---- C: B gradient, sources and the residual per solution point ------------
    // the RK coefficients of the stage, formed where used from the kernel
    // parameters (not held in registers through the phase)
    const double cdt = GEN && a.cases ? a.cases[cs].dt : a.dt;
    auto cf = [&](int i) -> double { return ((a.dt_mask >> i) & 1u) ? a.cb[i] * cdt : a.cb[i]; };
    double part_r = 0.0, part_d = 0.0;
    for (int t = tid; t < ncl * NN; t += NT) {
        const int i = t % N, j = (t / N) % N, c = t / NN;
        const int cell = c0 + c;
        const R *met = sNrm + c * NM;
        const double J = sJac[c * NJ + i + N * j];
        const R *Fx = sF + c * S::kF + (0 * N + j) * NP * 9;  // xi-line j
        const R *Fy = sF + c * S::kF + (1 * N + i) * NP * 9;  // eta-line i
        const R *Vx = sV + c * S::kV + (0 * N + j) * NP * NG;
        const R *Vy = sV + c * S::kV + (1 * N + i) * NP * NG;
        // nablaQsp (compflux.f90:107-157) for the variables kept
        double gB[2][2] = {{0.0, 0.0}, {0.0, 0.0}};  // [Bx,By][x,y]
        // with vismode == 0 the reference never fills nablaQs; its divB
        // source then reads the zeros of the fresh allocation
#pragma unroll
        for (int g = 0; g < NG; g++) {
            if (a.vismode != 1) break;
            R ax = (R)0, ay = (R)0, bx = (R)0, by = (R)0;
#pragma unroll
            for (int r = 0; r < NP; r++) {
                const R mx = Vx[r * NG + g] * sOpM[r * N + i];
                ax = ax + mx * met[ML::normal(0, j, r)];
                ay = ay + mx * met[ML::normal(0, j, r) + 1];
            }
#pragma unroll
            for (int r = 0; r < NP; r++) {
                const R my = Vy[r * NG + g] * sOpM[r * N + j];
                bx = bx + my * met[ML::normal(1, i, r)];
                by = by + my * met[ML::normal(1, i, r) + 1];
            }
            gB[g][0] = (double)(ax + bx) / J;
            gB[g][1] = (double)(ay + by) / J;
        }
        const double divB = gB[0][0] + gB[1][1];
        // compresid.f90:12-51 divergence of the inviscid flux: the line sums
        // of phase C1 sit in point slot i of xi-line j and slot j of eta-line i
        double res[9];
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const R dF = Fx[i * 9 + k], dG = Fy[j * 9 + k];
            res[k] = (double)(-(dF + dG));
            // the viscous chain (compresid.f90:34-49); it adds exactly +0.0
            // when mu == eta0 == 0 (which turns a -0.0 residual into +0.0)
            if (a.vismode == 1) res[k] = res[k] + (a.visc ? a.visc[(size_t)cell * NQ + 9 * (i + N * j) + k] : 0.0);
        }
        // compresid.f90:53-78: 1/Jac, Powell 8-wave and GLM sources
        const double *q = sQ + c * NQ + 9 * (i + N * j);
        quotients<9>(res, J, res);
        const double Bx = q[5], By = q[6], Bz = q[7], psi = q[8];
        double uu[3];
        quotients<3>(q + 1, q[0], uu);
        const double ux = uu[0], uy = uu[1], uz = uu[2];
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
        double *ap = sA + c * NQ + 9 * (i + N * j);
        // the RK stage update of this point (iterations.f90:88-213);
        // the point's state and RK register slot are read by this thread
        // only, so the output goes to the register slot in place
        const size_t g = (size_t)cell * NQ + 9 * (i + N * j);
        const int kind = a.rk_kind;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const double qk = q[k], r = res[k];
            double o;
            switch (kind) {
            case kRkAxpy: o = qk + cf(0) * r; break;
            case kRkTwoReg: o = (cf(1) * ap[k] + cf(2) * qk) + cf(0) * r; break;
            case kRkTwoRegT: o = (cf(1) * ap[k] + cf(2) * qk) + (cf(0) * r) * cf(3); break;
            default:
                o = ((((cf(1) * a.reg_a[g + k] + cf(2) * a.reg_b[g + k]) + cf(3) * a.reg_c[g + k]) + cf(4) * qk) +
                     cf(5) * a.reg_d[g + k]) +
                    cf(0) * r;
                break;
            }
            ap[k] = o;
            if (a.resid_w) a.resid_w[g + k] = r;
        }
        fence_proxy_async();  // sA is the source of the bulk store below
    }
    __syncthreads();

    // ---- the output slice (formed in sA) to q_out: one bulk store issued by one
    // thread, read from shared memory while phase F runs, or coalesced stores
    // when the slice is not 16-byte aligned ----------------------------------------
    double *dst = a.q_out + (size_t)c0 * NQ;
    const int n = ncl * NQ;
    const bool out_bulk = (((uintptr_t)dst | (size_t)n * sizeof(double)) & 15) == 0;
    if (out_bulk) {
        if (tid == 0) bulk_s2g(dst, sA, (unsigned)(n * sizeof(double)));
    } else {
        for (int e = tid; e < n; e += NT) dst[e] = sA[e];
    }

    // ---- F: face traces of the output state for the next stage's neighbours ---
    // (the barrier after phase C orders its output before these reads: in a
    // time step nothing between them writes shared memory)
    if (a.t_out) {
        R *to = reinterpret_cast<R *>(a.t_out);
        const R *qo = sA;
        // one thread per (cell, family, variable, line): the line's N values
        // give the traces at both of its ends (r = 0 and r = N), each summed
        // in order as phase A sums them
        for (int t = tid; t < ncl * 2 * 9 * N; t += NT) {
            const int line = t % N, k = (t / N) % 9, fam = (t / (9 * N)) % 2, c = t / (18 * N);
            const R *q = qo + c * NQ + (fam == 0 ? 9 * N * line : 9 * line) + k;
            const int stride = fam == 0 ? 9 : 9 * N;
            R qs[N];
#pragma unroll
            for (int s = 0; s < N; s++) qs[s] = q[stride * s];
            R a0 = (R)0, aN = (R)0;
#pragma unroll
            for (int s = 0; s < N; s++) {
                a0 = a0 + qs[s] * sOpL[s];
                aN = aN + qs[s] * sOpL[N * N + s];
            }
            // the faces at the line's ends (face_point inverted): xi line j
            // ends on local faces 4 (point N-j) and 2 (point j+1), eta
            // line i on local faces 1 (point i+1) and 3 (point N-i)
            const int lf0 = fam == 0 ? 4 : 1, nfp0 = fam == 0 ? N - line : line + 1;
            const int lfN = fam == 0 ? 2 : 3, nfpN = fam == 0 ? line + 1 : N - line;
            to[trace_at<N>(a.tfs, c0 + c, lf0, nfp0 - 1, k)] = a0;
            to[trace_at<N>(a.tfs, c0 + c, lfN, nfpN - 1, k)] = aN;
        }
    }

    // ---- reductions ------------------------------------------------------------
    {
        const int lane = tid & 31, wid = tid >> 5;
        constexpr int NW = (NT + 31) / 32;
        const double em = warp_max(eigmax), um = warp_max(umax);
        unsigned e = __reduce_or_sync(0xffffffffu, err);
        double pr = 0.0, pd = 0.0;
        if (a.mon_part) {
            pr = warp_sum(part_r);
            pd = warp_sum(part_d);
        }
        if (lane == 0) {
            sRed[wid] = em;
            sRed[NWR + wid] = um;
            sRed[2 * NWR + wid] = pr;
            sRed[3 * NWR + wid] = pd;
            if (e) raise_fault(a.err_flags, e);
        }
        __syncthreads();
        if (tid == 0) {
            double m0 = 0.0, m1 = 0.0, s0 = 0.0, s1 = 0.0;
            for (int w = 0; w < NW; w++) {
                m0 = sRed[w] > m0 ? sRed[w] : m0;
                m1 = sRed[NWR + w] > m1 ? sRed[NWR + w] : m1;
                s0 += sRed[2 * NWR + w];
                s1 += sRed[3 * NWR + w];
            }
            atomic_max_nonneg(&maxima[2 * a.slot_w], m0);
            atomic_max_nonneg(&maxima[2 * a.slot_w + 1], m1);
            if (first_tile) {  // carry the previous stages' maxima forward
                // (re-read: slot_r is not written during the stage)
                atomic_max_nonneg(&maxima[2 * a.slot_w], maxima[2 * a.slot_r]);
                atomic_max_nonneg(&maxima[2 * a.slot_w + 1], maxima[2 * a.slot_r + 1]);
            }
            if (a.mon_part) {
                a.mon_part[2 * tile] = s0;
                a.mon_part[2 * tile + 1] = s1;
            }
            if (a.cta_max) {  // where the running maxima were raised (the adjoint's argmax)
                a.cta_max[2 * tile] = m0;
                a.cta_max[2 * tile + 1] = m1;
            }
            // the bulk store must have read sA before the CTA's shared memory
            // goes or the next tile reuses it; the staging barrier is free
            if (out_bulk) bulk_wait_read();
            mbar_inval(&sBar);
        }
    }
    return true;
}

template <int N, int CPB, bool GEN>
__global__ void __launch_bounds__(stage_threads(N, CPB), (stage_min_blocks<N, CPB>()))
    stage_kernel(const StageArgs a, const Ops ops)
{
    stage_tile<N, CPB, GEN>(a, ops, blockIdx.x);
}

// a batch's stage as a persistent launch: each CTA walks the tile table with a
// grid stride
template <int N, int CPB>
__global__ void __launch_bounds__(stage_threads(N, CPB), (stage_min_blocks<N, CPB>()))
    stage_kernel_persistent(const StageArgs a, const Ops ops)
{
    for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
        if (!stage_tile<N, CPB, true>(a, ops, t)) return;
        fence_proxy_async();  // what this thread wrote, before the next tile's copies
        __syncthreads();      // tile t's last shared-memory reads before tile t + grid stages
    }
}

}  // namespace sddc
