// The exact form's RK stage by tiles: the reference's
// operations in its order, compiled with -fmad=false (no FMA contraction).
#include <algorithm>

#include "per_device.h"
#include "stage_kernel.cuh"

namespace sddc {

namespace {

template <int N, int CPB> struct TileLaunch {
    using Kern = void (*)(const StageArgs, const Ops);
    static constexpr size_t kSmem = stage_smem_bytes<N, CPB>();
    static constexpr int kThreads = stage_threads(N, CPB);

    // the kernels of a plain case, of batches and packed metrics, and of a
    // persistent batch
    static Kern kernel(int w)
    {
        static const Kern kerns[3] = {stage_kernel<N, CPB, false>, stage_kernel<N, CPB, true>,
                                      stage_kernel_persistent<N, CPB>};
        return kerns[w];
    }
    // CTAs of kernel w resident at once (its attributes are set on the way)
    static cudaError_t residency(int w, int *out)
    {
        static PerDevice resident[3];
        return resident[w].get(out, [&](int dev, int *n) { return resident_ctas(kernel(w), kThreads, kSmem, dev, n); });
    }
    static cudaError_t run(const StageArgs &a, const Ops &ops, cudaStream_t st)
    {
        const int w = a.tiles && a.persistent ? 2 : a.tiles || !a.nrm ? 1 : 0;
        int resident = 0;
        const cudaError_t e = residency(w, &resident);
        if (e != cudaSuccess) return e;
        const int tiles = a.tiles ? a.ntiles : (a.ncell + CPB - 1) / CPB;
        kernel(w)<<<w == 2 ? std::min(tiles, resident) : tiles, kThreads, kSmem, st>>>(a, ops);
        return cudaGetLastError();
    }
};

}  // namespace

cudaError_t launch_tile_exact(int N, int cpb, const StageArgs &a, const Ops &ops, cudaStream_t st)
{
    switch (N) {
    case 2: return TileLaunch<2, 8>::run(a, ops, st);
    case 3: return TileLaunch<3, 4>::run(a, ops, st);
    case 4: return TileLaunch<4, 8>::run(a, ops, st);
    case 5: return TileLaunch<5, 6>::run(a, ops, st);
    case 6: return cpb == 6 ? TileLaunch<6, 6>::run(a, ops, st) : TileLaunch<6, 8>::run(a, ops, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace sddc
