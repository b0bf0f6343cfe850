// The exact form's RK stage by tiles: the reference's
// operations in its order, compiled with -fmad=false (no FMA contraction).
#include <algorithm>

#include "per_device.h"
#include "stage_kernel.cuh"

namespace sddc {

namespace {

template <int N, int CPB> cudaError_t launch_n(const StageArgs &a, const Ops &ops, cudaStream_t st)
{
    auto kern = stage_kernel<N, CPB>;
    constexpr size_t smem = stage_smem_bytes<N, CPB>();
    static PerDevice configured;  // per instantiation
    int set = 0;
    const cudaError_t e = configured.get(&set, [&](int, int *out) {
        *out = 1;
        return set_smem(kern, smem);
    });
    if (e != cudaSuccess) return e;
    kern<<<(a.ncell + CPB - 1) / CPB, stage_threads(N, CPB), smem, st>>>(a, ops);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_tile_exact(int N, int cpb, const StageArgs &a, const Ops &ops, cudaStream_t st)
{
    switch (N) {
    case 2: return launch_n<2, 8>(a, ops, st);
    case 3: return launch_n<3, 4>(a, ops, st);
    case 4: return launch_n<4, 8>(a, ops, st);
    case 5: return launch_n<5, 6>(a, ops, st);
    case 6: return cpb == 6 ? launch_n<6, 6>(a, ops, st) : launch_n<6, 8>(a, ops, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace sddc
