// pencil_inst.cu — the pencil sweeps of one species count (FLAME_PENCIL_NS, set by the build).
#include "pencil_kernels.cuh"

#ifndef FLAME_PENCIL_NS
#error "compile with -DFLAME_PENCIL_NS=1..9"
#endif

namespace flame {
namespace pencil {

template <>
const PencilOps &pencil_ops<FLAME_PENCIL_NS>() {
    constexpr int N = FLAME_PENCIL_NS;
    static const PencilOps ops = {
        {launch<N, double>, launch<N, float>},
        {batch_dims<N, double, double>, batch_dims<N, float, float>},
        {batch_grid<N, double, double>, batch_grid<N, float, float>},
        {batch_launch<N, double, double>, batch_launch<N, float, float>}};
    return ops;
}

}  // namespace pencil
}  // namespace flame
