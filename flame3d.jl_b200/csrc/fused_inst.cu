// fused_inst.cu — the tile kernels of one species count (FLAME_FUSED_NS, set by the build).
#include "fused_kernels.cuh"

#ifndef FLAME_FUSED_NS
#error "compile with -DFLAME_FUSED_NS=1..9"
#endif

namespace flame {
namespace fused {

FLAME_FUSED_LAUNCHES(, FLAME_FUSED_NS)

}  // namespace fused
}  // namespace flame
