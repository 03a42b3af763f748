// zm_axis_c64_inv.cu -- tile shapes of the axis pass sized by N alone, c64, inverse.
#include "zm_axis.cuh"
#include "zm_axis_tiles.h"

namespace zm {

cudaError_t launch_axis_c64_inv(const AxisParams &p, int64_t nlines, cudaStream_t st) {
    switch (p.g.logN << 16 | p.m.ltl << 8 | p.m.lp << 4 | p.m.le) {
#define ZM_CASE(LN, LTL, LP, LE) \
    case LN << 16 | LTL << 8 | LP << 4 | LE: return launch_axis<float, LN, LTL, LP, LE, true>(p, nlines, st);
        ZM_AXIS_TILES_C64(ZM_CASE)
#undef ZM_CASE
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace zm
