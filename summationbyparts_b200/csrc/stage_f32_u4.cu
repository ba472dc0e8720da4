// Instantiations of the fused stage kernel: Upwind4/Upwind4h2 operator pairs, compensated f32 state.
#include "stage_dispatch.h"
#include "stage_kernel.cuh"
#include "stage_kernel_vec.cuh"

namespace sbp {

// 16-row tiles: stage_kernel; 32-row tiles: the 2 x 2 micro-tile kernel (stage_kernel_vec).
#define CASE(OX, OY, UPW, TYV)                                                        \
    if (opx == OX && opy == OY && upw == UPW && ty == 16 && TYV == 16)                \
        return reinterpret_cast<const void*>(&stage_kernel<OX, OY, float, UPW, true, 16, false>); \
    if (opx == OX && opy == OY && upw == UPW && ty == kVecRows && TYV == kVecRows)    \
        return vec_entry<OX, OY, UPW>(sc);

// the fused form
#define FUSED(OX, OY, UPW)                                                                                          \
    if (opx == OX && opy == OY && upw == UPW && ty == (8 | kTileFused))                                             \
        return reinterpret_cast<const void*>(&stage_kernel<OX, OY, float, UPW, true, 8, true>);                   \
    if (opx == OX && opy == OY && upw == UPW && ty == (16 | kTileFused))                                            \
        return reinterpret_cast<const void*>(&stage_kernel<OX, OY, float, UPW, true, 16, true>);

const void* stage_ptr_f32_u4(int opx, int opy, bool upw, int ty, int sc) {
    CASE(UPWIND4, UPWIND4, true, 16)
    FUSED(UPWIND4, UPWIND4, true)
    CASE(UPWIND4, UPWIND4, true, 32)
    CASE(UPWIND4, UPWIND4, false, 16)
    FUSED(UPWIND4, UPWIND4, false)
    CASE(UPWIND4, UPWIND4, false, 32)
    CASE(UPWIND4H2, UPWIND4H2, true, 16)
    FUSED(UPWIND4H2, UPWIND4H2, true)
    CASE(UPWIND4H2, UPWIND4H2, true, 32)
    CASE(UPWIND4H2, UPWIND4H2, false, 16)
    FUSED(UPWIND4H2, UPWIND4H2, false)
    CASE(UPWIND4H2, UPWIND4H2, false, 32)
    CASE(UPWIND4, UPWIND4H2, true, 16)
    FUSED(UPWIND4, UPWIND4H2, true)
    CASE(UPWIND4, UPWIND4H2, true, 32)
    CASE(UPWIND4, UPWIND4H2, false, 16)
    FUSED(UPWIND4, UPWIND4H2, false)
    CASE(UPWIND4, UPWIND4H2, false, 32)
    CASE(UPWIND4H2, UPWIND4, true, 16)
    FUSED(UPWIND4H2, UPWIND4, true)
    CASE(UPWIND4H2, UPWIND4, true, 32)
    CASE(UPWIND4H2, UPWIND4, false, 16)
    FUSED(UPWIND4H2, UPWIND4, false)
    CASE(UPWIND4H2, UPWIND4, false, 32)
    return nullptr;
}

}  // namespace sbp
