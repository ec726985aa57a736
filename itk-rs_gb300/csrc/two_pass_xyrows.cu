// x-y pass tables of the two-kernel 3-D forward with 96- and 64-row tiles (f32
// and i16 inputs, radii 1 .. 8): images whose height 128-row tiles would pad more.
#include "two_pass.cuh"

namespace itkg {
namespace twopass {
namespace {
#define ITKG_XY_ROWS_TABLE(T, DT, TY)                                                                   \
  {                                                                                                    \
    make_xy<1, T, TY>(DT), make_xy<2, T, TY>(DT), make_xy<3, T, TY>(DT), make_xy<4, T, TY>(DT),         \
        make_xy<5, T, TY>(DT), make_xy<6, T, TY>(DT), make_xy<7, T, TY>(DT), make_xy<8, T, TY>(DT)      \
  }
const XYEntry kF32[2][8] = {ITKG_XY_ROWS_TABLE(float, ITKG_F32, 96), ITKG_XY_ROWS_TABLE(float, ITKG_F32, 64)};
const XYEntry kI16[2][8] = {ITKG_XY_ROWS_TABLE(int16_t, ITKG_I16, 96), ITKG_XY_ROWS_TABLE(int16_t, ITKG_I16, 64)};
}  // namespace
const XYEntry* xy_rows_f32(int rows) { return kF32[rows == 64]; }
const XYEntry* xy_rows_i16(int rows) { return kI16[rows == 64]; }
}  // namespace twopass
}  // namespace itkg
