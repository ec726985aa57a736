// x-y pass tables of the two-kernel 3-D forward with 96-row tiles (f32 and i16
// inputs, radii 1 .. 8): images whose height 128-row tiles would pad more.
#include "two_pass.cuh"

namespace itkg {
namespace twopass {
namespace {
#define ITKG_XY96_TABLE(T, DT)                                                                          \
  {                                                                                                    \
    make_xy<1, T, 96>(DT), make_xy<2, T, 96>(DT), make_xy<3, T, 96>(DT), make_xy<4, T, 96>(DT),         \
        make_xy<5, T, 96>(DT), make_xy<6, T, 96>(DT), make_xy<7, T, 96>(DT), make_xy<8, T, 96>(DT)      \
  }
const XYEntry kF32[] = ITKG_XY96_TABLE(float, ITKG_F32);
const XYEntry kI16[] = ITKG_XY96_TABLE(int16_t, ITKG_I16);
}  // namespace
const XYEntry* xy96_f32() { return kF32; }
const XYEntry* xy96_i16() { return kI16; }
}  // namespace twopass
}  // namespace itkg
