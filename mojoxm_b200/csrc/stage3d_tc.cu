// Shape queries of the tensor-core 3D stage.
#include "stage3d_tc.cuh"

namespace mxm {

int tc_tile_cubes(int P, int NC, int kind) {
  auto ec = [&](auto op) -> int {
    using O = decltype(op);
    switch (NC) {
      case 1: return P == 2 ? TcShape<2, 1, O>::EC : P == 3 ? TcShape<3, 1, O>::EC : P == 4 ? TcShape<4, 1, O>::EC : TcShape<5, 1, O>::EC;
      case 3: return P == 2 ? TcShape<2, 3, O>::EC : P == 3 ? TcShape<3, 3, O>::EC : P == 4 ? TcShape<4, 3, O>::EC : TcShape<5, 3, O>::EC;
      case 5: return P == 2 ? TcShape<2, 5, O>::EC : P == 3 ? TcShape<3, 5, O>::EC : P == 4 ? TcShape<4, 5, O>::EC : TcShape<5, 5, O>::EC;
      case 6: return P == 2 ? TcShape<2, 6, O>::EC : P == 3 ? TcShape<3, 6, O>::EC : P == 4 ? TcShape<4, 6, O>::EC : TcShape<5, 6, O>::EC;
      case 9: return P == 2 ? TcShape<2, 9, O>::EC : P == 3 ? TcShape<3, 9, O>::EC : P == 4 ? TcShape<4, 9, O>::EC : TcShape<5, 9, O>::EC;
    }
    return 0;
  };
  return kind == TC_TF32 ? ec(OpTF32{}) : ec(OpBF16{});
}

bool tc_shape_fits(int P, int NC, int kind) {
  auto fits = [&](auto op) -> bool {
    using O = decltype(op);
    switch (NC) {
      case 1: return P == 2 ? TcShape<2, 1, O>::FITS : P == 3 ? TcShape<3, 1, O>::FITS : P == 4 ? TcShape<4, 1, O>::FITS : TcShape<5, 1, O>::FITS;
      case 3: return P == 2 ? TcShape<2, 3, O>::FITS : P == 3 ? TcShape<3, 3, O>::FITS : P == 4 ? TcShape<4, 3, O>::FITS : TcShape<5, 3, O>::FITS;
      case 5: return P == 2 ? TcShape<2, 5, O>::FITS : P == 3 ? TcShape<3, 5, O>::FITS : P == 4 ? TcShape<4, 5, O>::FITS : TcShape<5, 5, O>::FITS;
      case 6: return P == 2 ? TcShape<2, 6, O>::FITS : P == 3 ? TcShape<3, 6, O>::FITS : P == 4 ? TcShape<4, 6, O>::FITS : TcShape<5, 6, O>::FITS;
      case 9: return P == 2 ? TcShape<2, 9, O>::FITS : P == 3 ? TcShape<3, 9, O>::FITS : P == 4 ? TcShape<4, 9, O>::FITS : TcShape<5, 9, O>::FITS;
    }
    return false;
  };
  if (P < 2 || P > 5) return false;
  return kind == TC_TF32 ? fits(OpTF32{}) : fits(OpBF16{});
}

}  // namespace mxm
