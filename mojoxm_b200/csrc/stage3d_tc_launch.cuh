// Launch configuration of the tensor-core 3D stage (split-BF16 or split-TF32
// operands) for P = 2..5 where the shape fits shared memory; P = 1 uses the
// FP32 SIMT kernel.  Included by the per-physics units.
#pragma once
#include <type_traits>

#include "stage3d_tc.cuh"

namespace mxm {

// Threads per block.  A warp of this kernel wants up to 168 registers, and a
// scheduler's 16 K registers hold three such warps, so the SM holds 12 warps
// however they are split into blocks: four warps each where shared memory
// holds several blocks (Euler/Rusanov P3, 32^3: 155 us a stage; 256 threads
// at 80 registers spill, 295 us), all of them in one block where it holds
// one, as far as the phases have works for them: split-TF32 P4 (210 to 540
// element-pair works per phase) is best at 224 threads (209 us Euler, 311 to
// 325 us Maxwell, against 230 and 333 at 384), split-BF16 P5 (336 to 756) at
// 384 (HLLEC 155 us at 20^3; 161 at 256).
template <class Phys, int P, class Op>
__host__ __device__ constexpr int tc_threads() {
  using S = TcShape<P, Phys::NC, Op>;
  return S::blocks_for(S::SMEM) >= 2 ? 128 : (P >= 5 ? 384 : 224);
}

// Blocks per SM the register allocation must allow: what fits in shared
// memory, at most four (128 registers) for light fluxes of up to six
// components and three (168) for the others (P2, 32^3: Rusanov 96 us with
// four and 106 with three, MHD 136 and 126).
template <class Phys, int P, class Op>
__host__ __device__ constexpr int tc_min_blocks() {
  using S = TcShape<P, Phys::NC, Op>;
  constexpr int fit = int(S::blocks_for(S::SMEM)), cap = Phys::kLightFlux && Phys::NC <= 6 ? 4 : 3;
  return fit < cap ? fit : cap;
}

// Launch shape of one instantiation.  Batched launches keep the current
// solve's arguments behind the tile's shared memory.
template <class Phys, int P, class Op, bool BATCH>
struct TcLaunch {
  using S = TcShape<P, Phys::NC, Op>;
  static constexpr int NT = tc_threads<Phys, P, Op>();
  static constexpr int MINB = tc_min_blocks<Phys, P, Op>();
  static constexpr size_t smem = BATCH ? S::BATCH_SMEM : S::SMEM;
  static cudaError_t blocks_per_sm(int* out) {
    static int bps = -1;
    if (bps < 0) {
      cudaError_t e = persistent_blocks_per_sm((const void*)stage3d_tc_kernel<Phys, P, NT, MINB, Op, BATCH>, NT, smem, &bps);
      if (e != cudaSuccess) return e;
    }
    *out = bps;
    return cudaSuccess;
  }
  // persistent grid: every resident block, at most one per tile
  static cudaError_t grid(int nsm, int ntiles, int* out) {
    int bps = 0;
    cudaError_t e = blocks_per_sm(&bps);
    if (e != cudaSuccess) return e;
    int nblk = nsm * bps;
    if (nblk > ntiles) nblk = ntiles;
    *out = nblk < 1 ? 1 : nblk;
    return cudaSuccess;
  }
};

template <class Phys, int P, class Op, bool BATCH>
cudaError_t launch_tc_p(const Stage3DArgs<float>& a, const Tc3Batch& bat, const Phys& ph, const unsigned char* img, int nsm, cudaStream_t st) {
  using S = TcShape<P, Phys::NC, Op>;
  if constexpr (!S::FITS) {
    return cudaErrorInvalidValue;  // the create call refuses these shapes
  } else {
    using L = TcLaunch<Phys, P, Op, BATCH>;
    static_assert(sizeof(Stage3DArgs<float>) <= 256, "batched arguments slot");
    const int ntiles = BATCH ? bat.nitems : (a.ncell - a.cbeg + S::EC - 1) / S::EC;
    if (ntiles <= 0) return cudaSuccess;
    int nblk = 1;
    cudaError_t e = L::grid(nsm, ntiles, &nblk);
    if (e != cudaSuccess) return e;
    auto kern = stage3d_tc_kernel<Phys, P, L::NT, L::MINB, Op, BATCH>;
    if constexpr (BATCH) {
      kern<<<nblk, L::NT, L::smem, st>>>(a, ph, img, bat);
      return cudaGetLastError();
    } else {
      return launch_dependent(kern, nblk, L::NT, L::smem, st, a, ph, img, bat);
    }
  }
}

template <class Phys, class Op>
cudaError_t batch_grid_kind(int P, int nsm, int ntiles, int* out) {
  auto one = [&](auto pc) -> cudaError_t {
    constexpr int PP = decltype(pc)::value;
    if constexpr (!TcShape<PP, Phys::NC, Op>::FITS) return cudaErrorInvalidValue;
    else return TcLaunch<Phys, PP, Op, true>::grid(nsm, ntiles, out);
  };
  switch (P) {
    case 2: return one(std::integral_constant<int, 2>{});
    case 3: return one(std::integral_constant<int, 3>{});
    case 4: return one(std::integral_constant<int, 4>{});
    case 5: return one(std::integral_constant<int, 5>{});
  }
  return cudaErrorInvalidValue;
}

// Blocks a batched launch of `ntiles` tiles runs (the same rule as the launch).
template <class Phys>
cudaError_t stage3d_tc_batch_grid(int P, int kind, const Phys&, int nsm, int ntiles, int* out) {
  return kind == TC_TF32 ? batch_grid_kind<Phys, OpTF32>(P, nsm, ntiles, out)
                         : batch_grid_kind<Phys, OpBF16>(P, nsm, ntiles, out);
}

template <class Phys, class Op, bool BATCH>
cudaError_t launch_tc_kind(int P, const Stage3DArgs<float>& a, const Tc3Batch& bat, const Phys& ph, const unsigned char* img, int nsm, cudaStream_t st) {
  switch (P) {
    case 2: return launch_tc_p<Phys, 2, Op, BATCH>(a, bat, ph, img, nsm, st);
    case 3: return launch_tc_p<Phys, 3, Op, BATCH>(a, bat, ph, img, nsm, st);
    case 4: return launch_tc_p<Phys, 4, Op, BATCH>(a, bat, ph, img, nsm, st);
    case 5: return launch_tc_p<Phys, 5, Op, BATCH>(a, bat, ph, img, nsm, st);
  }
  return cudaErrorInvalidValue;
}

template <class Phys>
cudaError_t launch_stage3d_tc(int P, int kind, const Stage3DArgs<float>& a, const Phys& ph, const unsigned char* img,
                              int nsm, cudaStream_t st) {
  const Tc3Batch none{nullptr, nullptr, 0};
  return kind == TC_TF32 ? launch_tc_kind<Phys, OpTF32, false>(P, a, none, ph, img, nsm, st)
                         : launch_tc_kind<Phys, OpBF16, false>(P, a, none, ph, img, nsm, st);
}

template <class Phys>
cudaError_t launch_stage3d_tc_batch(int P, int kind, const Tc3Batch& bat, const Phys& ph, const unsigned char* img,
                                    int nsm, cudaStream_t st) {
  static const Stage3DArgs<float> a0{};
  return kind == TC_TF32 ? launch_tc_kind<Phys, OpTF32, true>(P, a0, bat, ph, img, nsm, st)
                         : launch_tc_kind<Phys, OpBF16, true>(P, a0, bat, ph, img, nsm, st);
}

#define MXM_INST_TC(PH)                                                                                        \
  template cudaError_t launch_stage3d_tc<PH>(int, int, const Stage3DArgs<float>&, const PH&,                   \
                                             const unsigned char*, int, cudaStream_t);                         \
  template cudaError_t launch_stage3d_tc_batch<PH>(int, int, const Tc3Batch&, const PH&, const unsigned char*, \
                                                   int, cudaStream_t);                                         \
  template cudaError_t stage3d_tc_batch_grid<PH>(int, int, const PH&, int, int, int*);

}  // namespace mxm
