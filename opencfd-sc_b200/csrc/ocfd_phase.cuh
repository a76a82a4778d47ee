// ocfd_phase.cuh -- the three face sweeps and the viscous gradients of one RK
// stage in one launch (single instance, axis-aligned periodic grids).
//
// The four are independent of one another: all read the primitives and the
// metrics, each writes its own array.  A small grid's stage is bound by launch gaps
// and by SMs without a block; one launch has one gap and one last wave instead of
// four (WENO7 32^3 mixed 0.064 -> 0.046 ms per step; the line is in ocfd_api.cu).
#pragma once

#include "ocfd_face.cuh"
#include "ocfd_update_body.cuh"

namespace ocfd {

template <typename R>
struct PhaseArgs {
  FaceArgs<R> f[3];
  ViscArgs<R, R> v;
};
struct PhaseMaps {
  FaceTmaMaps d[3];
};

// Block ranges of the four roles in launch order: x, y, z sweep, viscous
// gradients.  (Alternating the roles block by block was measured and is far slower
// for the large bodies: characteristic OMP6 at 256^3 27.5 against 14.3 ms a step,
// the SMs then hold the code of all four at once.)
template <bool CHAR, int SCHEME, typename R, bool TMA>
struct PhaseShape {
  using X = FaceTile<0, CHAR, SCHEME, R, true>;
  using Y = FaceTile<1, CHAR, SCHEME, R, true>;
  using Z = FaceTile<2, CHAR, SCHEME, R, true>;
  static constexpr int NT = X::NT, ROWS = NT / 32, FPT = X::FPT;
  static_assert(Y::NT == NT && Z::NT == NT, "one block size for all roles");
  template <int D>
  static constexpr size_t smem_of() {
    using F = FaceTile<D, CHAR, SCHEME, R, true>;
    return TMA ? FaceTmaSmem<D, CHAR, SCHEME, F::NP, F::TF, R, R, true, F::FPT, true>::BYTES
               : face_smem<D, CHAR, SCHEME, F::NP, F::TF, R, true, F::FPT>();
  }
  static constexpr size_t smem() {
    size_t m = smem_of<0>();
    m = smem_of<1>() > m ? smem_of<1>() : m;
    return smem_of<2>() > m ? smem_of<2>() : m;
  }
  // grid of role D (the sweeps' own launch grids; 3: viscous gradients)
  template <int D>
  static __host__ __device__ int3 grid(const Grid& g) {
    auto up = [](int a, int b) { return (a + b - 1) / b; };
    if (D == 0) return make_int3(up(g.nx, X::TF), up(g.ny, X::NP), g.nz);
    if (D == 1) return make_int3(up(g.nx, Y::NP), up(g.ny, Y::TF), g.nz);
    if (D == 2) return make_int3(up(g.nx, Z::NP), up(g.nz, Z::TF), g.ny);
    return make_int3(up(g.nx, 32), up(g.ny, ROWS), g.nz);
  }
};

template <bool CHAR, int SCHEME, typename R, bool TMA>
__global__ void __launch_bounds__(PhaseShape<CHAR, SCHEME, R, TMA>::NT,
                                  PhaseShape<CHAR, SCHEME, R, TMA>::FPT > 1 ? OCFD_FACE64_MINBPAIR
                                  : PhaseShape<CHAR, SCHEME, R, TMA>::NT == 128 && sizeof(R) == 8
                                      ? OCFD_FACE64_MINB128_AX
                                      : OCFD_FACE_MINB * 256 / PhaseShape<CHAR, SCHEME, R, TMA>::NT)
    k_phase(const __grid_constant__ PhaseArgs<R> a, const __grid_constant__ PhaseMaps tm) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using P = PhaseShape<CHAR, SCHEME, R, TMA>;
  const Grid& G = a.v.g;
  int lin = blockIdx.x;
  int3 d = P::template grid<0>(G);
  int n = d.x * d.y * d.z, role = 0;
  if (lin >= n) {
    lin -= n;
    d = P::template grid<1>(G);
    n = d.x * d.y * d.z;
    role = 1;
    if (lin >= n) {
      lin -= n;
      d = P::template grid<2>(G);
      n = d.x * d.y * d.z;
      role = 2;
      if (lin >= n) {
        lin -= n;
        d = P::template grid<3>(G);
        role = 3;
      }
    }
  }
  const int bx = lin % d.x, t = lin / d.x, by = t % d.y, bz = t / d.y;
  R* const sm = reinterpret_cast<R*>(smem_raw);
  if (role == 0) {
    if constexpr (TMA)
      face_tma_block<0, CHAR, SCHEME, R, R, true, true>(a.f[0], tm.d[0], bx, by, bz, smem_raw);
    else
      face_body<0, CHAR, SCHEME, true, P::X::NP, P::X::TF, R, R, false, true, P::X::FPT>(a.f[0], bx, by, bz, sm);
  } else if (role == 1) {
    if constexpr (TMA)
      face_tma_block<1, CHAR, SCHEME, R, R, true, true>(a.f[1], tm.d[1], bx, by, bz, smem_raw);
    else
      face_body<1, CHAR, SCHEME, true, P::Y::NP, P::Y::TF, R, R, false, true, P::Y::FPT>(a.f[1], bx, by, bz, sm);
  } else if (role == 2) {
    if constexpr (TMA)
      face_tma_block<2, CHAR, SCHEME, R, R, true, true>(a.f[2], tm.d[2], bx, by, bz, smem_raw);
    else
      face_body<2, CHAR, SCHEME, true, P::Z::NP, P::Z::TF, R, R, false, true, P::Z::FPT>(a.f[2], bx, by, bz, sm);
  } else {
    visc_grad_body<R, R, true, P::ROWS>(a.v, bx, by, bz);
  }
}

template <bool CHAR, int SCHEME, typename R, bool TMA>
static cudaError_t launch_phase_t(const PhaseArgs<R>& a, cudaStream_t st) {
  using P = PhaseShape<CHAR, SCHEME, R, TMA>;
  constexpr size_t smem = P::smem();
  auto kern = k_phase<CHAR, SCHEME, R, TMA>;
  const Grid& g = a.v.g;
  if (g.n == 0) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  PhaseMaps tm;
  if constexpr (TMA) {
    if (!face_tma_maps<TmaBox<0, P::X::NP, P::X::TF, R, P::X::FPT>>(a.f[0], tm.d[0]) ||
        !face_tma_maps<TmaBox<1, P::Y::NP, P::Y::TF, R, P::Y::FPT>>(a.f[1], tm.d[1]) ||
        !face_tma_maps<TmaBox<2, P::Z::NP, P::Z::TF, R, P::Z::FPT>>(a.f[2], tm.d[2]))
      return cudaErrorInvalidValue;
  } else {
    memset(&tm, 0, sizeof(tm));
  }
  auto blocks = [](int3 d) { return (long long)d.x * d.y * d.z; };
  const long long n = blocks(P::template grid<0>(g)) + blocks(P::template grid<1>(g)) +
                      blocks(P::template grid<2>(g)) + blocks(P::template grid<3>(g));
  if (n > 2147483647LL) return cudaErrorInvalidValue;
  kern<<<(unsigned)n, P::NT, smem, st>>>(a, tm);
  return cudaGetLastError();
}

template <bool CHAR, int SCHEME, typename R>
static cudaError_t launch_phase_cs(const PhaseArgs<R>& a, cudaStream_t st) {
  if (a.v.g.n == 0) {
    cudaError_t e = launch_phase_t<CHAR, SCHEME, R, false>(a, st);
    if (sizeof(R) == 8 && e == cudaSuccess) e = launch_phase_t<CHAR, SCHEME, R, sizeof(R) == 8>(a, st);
    return e;
  }
  if (sizeof(R) == 8 && !a.f[0].no_tma && face_tma_enabled() && tma_strides_ok<R>(a.v.g))
    return launch_phase_t<CHAR, SCHEME, R, sizeof(R) == 8>(a, st);
  return launch_phase_t<CHAR, SCHEME, R, false>(a, st);
}

// (the strict build runs the sweeps one by one)
template <typename R>
cudaError_t launch_phase(bool chr, int scheme, const FaceArgs<R> f[3], const ViscArgs<R, R>& v, cudaStream_t st) {
  PhaseArgs<R> a;
  for (int d = 0; d < 3; d++) a.f[d] = f[d];
  a.v = v;
#if OCFD_FEWER_DIVS
#define OCFD_PHASE(C, SC) \
  if (chr == C && scheme == SC) return launch_phase_cs<C, SC, R>(a, st);
  OCFD_PHASE(false, SCH_WENO5)
  OCFD_PHASE(false, SCH_WENO7)
  OCFD_PHASE(false, SCH_OMP6)
  OCFD_PHASE(false, SCH_UD7L)
  OCFD_PHASE(false, SCH_HYBRID)
  OCFD_PHASE(true, SCH_WENO5)
  OCFD_PHASE(true, SCH_WENO7)
  OCFD_PHASE(true, SCH_OMP6)
  OCFD_PHASE(true, SCH_UD7L)
  OCFD_PHASE(true, SCH_HYBRID)
#undef OCFD_PHASE
#endif
  return cudaErrorInvalidValue;
}

// shared-memory limits of every kernel of one precision (call outside graph capture)
template <typename R>
static cudaError_t setup_phase() {
  const int schemes[5] = {SCH_WENO5, SCH_WENO7, SCH_OMP6, SCH_UD7L, SCH_HYBRID};
  FaceArgs<R> f[3];
  ViscArgs<R, R> v;
  memset(f, 0, sizeof(f));
  memset(&v, 0, sizeof(v));
  for (int c = 0; c < 2 && OCFD_FEWER_DIVS; c++)
    for (int s = 0; s < 5; s++) {
      cudaError_t e = launch_phase<R>(c == 1, schemes[s], f, v, 0);
      if (e != cudaSuccess) return e;
    }
  return cudaSuccess;
}

}  // namespace ocfd
