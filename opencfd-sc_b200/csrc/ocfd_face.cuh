// ocfd_face.cuh -- face-flux kernels of the inviscous terms, one launch per
// direction: split -> (characteristic projection) -> reconstruction, written
// as numerical fluxes h(i+1/2) per face.  The flux difference, the Jacobian
// scaling and the rest of the stage happen in the update kernel
// (ocfd_update.cu), which reads these faces.
//
// Reference: du_inviscous (OCFD_inviscous.f90:53-203) with OCFD2d_flux1/2
// (:210-361) for the flux-vector form, du_inviscous_Character
// (OCFD_inviscous_character.f90:3-159) with flux_charteric / flux_x1 / flux_x2
// (:162-416) for the characteristic form.
//
// Tiling: a block owns NP pencils x TF consecutive faces along the sweep
// direction (128 or 256 faces, one or two per thread).  Phase 1 loads the
// TF+7 points of its stencil (coalesced along i for x, across i for y/z),
// computes the split fluxes once per point and stages them in shared memory.
// Phase 2 computes the faces from their windows of 8 points; the uncommon ones
// (hybrid WENO, OMP6 limiter, boundary closure) go through lists of the block.
// For a periodic direction face 0 equals face n bit for bit, so only faces
// 1..n are computed: n faces for n points, no tile does extra work.
#pragma once
#include <cstring>

#include "ocfd_device.cuh"
#include "ocfd_kernels.h"
#include "ocfd_schemes.cuh"
#include "ocfd_tma.cuh"

namespace ocfd {

// Tile shapes (NP pencils x TF faces, one face per thread).  Variants 0 and 1
// (256 threads) are the choices of the batch autotuner -- variant 1 (TF = 32)
// wastes fewer threads on short pencils.  Variant 2 (128 threads) is the
// single-instance tile of the characteristic OMP6 and the hybrid sweeps: at 256^3
// it measured 5-9% faster with OMP6 than variant 0 (four blocks per SM overlap one
// another's barrier and load phases better than two), but slower on the WENO7
// sweeps, which keep variant 0.  (Tiles of 64 threads, or of 128 with TF = 32 along y and
// z, measured slower.)
template <int DIR, int V>
struct FaceTileV;
template <>
struct FaceTileV<0, 0> {
  static constexpr int NP = 4, TF = 64;
};
template <>
struct FaceTileV<0, 1> {
  static constexpr int NP = 8, TF = 32;
};
template <>
struct FaceTileV<1, 0> {
  static constexpr int NP = 16, TF = 16;
};
template <>
struct FaceTileV<1, 1> {
  static constexpr int NP = 8, TF = 32;
};
template <>
struct FaceTileV<2, 0> {
  static constexpr int NP = 16, TF = 16;
};
template <>
struct FaceTileV<2, 1> {
  static constexpr int NP = 8, TF = 32;
};
// 128-thread tiles (more, smaller blocks per SM)
template <>
struct FaceTileV<0, 2> {
  static constexpr int NP = 2, TF = 64;
};
template <>
struct FaceTileV<1, 2> {
  static constexpr int NP = 8, TF = 16;
};
template <>
struct FaceTileV<2, 2> {
  static constexpr int NP = 8, TF = 16;
};
// Tile of a single-instance sweep: NP pencils x TF faces, NT threads, each FPT
// consecutive faces.  Two faces a thread: the FP64 hybrid sweeps of periodic
// directions.  Their common face is the linear scheme, 80 multiply-adds on 80 values
// read from shared memory, and two neighbouring faces share seven of their eight
// points; the longer tile also recomputes 7 halo points for 32 faces instead of 16
// (isotropic turbulence 320^3, LLF: the three sweeps 11.4 -> 9.2 ms per step).  The
// characteristic OMP6 sweeps, with five times the arithmetic per value read, lost
// more to the halved number of threads (a step at 256^3 14.12 -> 14.31 ms).
template <int DIR, bool CHAR, int SCHEME, typename R, bool ALLIN>
struct FaceTile {
  static constexpr bool HYB = OCFD_FEWER_DIVS && SCHEME == SCH_HYBRID;
  static constexpr int FPT = (HYB && ALLIN && sizeof(R) == 8) ? 2 : 1;
  using V = FaceTileV<DIR, ((CHAR && SCHEME == SCH_OMP6) || HYB) ? 2 : 0>;
  static constexpr int NP = FPT > 1 ? 8 : V::NP, TF = FPT > 1 ? 32 : V::TF, NT = NP * TF / FPT;
};

// Grid of one launch: (x, y, z) blocks for a face sweep of instance a.
template <int DIR, int NP, int TF, typename S>
__host__ __forceinline__ dim3 face_grid(const FaceArgs<S>& a) {
  const int nf = a.fend - a.fbeg + 1;
  if (DIR == 0) return dim3((nf + TF - 1) / TF, (a.g.ny + NP - 1) / NP, a.g.nz);
  return dim3((a.g.nx + NP - 1) / NP, (nf + TF - 1) / TF, DIR == 1 ? a.g.nz : a.g.ny);
}

// ---------------------------------------------------------------------------
// Flux-vector form, boundary-aware reconstruction of one face (OCFD2d_flux1).
template <int SCHEME, typename R>
__device__ __forceinline__ R nc_flux1_bnd(const R* v, const R* U, int g, int nn, int ihy, const Phys& ph, int dir) {
  const int bi0 = ph.bi[2 * dir], bi1 = ph.bi[2 * dir + 1], sb0 = ph.sb[2 * dir], sb1 = ph.sb[2 * dir + 1];
  const int Ka = ph.ka1, Kb = ph.kb1;
  const int ib = (bi0 == 0 || sb0 == -1) ? 0 : -Ka + 1;
  const int ie = (bi1 == 0 || sb1 == -1) ? nn : nn - Kb;
  R h = R(0);
  if (g >= ib && g <= ie) h = schemeP<SCHEME>(v, U, ihy);
  if (bi0 == 1 && g <= -Ka) {
    if (sb0 == 0) {
      if (g == 0)
        h = (R(2) * v[1] + R(5) * v[2] - v[3]) / R(6);
      else if (g == 1)
        h = (R(2) * v[0] + R(5) * v[1] - v[2]) / R(6);
      else if (g == 2)
        h = weno5P_bnd(v, 1);
      else
        h = weno5P(v);
    } else if (sb0 == 1) {
      h = weno5P(v);
    }
  }
  if (bi1 == 1 && g >= nn - Kb + 1) {
    if (sb1 == 0) {
      if (g == nn)
        h = (R(2) * v[-2] - R(7) * v[-1] + R(11) * v[0]) / R(6);
      else if (g == nn - 1)
        h = weno5P_bnd(v, 2);
      else
        h = weno5P(v);
    } else if (sb1 == 1) {
      h = weno5P(v);
    }
  }
  return h;
}

// OCFD2d_flux2 (OCFD_inviscous.f90:287-361)
template <int SCHEME, typename R>
__device__ __forceinline__ R nc_flux2_bnd(const R* v, const R* U, int g, int nn, int ihy, const Phys& ph, int dir) {
  const int bi0 = ph.bi[2 * dir], bi1 = ph.bi[2 * dir + 1], sb0 = ph.sb[2 * dir], sb1 = ph.sb[2 * dir + 1];
  const int Ka = ph.ka2, Kb = ph.kb2;
  const int ib = (bi0 == 0 || sb0 == -1) ? 0 : -Ka + 1;
  const int ie = (bi1 == 0 || sb1 == -1) ? nn : nn - Kb;
  R h = R(0);
  if (g >= ib && g <= ie) h = schemeM<SCHEME>(v, U, ihy);
  if (bi0 == 1 && g <= -Ka) {
    if (sb0 == 0) {
      if (g == 0)
        h = (R(2) * v[3] - R(7) * v[2] + R(11) * v[1]) / R(6);
      else if (g == 1)
        h = weno5M_bnd(v, 1);
      else
        h = weno5M(v);
    } else if (sb0 == 1) {
      h = weno5M(v);
    }
  }
  if (bi1 == 1 && g >= nn - Kb + 1) {
    if (sb1 == 0) {
      if (g == nn)
        h = (R(2) * v[0] + R(5) * v[-1] - v[-2]) / R(6);
      else if (g == nn - 1)
        h = (R(2) * v[1] + R(5) * v[0] - v[-1]) / R(6);
      else if (g == nn - 2)
        h = weno5M_bnd(v, 2);
      else
        h = weno5M(v);
    } else if (sb1 == 1) {
      h = weno5M(v);
    }
  }
  return h;
}

// The boundary closures of one direction, by value (Bound_index, Scheme_boundary
// and the stencil ranges of the scheme).
struct FaceEnds {
  int bi0, bi1, sb0, sb1, ka1, kb1, ka2, kb2;
};
__device__ __forceinline__ FaceEnds face_ends(const Phys& ph, int dir) {
  return FaceEnds{ph.bi[2 * dir], ph.bi[2 * dir + 1], ph.sb[2 * dir], ph.sb[2 * dir + 1],
                  ph.ka1,         ph.kb1,             ph.ka2,         ph.kb2};
}

// Characteristic form: flux_x1 (OCFD_inviscous_character.f90:313-364) for a
// face that is not an interior face.
template <typename R>
__device__ __forceinline__ R ch_flux1_bnd(const R* ff, int g, int nn, const FaceEnds& fe) {
  const int bi0 = fe.bi0, bi1 = fe.bi1, sb0 = fe.sb0, sb1 = fe.sb1;
  const int Ka = fe.ka1, Kb = fe.kb1;
  if (g <= -Ka && bi0 == 1 && sb0 != -1) {
    if (sb0 == 0) {
      if (g == 1) return (R(2) * ff[0] + R(5) * ff[1] - ff[2]) / R(6);
      if (g == 2) return weno5P_bnd(ff, 1);
      return weno5P(ff);
    } else if (sb0 == 1) {
      return weno5P(ff);
    }
  } else if (g > nn - Kb && bi1 == 1 && sb1 != -1) {
    if (sb1 == 0) {
      if (g == nn - 1) return weno5P_bnd(ff, 2);
      return weno5P(ff);
    } else if (sb1 == 1) {
      return weno5P(ff);
    }
  }
  return R(0);
}

// flux_x2 (OCFD_inviscous_character.f90:367-416), non-interior face
template <typename R>
__device__ __forceinline__ R ch_flux2_bnd(const R* ff, int g, int nn, const FaceEnds& fe) {
  const int bi0 = fe.bi0, bi1 = fe.bi1, sb0 = fe.sb0, sb1 = fe.sb1;
  const int Ka = fe.ka2, Kb = fe.kb2;
  if (g <= -Ka && bi0 == 1 && sb0 != -1) {
    if (sb0 == 0) {
      if (g == 1) return weno5M_bnd(ff, 1);
      return weno5M(ff);
    } else if (sb0 == 1) {
      return weno5M(ff);
    }
  } else if (g > nn - Kb && bi1 == 1 && sb1 != -1) {
    if (sb1 == 0) {
      if (g == nn - 1) return (R(2) * ff[1] + R(5) * ff[0] - ff[-1]) / R(6);
      if (g == nn - 2) return weno5M_bnd(ff, 2);
      return weno5M(ff);
    } else if (sb1 == 1) {
      return weno5M(ff);
    }
  }
  return R(0);
}

// Stencil ranges of the projected values each scheme reads (set_parameters,
// OCFD_readpara.f90:288-315).  The hybrid's WENO5/WENO7 faces read subsets.
template <int SCHEME>
struct Stencil {
  static constexpr int PLO = -3, PHI = 4, MLO = -3, MHI = 4;
};
template <>
struct Stencil<SCH_WENO7> {
  static constexpr int PLO = -3, PHI = 3, MLO = -2, MHI = 4;
};
template <>
struct Stencil<SCH_WENO5> {
  static constexpr int PLO = -2, PHI = 2, MLO = -1, MHI = 3;
};

// Block-wide queue of OMP6 limiter evaluations (characteristic form,
// production build).  The monotonicity test of the ten characteristic
// components of a face is cheap; the limiter that a failed test calls is not,
// and the faces that need it are scattered, so a warp running it for one lane
// would idle the other 31.  Instead each flagged (face, component) is queued
// in shared memory -- its distance from the upwind point's value and a 16-bit
// tag (face of the tile, component, side) -- and the whole block evaluates the
// queue, one entry per thread: eigenvector row, the five projected stencil
// values and the limiter.
// Shared-memory layout of a tile's points.  FP32 characteristic form, x and y
// sweeps: one record of 20 floats a point (F+, unused x3, F-, u, v, w, c, A1,
// A2, A3).  Otherwise one array per variable (10 split fluxes, +7 face-state
// arrays for the characteristic form).  Measured at 256^3 against the arrays:
// FP32 x 3% and y 2% faster, z 0.6% slower; FP64 records of 18 doubles (two
// 16-byte halves of F+ and F-) 17% slower on y and z, whose blocks then no
// longer fit four to an SM.
template <int DIR, bool CHAR, typename R>
constexpr int face_ps() {
  return (CHAR && sizeof(R) == 4 && DIR != 2) ? 20 : 1;
}

// The mixed-precision hybrid: FP32 sweeps with the reference's splitting sums and
// schemes on stencil values (ocfd_face_values.cuh gives the reason).
template <int SCHEME, typename R>
constexpr bool face_on_values() {
  return OCFD_FEWER_DIVS && SCHEME == SCH_HYBRID && sizeof(R) == 4;
}

// Block-wide list of the faces that leave a sweep's common path (production
// build): the hybrid scheme's WENO faces, and in the characteristic form of a
// non-periodic direction the faces of the boundary closures.  Where the sensor is
// low a hybrid face is the linear scheme, 16 multiply-adds a component; the others
// need some ten times that, and their code would set the sweep's registers and
// hold up every warp that meets one.  So the common faces are finished at once,
// the others listed in shared memory (WENO7 faces from the front, the rest from
// the back), and the block evaluates (face, component) pairs one a thread,
// neighbouring threads on one component of neighbouring entries (long lists of hybrid
// faces: on two or three).  The characteristic form keeps
// the five values of a face (the change relative to its upwind points) for the
// face's own thread to project back.
template <int NF, bool CHAR>
struct FaceList {
  static constexpr int NVAL = CHAR ? 5 * NF : 0;
  template <typename R>
  static constexpr size_t bytes() {  // values, list
    return ((size_t)NVAL * sizeof(R) + NF * sizeof(unsigned short) + 15) / 16 * 16;
  }
};
template <bool CHAR, int SCHEME, bool ALLIN, typename R>
constexpr bool face_has_list() {
  if (face_on_values<SCHEME, R>()) return !CHAR;
  return OCFD_FEWER_DIVS && (SCHEME == SCH_HYBRID || (CHAR && !ALLIN));
}
template <bool CHAR, int SCHEME>
constexpr bool face_has_limiter() {
  return OCFD_FEWER_DIVS && CHAR && SCHEME == SCH_OMP6;
}
// points of a tile (two faces a thread: an even number of rows, which are swapped in pairs)
template <int FPT, int NP, int TF>
constexpr int face_points() {
  return NP * (FPT > 1 ? TF + 8 : TF + 7);
}
// values of a staged point: split fluxes (+ face state: u, v, w, c and, unless the
// sweep is axis aligned, the metric row), or the record's stride
template <bool CHAR, bool AXS, int PS>
constexpr int face_nvar() {
  return PS > 1 ? PS : (CHAR ? (AXS ? 14 : 17) : 10);
}

template <int NF>  // faces per block
struct LimQueue {
  static constexpr int CAP = 10 * NF;
  static_assert(16 * NF <= 65536, "a tag holds the face index and four bits");
  template <typename R>
  static constexpr size_t bytes() {  // values, tags
    return ((size_t)CAP * (sizeof(R) + sizeof(unsigned short)) + 15) / 16 * 16;
  }
};

// bytes of a sweep's queues in shared memory: limiter queue, face list, three counts
template <bool CHAR, int SCHEME, bool ALLIN, int NF, typename R>
constexpr size_t face_queue() {
  constexpr bool lim = face_has_limiter<CHAR, SCHEME>(), list = face_has_list<CHAR, SCHEME, ALLIN, R>();
  return (lim ? LimQueue<NF>::template bytes<R>() : 0) + (list ? FaceList<NF, CHAR>::template bytes<R>() : 0) +
         (lim || list ? 16 : 0);
}

}  // namespace ocfd

#include "ocfd_face_values.cuh"

namespace ocfd {

// Characteristic basis of one face, production build: the rows of L = S and
// R = S^-1 of flux_charteric (OCFD_inviscous_character.f90:216-248) applied
// without forming the matrices.  AXS: the sweep's metric row has a single
// non-zero component (box and 1-D grids), so the unit vectors are the coordinate
// axes and drop out of the projections.  Their signs are free: -l or -m changes
// the sign of one characteristic variable, -n swaps the two acoustic ones, and
// the schemes are odd and treat the components alike.
//
// With f'_i = f_i - u_i f_0 (the momentum part relative to the face's velocity)
// and A = f_4 - u.f' - V2 f_0, the five rows are
//   row 0  f_0 - (gamma-1)/c^2 A      rows 1, 2  l.f', m.f'
//   rows 3, 4  ((gamma-1) A -+ c n.f') / (2 c^2)
// and back: with s = d_3 + d_4, h_0 = d_0 + s and q = l d_1 + m d_2 + c (d_4 - d_3) n,
//   h_i = u_i h_0 + q_i,  h_4 = V2 h_0 + u.q + c^2/(gamma-1) s.
template <int DIR, bool AXS, typename R>
struct CharBasis {
  static constexpr int LI = DIR == 0 ? 1 : 0;  // AXS: the velocity component along l
  static constexpr int MI = DIR == 2 ? 1 : 2;  // and along m
  R u, v, w, c;
  R n1, n2, n3, l1, l2, l3;  // AXS: unused

  __device__ __forceinline__ void init(R u1, R v1, R w1, R c1, R a1, R a2, R a3) {
    u = u1;
    v = v1;
    w = w1;
    c = c1;
    if constexpr (!AXS) unit(a1, a2, a3, n1, n2, n3, l1, l2, l3);
  }
  // n = a / |a| and l normal to it (OCFD_inviscous_character.f90:216-230)
  static __device__ __forceinline__ void unit(R a1, R a2, R a3, R& n1, R& n2, R& n3, R& l1, R& l2, R& l3) {
    const R rs = rsqrt(xfma(a3, a3, xfma(a2, a2, xmul(a1, a1))));
    n1 = xmul(a1, rs);
    n2 = xmul(a2, rs);
    n3 = xmul(a3, rs);
    if (fabs(n3) <= fabs(n2)) {
      const R rl = rsqrt(xfma(n2, n2, xmul(n1, n1)));
      l1 = -xmul(n2, rl);
      l2 = xmul(n1, rl);
      l3 = R(0);
    } else {
      const R rl = rsqrt(xfma(n3, n3, xmul(n1, n1)));
      l1 = -xmul(n3, rl);
      l3 = xmul(n1, rl);
      l2 = R(0);
    }
  }
  __device__ __forceinline__ R vel(int q) const { return q == 0 ? u : (q == 1 ? v : w); }
  // m = n x l
  __device__ __forceinline__ R m1() const { return xfma(n2, l3, -xmul(n3, l2)); }
  __device__ __forceinline__ R m2() const { return xfma(n3, l1, -xmul(n1, l3)); }
  __device__ __forceinline__ R m3() const { return xfma(n1, l2, -xmul(n2, l1)); }
  __device__ __forceinline__ R V2() const { return xmul(xfma(w, w, xfma(v, v, xmul(u, u))), R(0.5)); }
  // A, n.f', l.f', m.f' of one vector f
  __device__ __forceinline__ void parts(const R* f, R V2_, R& A, R& fn, R& fl, R& fm) const {
    const R q[3] = {xfma(-u, f[0], f[1]), xfma(-v, f[0], f[2]), xfma(-w, f[0], f[3])};
    A = xfma(-V2_, f[0], xfma(-u, q[0], xfma(-v, q[1], xfma(-w, q[2], f[4]))));
    if constexpr (AXS) {
      fn = q[DIR];
      fl = q[LI];
      fm = q[MI];
    } else {
      fn = xfma(n3, q[2], xfma(n2, q[1], xmul(n1, q[0])));
      fl = xfma(l3, q[2], xfma(l2, q[1], xmul(l1, q[0])));
      fm = xfma(m3(), q[2], xfma(m2(), q[1], xmul(m1(), q[0])));
    }
  }
  // c = L f for one vector
  __device__ __forceinline__ void proj(const R* f, R KK, R KK1, R X1, R V2_, R* cc) const {
    R A, fn;
    parts(f, V2_, A, fn, cc[1], cc[2]);
    const R KA = xmul(KK1, A);
    cc[0] = xfma(-KK, A, f[0]);
    cc[3] = xfma(-X1, fn, KA);
    cc[4] = xfma(X1, fn, KA);
  }
  // the same with row 0 times c^2 and rows 3, 4 times 2 c^2 (no division by c)
  __device__ __forceinline__ void proj_scaled(const R* f, R g1, R c2, R V2_, R* cc) const {
    R A, fn;
    parts(f, V2_, A, fn, cc[1], cc[2]);
    const R GA = xmul(g1, A);
    cc[0] = xfma(c2, f[0], -GA);
    cc[3] = xfma(-c, fn, GA);
    cc[4] = xfma(c, fn, GA);
  }
  // coefficients of row r of L (OCFD_inviscous_character.f90:233-243): KK = (gamma-1)/c^2,
  // X1 = 1/(2c)
  __device__ __forceinline__ void row(int r, R KK, R X1, R V2_, R* q) const {
    const R na = AXS ? R(DIR == 0) : n1, nb = AXS ? R(DIR == 1) : n2, nc = AXS ? R(DIR == 2) : n3;
    if (r == 1 || r == 2) {
      R x1 = AXS ? R(LI == 0) : l1, x2 = AXS ? R(LI == 1) : l2, x3 = AXS ? R(0) : l3;
      if (r == 2) {
        x1 = AXS ? R(0) : m1();
        x2 = AXS ? R(MI == 1) : m2();
        x3 = AXS ? R(MI == 2) : m3();
      }
      q[0] = -xfma(w, x3, xfma(v, x2, xmul(u, x1)));
      q[1] = x1;
      q[2] = x2;
      q[3] = x3;
      q[4] = R(0);
    } else if (r == 0) {
      q[0] = xfma(-KK, V2_, R(1));
      q[1] = xmul(KK, u);
      q[2] = xmul(KK, v);
      q[3] = xmul(KK, w);
      q[4] = -KK;
    } else {
      const R KK1 = xmul(KK, R(0.5)), sX = r == 3 ? X1 : -X1;
      const R un = xfma(w, nc, xfma(v, nb, xmul(u, na)));
      q[0] = xfma(sX, un, xmul(KK1, V2_));
      q[1] = xfma(-sX, na, -xmul(KK1, u));
      q[2] = xfma(-sX, nb, -xmul(KK1, v));
      q[3] = xfma(-sX, nc, -xmul(KK1, w));
      q[4] = KK1;
    }
  }
  // the same in proj_scaled's scaling, without branches: with k the row's weights of
  // f' and kA its weight of A, the coefficients are k - kA u, kA, and kA V2 - k.u
  // (plus c^2 for row 0)
  __device__ __forceinline__ void row_scaled(int r, R g1, R* q) const {
    const R kA = r == 0 ? -g1 : (r >= 3 ? g1 : R(0));
    const R kn = r == 3 ? -c : (r == 4 ? c : R(0));
    R k[3];
    if constexpr (AXS) {
      k[DIR] = kn;
      k[LI] = r == 1 ? R(1) : R(0);
      k[MI] = r == 2 ? R(1) : R(0);
    } else {
      k[0] = r == 1 ? l1 : (r == 2 ? m1() : xmul(kn, n1));
      k[1] = r == 1 ? l2 : (r == 2 ? m2() : xmul(kn, n2));
      k[2] = r == 1 ? l3 : (r == 2 ? m3() : xmul(kn, n3));
    }
    q[0] = xfma(kA, V2(), xfma(-w, k[2], xfma(-v, k[1], xfma(-u, k[0], r == 0 ? xmul(c, c) : R(0)))));
    q[1] = xfma(-kA, u, k[0]);
    q[2] = xfma(-kA, v, k[1]);
    q[3] = xfma(-kA, w, k[2]);
    q[4] = kA;
  }
  // hh = R h0 (OCFD_inviscous_character.f90:284-288)
  __device__ __forceinline__ void back(const R* h0, R* hh, R inv_gm1) const {
    const R s = xadd(h0[3], h0[4]);
    const R k = xmul(c, xadd(h0[4], -h0[3]));
    hh[0] = xadd(h0[0], s);
    R q[3];
    if constexpr (AXS) {
      q[DIR] = k;
      q[LI] = h0[1];
      q[MI] = h0[2];
    } else {
      q[0] = xfma(k, n1, xfma(m1(), h0[2], xmul(l1, h0[1])));
      q[1] = xfma(k, n2, xfma(m2(), h0[2], xmul(l2, h0[1])));
      q[2] = xfma(k, n3, xfma(m3(), h0[2], xmul(l3, h0[1])));
    }
    hh[1] = xfma(u, hh[0], q[0]);
    hh[2] = xfma(v, hh[0], q[1]);
    hh[3] = xfma(w, hh[0], q[2]);
    hh[4] = xfma(V2(), hh[0], xfma(u, q[0], xfma(v, q[1], xfma(w, q[2], xmul(xmul(xmul(c, c), inv_gm1), s)))));
  }
};

// CharBasis::proj_scaled of two vectors at once, in the two lanes of packed FP32
// operations; each lane performs its own explicitly rounded operations (a
// negation is a product with -1, which is exact), so both lanes give its bits.
template <int DIR, bool AXS>
__device__ __forceinline__ void char_proj2(const CharBasis<DIR, AXS, float>& b, const F2* f, float g1, float c2,
                                           float V2_, F2* cc) {
  const F2 q[3] = {fma2(f2(-b.u), f[0], f[1]), fma2(f2(-b.v), f[0], f[2]), fma2(f2(-b.w), f[0], f[3])};
  const F2 A = fma2(f2(-V2_), f[0], fma2(f2(-b.u), q[0], fma2(f2(-b.v), q[1], fma2(f2(-b.w), q[2], f[4]))));
  const F2 GA = mul2(f2(g1), A);
  F2 fn;
  if constexpr (AXS) {
    fn = q[DIR];
    cc[1] = q[CharBasis<DIR, AXS, float>::LI];
    cc[2] = q[CharBasis<DIR, AXS, float>::MI];
  } else {
    fn = fma2(f2(b.n3), q[2], fma2(f2(b.n2), q[1], mul2(f2(b.n1), q[0])));
    cc[1] = fma2(f2(b.l3), q[2], fma2(f2(b.l2), q[1], mul2(f2(b.l1), q[0])));
    cc[2] = fma2(f2(b.m3()), q[2], fma2(f2(b.m2()), q[1], mul2(f2(b.m1()), q[0])));
  }
  cc[0] = fma2(f2(c2), f[0], mul2(f2(-1.0f), GA));
  cc[3] = fma2(f2(-b.c), fn, GA);
  cc[4] = fma2(f2(b.c), fn, GA);
}

// One queued limiter evaluation (OCFD_inviscous_character.f90:205-248 for the
// face state and row r of the left eigenvector matrix, :256-270 for the
// projection, OCFD_Schemes_1.f90:212-224 for the limiter): the face whose
// stencil window starts at wb, component r, F+ points -2..2 (window 1..5) or
// F- mirrored (window 6..2).  p0: the unlimited value minus the upwind point's,
// in proj_scaled's scaling; returns the limiter's change of the value, in the
// same scaling (the limiter is homogeneous, so no entry divides: the entries of a
// tile keep one warp of the block busy, and the others wait for it).
// Written in explicitly rounded operations, so that every kernel that inlines
// it produces the same bits.
// win(var, q): value var at point q of the face's window.
template <int DIR, bool AXS, typename R, typename W>
__device__ __forceinline__ R lim_eval(const W& win, int r, int minus, R p0, R gm1) {
  auto mean = [&](int var) { return xmul(xadd(win(var, 3), win(var, 4)), R(0.5)); };
  CharBasis<DIR, AXS, R> cb;
  cb.init(mean(10), mean(11), mean(12), mean(13), AXS ? R(0) : mean(14), AXS ? R(0) : mean(15),
          AXS ? R(0) : mean(16));
  R c[5];
  cb.row_scaled(r, gm1, c);
  const int v0 = minus ? 5 : 0;
  R x[5];
#pragma unroll
  for (int k = 0; k < 5; k++) {
    const int q = minus ? 6 - k : 1 + k;
    x[k] = xfma(c[4], win(v0 + 4, q),
                xfma(c[3], win(v0 + 3, q), xfma(c[2], win(v0 + 2, q), xfma(c[1], win(v0 + 1, q), xmul(c[0], win(v0, q))))));
  }
  // everything relative to the upwind point x[2]; vlc: the lc reference
  const R y1 = xadd(x[1], -x[2]), y3 = xadd(x[3], -x[2]);
  const R vlc = minus ? y3 : y1;
  const R kappa = R(Omp6C::kappa);
  const R d1 = xfma(R(-2), y1, xadd(x[0], -x[2]));
  const R d2 = xadd(y1, y3);
  const R d3 = xfma(R(-2), y3, xadd(x[4], -x[2]));
  const R ul = -xmul(kappa, y1);
  const R md = xfma(R(-0.5), minmod4(xfma(R(4), d2, -d3), xfma(R(4), d3, -d2), d2, d3), xmul(R(0.5), y3));
  const R lc = xfma(R(Omp6C::kappa / 3.0), minmod4(xfma(R(4), d1, -d2), xfma(R(4), d2, -d1), d2, d1),
                    xmul(R(-0.5), vlc));
  const R fmin = rmax(rmin(rmin(R(0), y3), md), rmin(rmin(R(0), ul), lc));
  const R fmax = rmin(rmax(rmax(R(0), y3), md), rmax(rmax(R(0), ul), lc));
  return minmod2(xadd(fmax, -p0), xadd(fmin, -p0));
}

// ---------------------------------------------------------------------------
// ALLIN: every face of the launch is an interior face (periodic direction), so
// the boundary-closure paths are compiled out.
// The body of one block; (bx, by, bz) are its block coordinates within the
// instance's own launch grid.
// TMA: the eight input arrays were staged in shared memory by the caller
// (tile: TmaBox slots of d, u, v, w, T, A1, A2, A3; toff: offset of the first
// stencil point / pencil in the tile's innermost dimension).
// AXS (production build, ALLIN sweeps): the sweep's metric row has a single
// non-zero component (axis_aligned); the splitting and the characteristic
// basis use the axis-aligned forms.
// FPT > 1: that many consecutive faces a thread (NP * TF / FPT threads).
template <int DIR, bool CHAR, int SCHEME, bool ALLIN, int NP, int TF, typename R, typename S, bool TMA, bool AXS,
          int FPT>
__device__ __forceinline__ void face_body_main(const FaceArgs<S>& a, const int bx, const int by, const int bz, R* sm,
                                               const S* tile, int toff, R* qbase, int* qcount) {
  constexpr int LT = TF + 7;
  // shared memory (face_ps).  Records (PS > 1): F+ and F- each start on a
  // 16-byte boundary (GAP unused values after F+), so that four components of
  // a stencil point come in one 16-byte load; the 80-byte record stride keeps
  // a warp's 16-byte accesses free of bank conflicts.
  constexpr int PS = FPT > 1 ? 1 : face_ps<DIR, CHAR, R>();
  constexpr int GAP = PS > 1 ? 3 : 0;
  constexpr int NT = NP * TF / FPT;
  static_assert(FPT == 1 || (FPT == 2 && ALLIN && NP == 8 && SCHEME == SCH_HYBRID), "two faces a thread");
  constexpr int VS = PS > 1 ? 1 : face_points<FPT, NP, TF>();  // stride between variables
  // point of the tile.  Two faces a thread: a row of eight pencils is half the
  // banks, and a half warp reads rows l and l + 2; swapping the rows of every other
  // pair puts them in different halves.
  auto row = [](int l) -> int { return l ^ ((l >> 1) & 1); };
  auto PI = [&](int l, int p) -> int {
    if (FPT > 1) return row(l) * NP + p;
    return DIR == 0 ? p * LT + l : l * NP + p;
  };
  auto SI = [&](int var, int l, int p) -> int { return var * VS + (var >= 5 ? GAP : 0) + PI(l, p) * PS; };

  const Grid& G = a.g;
  const Phys& ph = a.ph;
  const int nn = G.len(DIR);
  int g0, pbase;
  if (DIR == 0) {
    g0 = a.fbeg + bx * TF;
    pbase = by * NP;  // NP consecutive j of plane k = bz + 1
  } else {
    g0 = a.fbeg + by * TF;
    pbase = bx * NP;
  }
  // pencil p -> (i,j,k) with the along-direction index left at 0
  auto pencil = [&](int p, int& i, int& j, int& k) -> bool {
    if (DIR == 0) {
      i = 0;
      j = pbase + p + 1;
      k = bz + 1;
      return j <= G.ny;
    } else if (DIR == 1) {
      i = pbase + p + 1;
      j = 0;
      k = bz + 1;
      return i <= G.nx;
    } else {
      i = pbase + p + 1;
      j = bz + 1;
      k = 0;
      return i <= G.nx;
    }
  };
  const long long hs = G.hstride(DIR);
  const R gam = R(ph.gamma), ma = R(ph.ma);
  // The queues, after the staged points (or at qbase, where they may share memory
  // with the staged input tile, dead after phase 1; the counts, written before
  // phase 1, then lie past that tile, at qcount).  Deferred OMP6 limiter: JC values,
  // JC tags (face of the tile * 16 + component * 2 + side); face list: values, faces.
  constexpr bool DEFER = face_has_limiter<CHAR, SCHEME>(), LIST = face_has_list<CHAR, SCHEME, ALLIN, R>();
  constexpr bool HQ = SCHEME == SCH_HYBRID && OCFD_FEWER_DIVS;
  // WENO sweeps of the production build work on stencil differences
  constexpr bool WDIFF = (SCHEME == SCH_WENO5 || SCHEME == SCH_WENO7) && OCFD_FEWER_DIVS;
  constexpr int JC = LimQueue<NP * TF>::CAP;
  R* const jv = qbase ? qbase : sm + face_nvar<CHAR, AXS, PS>() * face_points<FPT, NP, TF>();
  unsigned short* const jtag = reinterpret_cast<unsigned short*>(jv + JC);
  R* const lv = DEFER ? jv + LimQueue<NP * TF>::template bytes<R>() / sizeof(R) : jv;
  unsigned short* const ltag = reinterpret_cast<unsigned short*>(lv + FaceList<NP * TF, CHAR>::NVAL);
  int* const jn = qbase ? qcount
                        : reinterpret_cast<int*>(LIST ? lv + FaceList<NP * TF, CHAR>::template bytes<R>() / sizeof(R)
                                                      : jv + LimQueue<NP * TF>::template bytes<R>() / sizeof(R));
  int* const ln = jn + 1;  // the list's two counts
  if ((DEFER || LIST) && threadIdx.x < 3) jn[threadIdx.x] = 0;

  // ---- phase 1: split fluxes of the tile's points into shared memory
  // (blockDim.x == NT, so the trip count is known)
#pragma unroll
  for (int t0 = 0; t0 < NP * LT; t0 += NT) {
    const int t = t0 + threadIdx.x;
    if (t >= NP * LT) break;
    int l, p;
    if (DIR == 0 && FPT == 1) {
      l = t % LT;
      p = t / LT;
    } else {
      p = t % NP;
      l = t / NP;
    }
    int i, j, k;
    bool ok = pencil(p, i, j, k);
    const int gl = g0 - 3 + l;  // point index along DIR
    ok = ok && gl <= nn + LAP;
    R d = R(1), u = R(1), v = R(1), w = R(1), T = R(1), A1 = R(1), A2 = R(1), A3 = R(1);
    if (ok && TMA) {
      using B = TmaBox<DIR, NP, TF, S, FPT>;
      const int e = DIR == 0 ? p * B::BX + l + toff : l * B::BX + p + toff;
      d = R(tile[e]);
      if constexpr (sizeof(S) == 4) {  // slots 1-4: the interleaved u,v,w,T tile
        const float4 t = reinterpret_cast<const float4*>(tile + B::SLOT_ELEMS)[e];
        u = R(t.x);
        v = R(t.y);
        w = R(t.z);
        T = R(t.w);
      } else {
        u = R(tile[B::SLOT_ELEMS + e]);
        v = R(tile[2 * B::SLOT_ELEMS + e]);
        w = R(tile[3 * B::SLOT_ELEMS + e]);
        T = R(tile[4 * B::SLOT_ELEMS + e]);
      }
      const int m0 = 13 + 3 * DIR;
      if constexpr (AXS) {
        const R Ad = R(tile[5 * B::SLOT_ELEMS + e]);  // the direction's metric
        A1 = DIR == 0 ? Ad : R(0);
        A2 = DIR == 1 ? Ad : R(0);
        A3 = DIR == 2 ? Ad : R(0);
      } else {
        A1 = ((ph.metzero >> m0) & 1u) ? R(0) : R(tile[5 * B::SLOT_ELEMS + e]);
        A2 = ((ph.metzero >> (m0 + 1)) & 1u) ? R(0) : R(tile[6 * B::SLOT_ELEMS + e]);
        A3 = ((ph.metzero >> (m0 + 2)) & 1u) ? R(0) : R(tile[7 * B::SLOT_ELEMS + e]);
      }
    } else if (ok) {
      long long h = G.ih(i, j, k) + (long long)gl * hs;
      d = R(__ldg(a.d + h));
      if constexpr (sizeof(S) == 4) {  // FP32 copies: u,v,w,T interleaved
        const float4 t = __ldg(reinterpret_cast<const float4*>(a.q4) + h);
        u = R(t.x);
        v = R(t.y);
        w = R(t.z);
        T = R(t.w);
      } else {
        u = R(__ldg(a.u + h));
        v = R(__ldg(a.v + h));
        w = R(__ldg(a.w + h));
        T = R(__ldg(a.T + h));
      }
      if constexpr (AXS) {
        A1 = DIR == 0 ? R(__ldg(a.A1 + h)) : R(0);
        A2 = DIR == 1 ? R(__ldg(a.A2 + h)) : R(0);
        A3 = DIR == 2 ? R(__ldg(a.A3 + h)) : R(0);
      } else {
        A1 = met_at<R>(ph, 13 + 3 * DIR, a.A1, h);
        A2 = met_at<R>(ph, 14 + 3 * DIR, a.A2, h);
        A3 = met_at<R>(ph, 15 + 3 * DIR, a.A3, h);
      }
    }
#if OCFD_FEWER_DIVS
    const R c = sqrt(T) * R(ph.inv_ma);
#else
    const R c = sqrt(T) / ma;  // cc: OCFD_inviscous.f90:67
#endif
    R fp[5], fm[5];
#if OCFD_FEWER_DIVS
    if constexpr (AXS) {
      const R Ad = DIR == 0 ? A1 : (DIR == 1 ? A2 : A3);
      if (a.split == 1)
        split_sw_axis<DIR>(ph, gam, c, d, u, v, w, Ad, fp, fm);
      else
        split_llf_axis<DIR>(ph, gam, c, d, u, v, w, Ad, fp, fm);
    } else {
      if (a.split == 1)
        split_sw(ph, gam, c, d, u, v, w, A1, A2, A3, fp, fm);
      else
        split_llf(ph, gam, c, d, u, v, w, A1, A2, A3, fp, fm);
    }
#else
    if (a.split == 1)
      split_sw_ref(ph, gam, c, d, u, v, w, A1, A2, A3, fp, fm);
    else
      split_llf_ref(ph, gam, c, d, u, v, w, A1, A2, A3, fp, fm);
#endif
    if constexpr (PS > 1) {
      // the point's record in 16-byte stores (the unused slots get zeros)
      float4* r4 = reinterpret_cast<float4*>(sm + PI(l, p) * PS);
      r4[0] = make_float4(fp[0], fp[1], fp[2], fp[3]);
      r4[1] = make_float4(fp[4], 0.f, 0.f, 0.f);
      r4[2] = make_float4(fm[0], fm[1], fm[2], fm[3]);
      r4[3] = make_float4(fm[4], u, v, w);
      r4[4] = make_float4(c, A1, A2, A3);
    } else {
#pragma unroll
      for (int m = 0; m < 5; m++) {
        sm[SI(m, l, p)] = fp[m];
        sm[SI(5 + m, l, p)] = fm[m];
      }
      if (CHAR) {
        sm[SI(10, l, p)] = u;
        sm[SI(11, l, p)] = v;
        sm[SI(12, l, p)] = w;
        sm[SI(13, l, p)] = c;
        if (!AXS) {  // the axis-aligned basis needs no metrics
          sm[SI(14, l, p)] = A1;
          sm[SI(15, l, p)] = A2;
          sm[SI(16, l, p)] = A3;
        }
      }
    }
  }
  __syncthreads();

  // ---- phase 2: one face per thread
  R U[8];
#pragma unroll
  for (int q = 0; q < 8; q++) U[q] = R(ph.ud7l[q]);
  R* out = reinterpret_cast<R*>(a.hh);
  // window element (var, stencil offset s) of this thread's face at
  // wb[var*VS + (var >= 5 ? GAP : 0) + (s+3)*QS]
  constexpr int QS = (DIR == 0 ? 1 : NP) * PS;
  // state of a face with queued limiter evaluations: its unlimited flux, the
  // flags of the queued components (F+ bits 0-4, F- bits 5-9), each side's first
  // queue entry, and the face's output offset
  R dH[5];
  unsigned dfl = 0;
  int djP = 0, djM = 0;
  // output offset of a face finished after a queue, and a listed face's entry
  long long dfo[FPT];
  int hslot[FPT];
#pragma unroll
  for (int n = 0; n < FPT; n++) {
    dfo[n] = 0;
    hslot[n] = -1;
  }
  // face x of the tile (0 .. NP * TF - 1): its pencil, its index in the tile, and a
  // window accessor
  auto face_of = [&](int x, int& f, int& p) {
    if (DIR == 0 && FPT == 1) {
      f = x % TF;
      p = x / TF;
    } else {
      p = x % NP;
      f = x / NP;
    }
  };
  auto window = [&](int x) {
    int f, p;
    face_of(x, f, p);
    if constexpr (FPT > 1) {
      return [=](int var, int q) -> R { return sm[var * VS + ((f + q) ^ (((f + q) >> 1) & 1)) * NP + p]; };
    } else {
      const R* wb = sm + PI(f, p) * PS;
      return [=](int var, int q) -> R { return wb[var * VS + (var >= 5 ? GAP : 0) + q * QS]; };
    }
  };
  // queue entries of one side's flagged components, in the order of r
  auto push = [&](unsigned fl, const R* p0, int side, int x) -> int {
    const int first = atomicAdd(jn, __popc(fl));
    int e = first;
#pragma unroll
    for (int r = 0; r < 5; r++) {
      if ((fl >> r) & 1u) {
        jv[e] = p0[r];
        jtag[e] = (unsigned short)(16 * x + 2 * r + side);
        e++;
      }
    }
    return first;
  };
  // front: a WENO7 face; returns the entry
  auto list_face = [&](int x, bool front) -> int {
    const int n = atomicAdd(ln + (front ? 0 : 1), 1);
    const int slot = front ? n : NP * TF - 1 - n;
    ltag[slot] = (unsigned short)x;
    return slot;
  };

  if constexpr (FPT > 1) {
    // ---- two consecutive faces (a: f0, b: f0 + 1) from their nine points
    const int p = threadIdx.x % NP, f0 = 2 * (threadIdx.x / NP);
    int i, j, k;
    const bool ok = pencil(p, i, j, k);
    // row f0 + x of the tile (f0 even): pair x / 2, the half of the pair from the
    // parities of x, x / 2 and f0 / 2
    const int odd = (f0 >> 1) & 1;
    const R* const even_row = sm + (f0 + odd) * NP + p;
    const R* const odd_row = sm + (f0 + 1 - odd) * NP + p;
    auto P = [&](int var, int x) -> R {
      return ((((x >> 1) ^ x) & 1) ? odd_row : even_row)[var * VS + (x >> 1) * 2 * NP];
    };
    bool act[2];
    long long fo[2];
    int type[2];
#pragma unroll
    for (int n = 0; n < 2; n++) {
      const int g = g0 + f0 + n;
      act[n] = ok && g <= a.fend;
      fo[n] = G.face(DIR, g, DIR == 0 ? g : i, DIR == 1 ? g : j, DIR == 2 ? g : k);
      type[n] = 0;
      if (SCHEME == SCH_HYBRID && act[n]) {
        const long long h = G.ih(i, j, k) + (long long)g * hs;
        type[n] = hybrid_index(rmax(__ldg(a.rh + h), __ldg(a.rh + h + hs)), ph.hyb1, ph.hyb2);
      }
    }
    R H[2][5];
    if constexpr (HQ) {
      // the linear scheme of both faces; the others go to the list
      if ((act[0] && type[0] == 1) || (act[1] && type[1] == 1)) {
        R X[2][5], f[5];
#pragma unroll
        for (int x = 0; x < 9; x++) {
#pragma unroll
          for (int v = 0; v < 5; v++) f[v] = P(v, x);
#pragma unroll
          for (int n = 0; n < 2; n++) {
            const int q = x - n;
            if (q < 0 || q > 7) continue;
#pragma unroll
            for (int v = 0; v < 5; v++) H[n][v] = q == 0 ? xmul(U[0], f[v]) : xfma(U[q], f[v], H[n][v]);
          }
        }
#pragma unroll
        for (int x = 8; x >= 0; x--) {
#pragma unroll
          for (int v = 0; v < 5; v++) f[v] = P(5 + v, x);
#pragma unroll
          for (int n = 0; n < 2; n++) {
            const int q = 7 - (x - n);
            if (q < 0 || q > 7) continue;
#pragma unroll
            for (int v = 0; v < 5; v++) X[n][v] = q == 0 ? xmul(U[0], f[v]) : xfma(U[q], f[v], X[n][v]);
          }
        }
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int v = 0; v < 5; v++) H[n][v] = xadd(H[n][v], X[n][v]);
      }
#pragma unroll
      for (int n = 0; n < 2; n++) {
        if (!act[n]) continue;
        if (type[n] == 1) {
          hf_store5(out, fo[n], a.fs, H[n]);
        } else {
          hslot[n] = list_face((f0 + n) * NP + p, type[n] == 2);
          dfo[n] = fo[n];
        }
      }
    }
  } else
  for (int once = 0; once < 1; once++) {
    const int t = threadIdx.x;
    int f, p;
    if (DIR == 0) {
      f = t % TF;
      p = t / TF;
    } else {
      p = t % NP;
      f = t / NP;
    }
    int i, j, k;
    if (!pencil(p, i, j, k)) continue;
    const int g = g0 + f;
    if (g > a.fend) continue;
    const R* wb = sm + PI(f, p) * PS;
    auto W = [&](int var, int q) -> R { return wb[var * VS + (var >= 5 ? GAP : 0) + q * QS]; };
    // components vb..vb+3 (vb = 0: F+, 5: F-) of stencil point q
    auto W4 = [&](int vb, int q, R* o) {
      if constexpr (PS > 1) {
        const float4 t = *reinterpret_cast<const float4*>(wb + vb + (vb >= 5 ? GAP : 0) + q * QS);
        o[0] = t.x;
        o[1] = t.y;
        o[2] = t.z;
        o[3] = t.w;
      } else {
#pragma unroll
        for (int v = 0; v < 4; v++) o[v] = W(vb + v, q);
      }
    };
    int ii = DIR == 0 ? g : i, jj = DIR == 1 ? g : j, kk = DIR == 2 ? g : k;
    const long long fo = G.face(DIR, g, ii, jj, kk);
    int ihy = 0;
    if (SCHEME == SCH_HYBRID) {
      // OCFD_inviscous.f90:76-81: Rhb0 = max(Rhybrid(g), Rhybrid(g+1))
      long long h = G.ih(i, j, k) + (long long)g * hs;
      double r0 = __ldg(a.rh + h), r1 = __ldg(a.rh + h + hs);
      ihy = hybrid_index(rmax(r0, r1), ph.hyb1, ph.hyb2);
    }
    const int bi0 = ph.bi[2 * DIR], bi1 = ph.bi[2 * DIR + 1], sb0 = ph.sb[2 * DIR], sb1 = ph.sb[2 * DIR + 1];
    // components vb..vb+4 of stencil point q
    auto load5 = [&](int vb, int q, R* f) {
      W4(vb, q, f);
      f[4] = W(vb + 4, q);
    };
    // production build: the linear schemes (UD7L and the hybrid's linear faces)
    // commute with the characteristic projection
    constexpr bool LIN = (SCHEME == SCH_UD7L || SCHEME == SCH_HYBRID) && OCFD_FEWER_DIVS;
    auto linear = [&](R* h) {
      R x[5], fp[5], fm[5];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        load5(0, q, fp);
        load5(5, 7 - q, fm);
#pragma unroll
        for (int v = 0; v < 5; v++) {
          h[v] = q == 0 ? xmul(U[0], fp[v]) : xfma(U[q], fp[v], h[v]);
          x[v] = q == 0 ? xmul(U[0], fm[v]) : xfma(U[q], fm[v], x[v]);
        }
      }
#pragma unroll
      for (int v = 0; v < 5; v++) h[v] = xadd(h[v], x[v]);
    };

    if (!CHAR) {
      // ---- flux-vector form: h1 (F+) and h2 (F-) per variable
      const int ib1 = (bi0 == 0 || sb0 == -1) ? 0 : -ph.ka1 + 1, ie1 = (bi1 == 0 || sb1 == -1) ? nn : nn - ph.kb1;
      const int ib2 = (bi0 == 0 || sb0 == -1) ? 0 : -ph.ka2 + 1, ie2 = (bi1 == 0 || sb1 == -1) ? nn : nn - ph.kb2;
      const bool inner = ALLIN || (g >= ib1 && g <= ie1 && g >= ib2 && g <= ie2);
      if (LIN && inner) {
        if (HQ && ihy != 1) {
          hslot[0] = list_face(t, ihy == 2);
        } else if (sizeof(R) == 4) {
          R h[5];
          linear(h);
          hf_store5(out, fo, a.fs, h);
        } else {
          // FP64: component by component; five at a time take 70 to 100 registers, a block
          // fewer per SM (UD7L, ms per step: 97x80x33 with walls 0.543 -> 0.475, periodic
          // 129x95x70 0.760 -> 0.724; FP32 gains 2% there and loses 5% in the merged launch)
#pragma unroll 1
          for (int m = 0; m < 5; m++) {
            R h = xmul(U[0], W(m, 0)), x = xmul(U[0], W(5 + m, 7));
#pragma unroll
            for (int q = 1; q < 8; q++) {
              h = xfma(U[q], W(m, q), h);
              x = xfma(U[q], W(5 + m, 7 - q), x);
            }
            out[hf_at(fo, a.fs, m)] = xadd(h, x);
          }
        }
        continue;
      }
      if (inner) {
#pragma unroll 1
        for (int m = 0; m < 5; m++) {
          R h1, h2;
          if constexpr (WDIFF) {
            R vp[7], vm[7];  // the F+ window and the F- window mirrored about the face
#pragma unroll
            for (int q = 0; q < 7; q++) {
              vp[q] = W(m, q);
              vm[q] = W(5 + m, 7 - q);
            }
            h1 = xadd(vp[3], vm[3]);
            h2 = weno_pair<SCHEME>(vp, vm);
          } else {
            R wv[8];
#pragma unroll
            for (int q = 0; q < 8; q++) wv[q] = W(m, q);
            h1 = schemeP<SCHEME>(wv + 3, U, ihy);
#pragma unroll
            for (int q = 0; q < 8; q++) wv[q] = W(5 + m, q);
            h2 = schemeM<SCHEME>(wv + 3, U, ihy);
          }
          if (OCFD_FV_SUMMED) {
            out[hf_at(fo, a.fs, m)] = h1 + h2;
          } else {
            out[fo + (long long)m * a.fs] = h1;
            out[fo + (long long)(5 + m) * a.fs] = h2;
          }
        }
      } else if (!ALLIN) {
#pragma unroll 1
        for (int m = 0; m < 5; m++) {
          R wv[8];
#pragma unroll
          for (int q = 0; q < 8; q++) wv[q] = W(m, q);
          const R h1 = nc_flux1_bnd<SCHEME>(wv + 3, U, g, nn, ihy, ph, DIR);
#pragma unroll
          for (int q = 0; q < 8; q++) wv[q] = W(5 + m, q);
          const R h2 = nc_flux2_bnd<SCHEME>(wv + 3, U, g, nn, ihy, ph, DIR);
          if (OCFD_FV_SUMMED) {
            out[hf_at(fo, a.fs, m)] = h1 + h2;
          } else {
            out[fo + (long long)m * a.fs] = h1;
            out[fo + (long long)(5 + m) * a.fs] = h2;
          }
        }
      }
      continue;
    }

    // ---- characteristic form (flux_charteric)
    const int ia = (bi0 == 0 || sb0 != 0) ? 0 : 1;
    const int ibf = (bi1 == 0 || sb1 != 0) ? nn : nn - 1;
    R hh[5];
    if (!ALLIN && (g < ia || g > ibf)) {
      // non-reflecting boundary faces, OCFD_inviscous_character.f90:295-309
#pragma unroll 1
      for (int m = 0; m < 5; m++) {
        if (g == 0)
          hh[m] = (R(2) * W(m, 4) + R(5) * W(m, 5) - W(m, 6) + R(2) * W(5 + m, 6) - R(7) * W(5 + m, 5) +
                   R(11) * W(5 + m, 4)) / R(6);
        else
          hh[m] = (R(2) * W(m, 1) - R(7) * W(m, 2) + R(11) * W(m, 3) + R(2) * W(5 + m, 3) + R(5) * W(5 + m, 2) -
                   W(5 + m, 1)) / R(6);
      }
    } else {
      const bool inner1 =
          ALLIN || ((bi0 == 0 || g > -ph.ka1 || sb0 == -1) && (bi1 == 0 || g <= nn - ph.kb1 || sb1 == -1));
      const bool inner2 =
          ALLIN || ((bi0 == 0 || g > -ph.ka2 || sb0 == -1) && (bi1 == 0 || g <= nn - ph.kb2 || sb1 == -1));
      const bool inner = inner1 && inner2;
      if (LIN && inner && (SCHEME == SCH_UD7L || ihy == 1)) {
        linear(hh);
      } else if (HQ && inner) {
        hslot[0] = list_face(t, ihy == 2);
        dfo[0] = fo;
        continue;
      } else if (ihy == 1) {
        // linear hybrid face: no characteristic projection (:192-194, :281-282)
#pragma unroll 1
        for (int m = 0; m < 5; m++) {
          R wv[8];
#pragma unroll
          for (int q = 0; q < 8; q++) wv[q] = W(m, q);
          const R h1 = (ALLIN || inner) ? schemeP<SCHEME>(wv + 3, U, ihy) : ch_flux1_bnd(wv + 3, g, nn, face_ends(ph, DIR));
#pragma unroll
          for (int q = 0; q < 8; q++) wv[q] = W(5 + m, q);
          const R h2 = (ALLIN || inner) ? schemeM<SCHEME>(wv + 3, U, ihy) : ch_flux2_bnd(wv + 3, g, nn, face_ends(ph, DIR));
          hh[m] = h1 + h2;
        }
      } else {
        // face state: arithmetic means of the two neighbours (:205-211)
        auto mean = [&](int var) -> R { return xmul(xadd(W(var, 3), W(var, 4)), R(0.5)); };
        const R u1 = mean(10);
        const R v1 = mean(11);
        const R w1 = mean(12);
        const R c1 = mean(13);
        const R a1 = AXS ? R(0) : mean(14);
        const R a2 = AXS ? R(0) : mean(15);
        const R a3 = AXS ? R(0) : mean(16);
        // orthonormal basis (n,l,m) and L = S, R = S^-1 (:216-248)
#if OCFD_FEWER_DIVS
        CharBasis<DIR, AXS, R> cb;
        cb.init(u1, v1, w1, c1, a1, a2, a3);
        const R V2 = cb.V2();
        const R g1 = xadd(R(ph.gamma), R(-1));
#else
        R ss = sqrt(a1 * a1 + a2 * a2 + a3 * a3);
        const R n1 = a1 / ss, n2 = a2 / ss, n3 = a3 / ss;
        R l1, l2, l3;
        if (fabs(n3) <= fabs(n2)) {
          ss = sqrt(n1 * n1 + n2 * n2);
          l1 = -n2 / ss;
          l2 = n1 / ss;
          l3 = R(0);
        } else {
          ss = sqrt(n1 * n1 + n3 * n3);
          l1 = -n3 / ss;
          l3 = n1 / ss;
          l2 = R(0);
        }
        const R m1 = n2 * l3 - n3 * l2, m2 = n3 * l1 - n1 * l3, m3 = n1 * l2 - n2 * l1;
        const R un = u1 * n1 + v1 * n2 + w1 * n3;
        const R ul = u1 * l1 + v1 * l2 + w1 * l3;
        const R um = u1 * m1 + v1 * m2 + w1 * m3;
        const R V2 = (u1 * u1 + v1 * v1 + w1 * w1) * R(0.5);
        const R KK = (R(ph.gamma) - R(1)) / (c1 * c1);
        const R KK1 = KK * R(0.5);
        const R X1 = R(1) / (R(2) * c1);
        const R L[5][5] = {{R(1) - KK * V2, KK * u1, KK * v1, KK * w1, -KK},
                           {-ul, l1, l2, l3, R(0)},
                           {-um, m1, m2, m3, R(0)},
                           {KK1 * V2 + X1 * un, -X1 * n1 - KK1 * u1, -X1 * n2 - KK1 * v1, -X1 * n3 - KK1 * w1, KK1},
                           {KK1 * V2 - X1 * un, X1 * n1 - KK1 * u1, X1 * n2 - KK1 * v1, X1 * n3 - KK1 * w1, KK1}};
        // projection of one stencil point (:256-260 / :266-270), row r
        auto proj_row = [&](int r, int vb, int q) -> R {
          const R f0 = W(vb, q), f1 = W(vb + 1, q), f2 = W(vb + 2, q), f3 = W(vb + 3, q);
          if (r == 1 || r == 2) return L[r][0] * f0 + L[r][1] * f1 + L[r][2] * f2 + L[r][3] * f3;
          return L[r][0] * f0 + L[r][1] * f1 + L[r][2] * f2 + L[r][3] * f3 + L[r][4] * W(vb + 4, q);
        };
#endif
        R h0[5];
        if (SCHEME == SCH_OMP6 && inner) {
          // OMP6, interior face: the linear part of hh_OMP6P/M (OCFD_Schemes_1.f90:211,244) is
          // accumulated while the stencil is projected point by point, in the
          // reference's term order; only v(-1..1) (F+) / v(0..2) (F-) are kept for
          // the monotonicity test, the two outer values are recomputed in the
          // (rare) limiter branch.
          const R oa[8] = {R(Omp6C::a1), R(Omp6C::a2), R(Omp6C::a3), R(Omp6C::a4),
                           R(Omp6C::a5), R(Omp6C::a6), R(Omp6C::a7), R(Omp6C::a8)};
          const R kap = R(Omp6C::kappa), ep = R(Omp6C::ep);
#if OCFD_FEWER_DIVS
          // production build: the scheme is linear up to the limiter, so a face
          // none of whose components is limited is the stencil sum G in physical
          // space, with no projection back; the limiter's changes are added to it
          // by the faces that have any.  The monotonicity test
          //   (mid - v0)(mid - mp) >= ep,  mp = v0 + minmod(v1 - v0, kappa (v0 - v-1))
          // needs only three differences of points, projected: G - F0, F1 - F0 and
          // F0 - F-1, in rows scaled by c^2 (the bound by c^4), so that no face
          // divides.  Per face and direction 330 instead of 470 FP64 operations.
          const R c2 = xmul(c1, c1);
          const R e0 = xmul(ep, xmul(c2, c2));
          const R et[5] = {e0, ep, ep, xmul(R(4), e0), xmul(R(4), e0)};
          R H[5];
          if constexpr (OCFD_F32X2 && sizeof(R) == 4 && PS == 1) {
            // production FP32, sweeps without point records (z): the F+ and F-
            // sides below in the two lanes of packed operations -- step s takes
            // F+(7 - s) and F-(s), both with oa[s]; every lane operation is the
            // scalar block's own explicitly rounded operation, so the results are
            // the same bits
            const F2 m1 = f2(-1.0f), kap2 = f2(float(kap));
            F2 G[5], B[5], M[5];
#pragma unroll
            for (int s = 0; s <= 7; s++) {
              F2 f[5];
#pragma unroll
              for (int v = 0; v < 5; v++) f[v] = f2(float(W(v, 7 - s)), float(W(5 + v, s)));
              const F2 c = f2(float(oa[s]));
#pragma unroll
              for (int v = 0; v < 5; v++) G[v] = s == 0 ? mul2(c, f[v]) : fma2(c, f[v], G[v]);
              if (s == 3) {
#pragma unroll
                for (int v = 0; v < 5; v++) B[v] = f[v];
              }
              if (s == 4 || s == 5) {
                F2 D[5], P[5];
#pragma unroll
                for (int v = 0; v < 5; v++) D[v] = fma2(m1, f[v], B[v]);
                char_proj2(cb, D, g1, c2, V2, P);
#pragma unroll
                for (int r = 0; r < 5; r++) {
                  if (s == 4) {
                    M[r] = P[r];
                    B[r] = f[r];
                  } else {
                    const F2 t2 = mul2(kap2, P[r]);
                    M[r] = f2(minmod2(M[r].v.x, t2.v.x), minmod2(M[r].v.y, t2.v.y));
                  }
                }
              }
            }
            F2 D[5], P[5];
#pragma unroll
            for (int v = 0; v < 5; v++) D[v] = fma2(m1, B[v], G[v]);
            char_proj2(cb, D, g1, c2, V2, P);
            unsigned fP = 0, fM = 0;
            R pP[5], pM[5];
#pragma unroll
            for (int r = 0; r < 5; r++) {
              const F2 tt = mul2(P[r], fma2(m1, M[r], P[r]));
              fP |= (tt.v.x >= float(et[r]) ? 1u : 0u) << r;
              fM |= (tt.v.y >= float(et[r]) ? 1u : 0u) << r;
              pP[r] = P[r].v.x;
              pM[r] = P[r].v.y;
              H[r] = xadd(G[r].v.x, G[r].v.y);
            }
            if (fP) djP = push(fP, pP, 0, t);
            if (fM) djM = push(fM, pM, 1, t);
            dfl = fP | (fM << 5);
          } else {
            // one side: stencil points in the order of oa (F+: 7..0, F-: 0..7);
            // step 4 is the upwind point v0, step 3 v1, step 5 v-1
            auto side_sum = [&](const int side, R* G, R* P) -> unsigned {
              R B[5], M[5];
#pragma unroll
              for (int s = 0; s <= 7; s++) {
                R f[5];
                load5(5 * side, side ? s : 7 - s, f);
#pragma unroll
                for (int v = 0; v < 5; v++) G[v] = s == 0 ? xmul(oa[0], f[v]) : xfma(oa[s], f[v], G[v]);
                if (s == 3) {
#pragma unroll
                  for (int v = 0; v < 5; v++) B[v] = f[v];
                }
                if (s == 4 || s == 5) {
                  R D[5];
#pragma unroll
                  for (int v = 0; v < 5; v++) D[v] = xadd(B[v], -f[v]);
                  cb.proj_scaled(D, g1, c2, V2, P);
#pragma unroll
                  for (int r = 0; r < 5; r++) {
                    if (s == 4) {
                      M[r] = P[r];
                      B[r] = f[r];
                    } else {
                      M[r] = minmod2(M[r], xmul(kap, P[r]));
                    }
                  }
                }
              }
              R D[5];
#pragma unroll
              for (int v = 0; v < 5; v++) D[v] = xadd(G[v], -B[v]);
              cb.proj_scaled(D, g1, c2, V2, P);
              unsigned fl = 0;
#pragma unroll
              for (int r = 0; r < 5; r++) fl |= (xmul(P[r], xadd(P[r], -M[r])) >= et[r] ? 1u : 0u) << r;
              return fl;
            };
            R P[5], G[5];
            const unsigned fP = side_sum(0, H, P);
            if (fP) djP = push(fP, P, 0, t);
            const unsigned fM = side_sum(1, G, P);
            if (fM) djM = push(fM, P, 1, t);
            dfl = fP | (fM << 5);
#pragma unroll
            for (int v = 0; v < 5; v++) H[v] = xadd(H[v], G[v]);
          }
          if (dfl == 0) {
            hf_store5(out, fo, a.fs, H);
          } else {
            dfo[0] = fo;
#pragma unroll
            for (int v = 0; v < 5; v++) dH[v] = H[v];
          }
          continue;
#else
          {
            R mid[5], vm1[5], v0[5], vp1[5];
#pragma unroll
            for (int s = 4; s >= -3; s--) {
              const int q = s + 3;
              const R f0 = W(0, q), f1 = W(1, q), f2 = W(2, q), f3 = W(3, q), f4 = W(4, q);
              R c[5];
              c[0] = L[0][0] * f0 + L[0][1] * f1 + L[0][2] * f2 + L[0][3] * f3 + L[0][4] * f4;
              c[1] = L[1][0] * f0 + L[1][1] * f1 + L[1][2] * f2 + L[1][3] * f3;
              c[2] = L[2][0] * f0 + L[2][1] * f1 + L[2][2] * f2 + L[2][3] * f3;
              c[3] = L[3][0] * f0 + L[3][1] * f1 + L[3][2] * f2 + L[3][3] * f3 + L[3][4] * f4;
              c[4] = L[4][0] * f0 + L[4][1] * f1 + L[4][2] * f2 + L[4][3] * f3 + L[4][4] * f4;
#pragma unroll
              for (int r = 0; r < 5; r++) {
                mid[r] = (s == 4) ? oa[0] * c[r] : mid[r] + oa[4 - s] * c[r];
                if (s == -1) vm1[r] = c[r];
                if (s == 0) v0[r] = c[r];
                if (s == 1) vp1[r] = c[r];
              }
            }
#pragma unroll
            for (int r = 0; r < 5; r++) {
              const R mp = v0[r] + minmod2((vp1[r] - v0[r]), kap * (v0[r] - vm1[r]));
              if ((mid[r] - v0[r]) * (mid[r] - mp) >= ep) {
                const R vm2 = proj_row(r, 0, 1), vp2 = proj_row(r, 0, 5);
                mid[r] = omp6_limit(mid[r], vm2, vm1[r], v0[r], vp1[r], vp2, vm1[r]);
              }
              h0[r] = mid[r];
            }
          }
          {
            R mid[5], v0[5], v1[5], v2[5];
#pragma unroll
            for (int s = -3; s <= 4; s++) {
              const int q = s + 3;
              const R f0 = W(5, q), f1 = W(6, q), f2 = W(7, q), f3 = W(8, q), f4 = W(9, q);
              R c[5];
              c[0] = L[0][0] * f0 + L[0][1] * f1 + L[0][2] * f2 + L[0][3] * f3 + L[0][4] * f4;
              c[1] = L[1][0] * f0 + L[1][1] * f1 + L[1][2] * f2 + L[1][3] * f3;
              c[2] = L[2][0] * f0 + L[2][1] * f1 + L[2][2] * f2 + L[2][3] * f3;
              c[3] = L[3][0] * f0 + L[3][1] * f1 + L[3][2] * f2 + L[3][3] * f3 + L[3][4] * f4;
              c[4] = L[4][0] * f0 + L[4][1] * f1 + L[4][2] * f2 + L[4][3] * f3 + L[4][4] * f4;
#pragma unroll
              for (int r = 0; r < 5; r++) {
                mid[r] = (s == -3) ? oa[0] * c[r] : mid[r] + oa[s + 3] * c[r];
                if (s == 0) v0[r] = c[r];
                if (s == 1) v1[r] = c[r];
                if (s == 2) v2[r] = c[r];
              }
            }
#pragma unroll
            for (int r = 0; r < 5; r++) {
              const R mp = v1[r] + minmod2((v0[r] - v1[r]), kap * (v1[r] - v2[r]));
              if ((mid[r] - v1[r]) * (mid[r] - mp) >= ep) {
                const R v3 = proj_row(r, 5, 6), vm1 = proj_row(r, 5, 2);
                mid[r] = omp6_limit(mid[r], v3, v2[r], v1[r], v0[r], vm1, v0[r]);
              }
              h0[r] = h0[r] + mid[r];
            }
          }
#endif
        } else {
#if OCFD_FEWER_DIVS
          const R rc = R(1) / c1;
          const R KK = xmul(g1, xmul(rc, rc));
          const R KK1 = xmul(KK, R(0.5));
          const R X1 = xmul(R(0.5), rc);
          if (WDIFF && (ALLIN || inner)) {
            // WENO face: the schemes see only differences of the stencil, so the
            // differences are projected (six a side instead of seven points, and
            // 30 live values instead of 40), and what comes back from
            // characteristic space is added to F+(v0) + F-(v1)
            R hb[5], wsum[5];
#pragma unroll
            for (int side = 0; side < 2; side++) {
              R e[5][6], f[5], fl[5], c[5];
#pragma unroll
              for (int k = 0; k < 7; k++) {  // offsets -3..3 (F+), 4..-2 (F- mirrored)
                load5(5 * side, side ? 7 - k : k, f);
                if (k > 0) {
                  R dfl[5];
#pragma unroll
                  for (int v = 0; v < 5; v++) dfl[v] = xsub(f[v], fl[v]);
                  cb.proj(dfl, KK, KK1, X1, V2, c);
#pragma unroll
                  for (int r = 0; r < 5; r++) e[r][k - 1] = c[r];
                }
#pragma unroll
                for (int v = 0; v < 5; v++) {
                  if (k == 3) hb[v] = side ? xadd(hb[v], f[v]) : f[v];
                  fl[v] = f[v];
                }
              }
#pragma unroll
              for (int r = 0; r < 5; r++) {
                const R h = weno_diff<SCHEME>(e[r]);
                wsum[r] = side ? xadd(wsum[r], h) : h;
              }
            }
            cb.back(wsum, hh, R(ph.inv_gm1));
#pragma unroll
            for (int v = 0; v < 5; v++) hh[v] = xadd(hb[v], hh[v]);
            hf_store5(out, fo, a.fs, hh);
            continue;
          }
          hslot[0] = list_face(t, false);  // a face of the boundary closures
          dfo[0] = fo;
          continue;
#else
          // ---- F+ projected onto the characteristic variables (:254-261), reconstructed
          {
            R q[5][8];
            constexpr int LO = Stencil<SCHEME>::PLO, HI = Stencil<SCHEME>::PHI;
#pragma unroll
            for (int s = -3; s <= 4; s++) {
#pragma unroll
              for (int r = 0; r < 5; r++) q[r][s + 3] = (s < LO || s > HI) ? R(0) : proj_row(r, 0, s + 3);
            }
            if (ALLIN || inner1) {
#pragma unroll
              for (int r = 0; r < 5; r++) h0[r] = schemeP<SCHEME>(q[r] + 3, U, ihy);
            } else {
#pragma unroll
              for (int r = 0; r < 5; r++) h0[r] = ch_flux1_bnd(q[r] + 3, g, nn, face_ends(ph, DIR));
            }
          }
          // ---- F- (:264-271)
          {
            R q[5][8];
            constexpr int LO = Stencil<SCHEME>::MLO, HI = Stencil<SCHEME>::MHI;
#pragma unroll
            for (int s = -3; s <= 4; s++) {
#pragma unroll
              for (int r = 0; r < 5; r++) q[r][s + 3] = (s < LO || s > HI) ? R(0) : proj_row(r, 5, s + 3);
            }
            if (ALLIN || inner2) {
#pragma unroll
              for (int r = 0; r < 5; r++) h0[r] = h0[r] + schemeM<SCHEME>(q[r] + 3, U, ihy);
            } else {
#pragma unroll
              for (int r = 0; r < 5; r++) h0[r] = h0[r] + ch_flux2_bnd(q[r] + 3, g, nn, face_ends(ph, DIR));
            }
          }
#endif
        }
        // ---- back to physical space, hh = R h0 (:284-288); R = S^-1 (:244-248)
#if !OCFD_FEWER_DIVS
        const R H = V2 + R(1) / KK;
        hh[0] = h0[0] + h0[3] + h0[4];
        hh[1] = u1 * h0[0] + l1 * h0[1] + m1 * h0[2] + (u1 - c1 * n1) * h0[3] + (u1 + c1 * n1) * h0[4];
        hh[2] = v1 * h0[0] + l2 * h0[1] + m2 * h0[2] + (v1 - c1 * n2) * h0[3] + (v1 + c1 * n2) * h0[4];
        hh[3] = w1 * h0[0] + l3 * h0[1] + m3 * h0[2] + (w1 - c1 * n3) * h0[3] + (w1 + c1 * n3) * h0[4];
        hh[4] = V2 * h0[0] + ul * h0[1] + um * h0[2] + (H - c1 * un) * h0[3] + (H + c1 * un) * h0[4];
#endif
      }
    }
    hf_store5(out, fo, a.fs, hh);
  }
  if constexpr (LIST) {
    __syncthreads();
    const int n7 = ln[0], nj = n7 + ln[1];
    const R gm1 = xadd(R(ph.gamma), R(-1));
    // Hybrid faces of the characteristic form.  A list longer than one round of one-row
    // items: an item is rows 0, 3, 4 or rows 1, 2 of a face, because one row an item reads
    // the window five times and a tile with many WENO faces is then bound by shared memory.
    // The three sweeps of 128x120x112 in ms per step, one row an item / grouped: noise
    // everywhere (every face listed) 3.17 / 2.04, noise at 3% of the points 1.19 / 1.10; a
    // short list has too few grouped items (noise at 1%: 0.86 / 0.93).
    constexpr bool GROUPS = CHAR && HQ && ALLIN;
    const bool group = GROUPS && 5 * nj > NT;
    if (GROUPS && group) {
      for (int e = threadIdx.x; e < 2 * nj; e += NT) {
        const bool lm = e >= nj;  // rows 1, 2
        const int x = lm ? e - nj : e, slot = x < n7 ? x : NP * TF - 1 - (x - n7);
        const auto win = window(ltag[slot]);
        auto mean = [&](int var) -> R { return xmul(xadd(win(var, 3), win(var, 4)), R(0.5)); };
        const int row[3] = {lm ? 1 : 0, lm ? 2 : 3, 4};
        R L[3][5];
        {
          CharBasis<DIR, AXS, R> cb;
          cb.init(mean(10), mean(11), mean(12), mean(13), AXS ? R(0) : mean(14), AXS ? R(0) : mean(15),
                  AXS ? R(0) : mean(16));
          const R rc = xrcp(cb.c), KK = xmul(gm1, xmul(rc, rc)), X1 = xmul(R(0.5), rc), V2 = cb.V2();
#pragma unroll
          for (int r = 0; r < 3; r++) cb.row(row[r], KK, X1, V2, L[r]);
        }
        R h[3];
#pragma unroll 1
        for (int side = 0; side < 2; side++) {
          R d[3][6], last[3];
#pragma unroll
          for (int k = 0; k < 7; k++) {  // F+ at offsets -3..3, F- mirrored (4..-2)
            R f[5];
#pragma unroll
            for (int v = 0; v < 5; v++) f[v] = win(5 * side + v, side ? 7 - k : k);
#pragma unroll
            for (int r = 0; r < 3; r++) {
              const R y =
                  xfma(L[r][4], f[4], xfma(L[r][3], f[3], xfma(L[r][2], f[2], xfma(L[r][1], f[1], xmul(L[r][0], f[0])))));
              if (k > 0) d[r][k - 1] = xsub(y, last[r]);
              last[r] = y;
            }
          }
#pragma unroll
          for (int r = 0; r < 3; r++) {
            if (r == 2 && lm) break;
            const R y = x < n7 ? weno_diff<SCH_WENO7>(d[r]) : weno_diff<SCH_WENO5>(d[r]);
            h[r] = side ? xadd(h[r], y) : y;
          }
        }
        lv[row[0] * NP * TF + slot] = h[0];
        lv[row[1] * NP * TF + slot] = h[1];
        if (!lm) lv[4 * NP * TF + slot] = h[2];
      }
    }
    for (int e = threadIdx.x; !group && e < 5 * nj; e += NT) {
      const int m = e / nj, x = e - m * nj;
      const int slot = x < n7 ? x : NP * TF - 1 - (x - n7);
      const int t = ltag[slot];
      const auto win = window(t);
      int f, p;
      face_of(t, f, p);
      const int g = g0 + f;
      R vp[8], vm[8];  // F+ at offsets -3..4, F- mirrored (4..-3)
      if constexpr (CHAR) {
        auto mean = [&](int var) -> R { return xmul(xadd(win(var, 3), win(var, 4)), R(0.5)); };
        CharBasis<DIR, AXS, R> cb;
        cb.init(mean(10), mean(11), mean(12), mean(13), AXS ? R(0) : mean(14), AXS ? R(0) : mean(15),
                AXS ? R(0) : mean(16));
        const R rc = xrcp(cb.c);
        R L[5];
        cb.row(m, xmul(gm1, xmul(rc, rc)), xmul(R(0.5), rc), cb.V2(), L);
        auto value = [&](int v, int q) -> R {
          return xfma(L[4], win(v + 4, q),
                      xfma(L[3], win(v + 3, q), xfma(L[2], win(v + 2, q), xfma(L[1], win(v + 1, q), xmul(L[0], win(v, q))))));
        };
#pragma unroll
        for (int k = 0; k < (ALLIN ? 7 : 8); k++) {
          vp[k] = value(0, k);
          vm[k] = value(5, 7 - k);
        }
        bool inner1 = true, inner2 = true;
        if constexpr (!ALLIN) {
          const FaceEnds fe = face_ends(ph, DIR);
          inner1 = (fe.bi0 == 0 || g > -fe.ka1 || fe.sb0 == -1) && (fe.bi1 == 0 || g <= nn - fe.kb1 || fe.sb1 == -1);
          inner2 = (fe.bi0 == 0 || g > -fe.ka2 || fe.sb0 == -1) && (fe.bi1 == 0 || g <= nn - fe.kb2 || fe.sb1 == -1);
        }
        R h;
        if (!ALLIN && !(inner1 && inner2)) {
          // boundary closure (only the WENO stencils reach further on one side)
          const FaceEnds fe = face_ends(ph, DIR);
          const R* const none = nullptr;
          R fw[8];
#pragma unroll
          for (int k = 0; k < 8; k++) fw[k] = vm[7 - k];
          h = (WDIFF && inner1) ? schemeP<SCHEME>(vp + 3, none, 0) : ch_flux1_bnd(vp + 3, g, nn, fe);
          h = xadd(xadd(h, -vp[3]),
                   xadd((WDIFF && inner2) ? schemeM<SCHEME>(fw + 3, none, 0) : ch_flux2_bnd(fw + 3, g, nn, fe), -vm[3]));
        } else {
          h = x < n7 ? weno_pair<SCH_WENO7>(vp, vm) : weno_pair<SCH_WENO5>(vp, vm);
        }
        lv[m * NP * TF + slot] = h;
      } else {
#pragma unroll
        for (int k = 0; k < 7; k++) {
          vp[k] = win(m, k);
          vm[k] = win(5 + m, 7 - k);
        }
        const R h = x < n7 ? weno_pair<SCH_WENO7>(vp, vm) : weno_pair<SCH_WENO5>(vp, vm);
        int i, j, k;
        pencil(p, i, j, k);
        out[hf_at(G.face(DIR, g, DIR == 0 ? g : i, DIR == 1 ? g : j, DIR == 2 ? g : k), a.fs, m)] =
            xadd(xadd(vp[3], vm[3]), h);
      }
    }
    if (CHAR && nj > 0) {
      __syncthreads();
#pragma unroll
      for (int n = 0; n < FPT; n++) {
        if (hslot[n] < 0) continue;
        const auto win = window(ltag[hslot[n]]);
        auto mean = [&](int var) -> R { return xmul(xadd(win(var, 3), win(var, 4)), R(0.5)); };
        CharBasis<DIR, AXS, R> cb;
        cb.init(mean(10), mean(11), mean(12), mean(13), AXS ? R(0) : mean(14), AXS ? R(0) : mean(15),
                AXS ? R(0) : mean(16));
        R ch[5], hh[5];
#pragma unroll
        for (int r = 0; r < 5; r++) ch[r] = lv[r * NP * TF + hslot[n]];
        cb.back(ch, hh, R(ph.inv_gm1));
#pragma unroll
        for (int r = 0; r < 5; r++) hh[r] = xadd(xadd(win(r, 3), win(5 + r, 4)), hh[r]);
        hf_store5(out, dfo[n], a.fs, hh);
      }
    }
  }
  if constexpr (DEFER) {
    __syncthreads();
    const int nj = min(*jn, JC);
    if (nj == 0) return;
    const R gm1 = xadd(R(ph.gamma), R(-1));
    for (int e = threadIdx.x; e < nj; e += NT) {
      const int tag = jtag[e];
      jv[e] = lim_eval<DIR, AXS>(window(tag >> 4), (tag >> 1) & 7, tag & 1, jv[e], gm1);
    }
    __syncthreads();
    if (dfl == 0) return;
    // the limited components' changes, projected back and added to the unlimited
    // flux (OCFD_inviscous_character.f90:284-288)
    const auto win = window(threadIdx.x);
    auto mean = [&](int var) -> R { return xmul(xadd(win(var, 3), win(var, 4)), R(0.5)); };
    CharBasis<DIR, AXS, R> cb;
    cb.init(mean(10), mean(11), mean(12), mean(13), AXS ? R(0) : mean(14), AXS ? R(0) : mean(15),
            AXS ? R(0) : mean(16));
    R ch[5], hh[5];
#pragma unroll
    for (int r = 0; r < 5; r++) {
      ch[r] = R(0);
      if ((dfl >> r) & 1u) ch[r] = jv[djP++];
      if ((dfl >> (5 + r)) & 1u) ch[r] = xadd(ch[r], jv[djM++]);
    }
    const R rc2 = xrcp(xmul(cb.c, cb.c));  // proj_scaled's scaling undone
    ch[0] = xmul(ch[0], rc2);
    ch[3] = xmul(ch[3], xmul(R(0.5), rc2));
    ch[4] = xmul(ch[4], xmul(R(0.5), rc2));
    cb.back(ch, hh, R(ph.inv_gm1));
#pragma unroll
    for (int r = 0; r < 5; r++) hh[r] = xadd(dH[r], hh[r]);
    hf_store5(out, dfo[0], a.fs, hh);
  }
}

// The body of every sweep: the mixed-precision hybrid keeps its own arithmetic
// (ocfd_face_values.cuh).
template <int DIR, bool CHAR, int SCHEME, bool ALLIN, int NP, int TF, typename R, typename S, bool TMA = false,
          bool AXS = false, int FPT = 1>
__device__ __forceinline__ void face_body(const FaceArgs<S>& a, const int bx, const int by, const int bz, R* sm,
                                          const S* tile = nullptr, int toff = 0, R* qbase = nullptr,
                                          int* qcount = nullptr) {
  if constexpr (face_on_values<SCHEME, R>())
    face_body_values<DIR, CHAR, ALLIN, NP, TF, R, S, TMA, AXS>(a, bx, by, bz, sm, tile, toff, qbase, qcount);
  else
    face_body_main<DIR, CHAR, SCHEME, ALLIN, NP, TF, R, S, TMA, AXS, FPT>(a, bx, by, bz, sm, tile, toff, qbase,
                                                                         qcount);
}

template <int DIR, bool CHAR, int SCHEME, int NP, int TF, typename R, bool AXS = false, int FPT = 1>
constexpr size_t face_smem_points() {
  constexpr bool ax = AXS && !face_on_values<SCHEME, R>();
  return (size_t)face_nvar<CHAR, ax, (FPT > 1 ? 1 : face_ps<DIR, CHAR, R>())>() * face_points<FPT, NP, TF>() *
         sizeof(R);
}
template <int DIR, bool CHAR, int SCHEME, int NP, int TF, typename R, bool AXS = false, int FPT = 1, bool ALLIN = true>
constexpr size_t face_smem() {
  return face_smem_points<DIR, CHAR, SCHEME, NP, TF, R, AXS, FPT>() + face_queue<CHAR, SCHEME, ALLIN, NP * TF, R>();
}
// TMA sweeps: the queue shares memory with the staged input tiles
// (read only in phase 1, the queue is used after phase 1's barrier); its entry
// count, written before phase 1, lies past both.  An axis-aligned sweep stages
// six arrays (d, u, v, w, T and its direction's metric), the others eight.
template <int DIR, bool CHAR, int SCHEME, int NP, int TF, typename R, typename S, bool AXS, int FPT, bool ALLIN>
struct FaceTmaSmem {
  using B = TmaBox<DIR, NP, TF, S, FPT>;
  static constexpr size_t TILE = (AXS ? 6 : 8) * (size_t)B::SLOT;
  static constexpr size_t QB = face_queue<CHAR, SCHEME, ALLIN, NP * TF, R>();
  static constexpr bool QUEUE = QB != 0;
  static constexpr size_t COUNT_AT = TILE > QB ? TILE : QB;
  static constexpr size_t UNION = QUEUE ? COUNT_AT + 128 : TILE;  // before the staged points
  static constexpr size_t BYTES = 128 + UNION + face_smem_points<DIR, CHAR, SCHEME, NP, TF, R, AXS, FPT>();
};

// Minimum resident blocks per SM.  FP64: two (<= 128 registers) measured
// faster than one.  FP32: four (<= 64 registers) -- 17% faster than two on the
// characteristic OMP6 sweeps at 256^3 despite a few spilled registers, equal on
// the flux-vector sweeps.
#ifndef OCFD_FACE32_MINB
#define OCFD_FACE32_MINB 4
#endif
#define OCFD_FACE_MINB (sizeof(R) == 8 ? 2 : OCFD_FACE32_MINB)
// threads and minimum resident blocks of the single-instance sweeps
#define OCFD_FACE_NT (FaceTile<DIR, CHAR, SCHEME, R, ALLIN>::NT)
#ifndef OCFD_FACE64_MINBPAIR
#define OCFD_FACE64_MINBPAIR (CHAR ? 4 : 5)  // FP64, two faces a thread: blocks of 128.  Flux-vector
                                            // form 5 (four: 0.5% slower); the shared memory of
                                            // the characteristic form allows four
#endif
#ifndef OCFD_FACE64_MINB128
#define OCFD_FACE64_MINB128 4  // FP64, 128-thread tiles: 4 blocks (128 registers); 5 (96
                               // registers) measured 2% faster on x, 8% slower on y and z
#endif
#ifndef OCFD_FACE64_MINB128_AX
#define OCFD_FACE64_MINB128_AX 6  // the axis-aligned variants (80 registers; five blocks measured 2% slower)
#endif
#define OCFD_FACE_BOUNDS                                                                                     \
  __launch_bounds__(OCFD_FACE_NT,                                                                            \
                    FaceTile<DIR, CHAR, SCHEME, R, ALLIN>::FPT > 1 ? OCFD_FACE64_MINBPAIR                          \
                    : (OCFD_FACE_NT == 128 && sizeof(R) == 8) ? (AXS ? OCFD_FACE64_MINB128_AX : OCFD_FACE64_MINB128) \
                                                              : OCFD_FACE_MINB * 256 / OCFD_FACE_NT)
template <int DIR, bool CHAR, int SCHEME, bool ALLIN, typename R, typename S, bool AXS = false>
__global__ void OCFD_FACE_BOUNDS k_face(FaceArgs<S> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using T = FaceTile<DIR, CHAR, SCHEME, R, ALLIN>;
  face_body<DIR, CHAR, SCHEME, ALLIN, T::NP, T::TF, R, S, false, AXS, T::FPT>(a, blockIdx.x, blockIdx.y, blockIdx.z, reinterpret_cast<R*>(smem_raw));
}

// Batched launch: the blocks of all instances in one 1-D grid; each block finds
// its instance and its block coordinates from the batch table.  Periodic
// instances only (ALLIN).
template <int DIR, bool CHAR, int SCHEME, int V, typename R, typename S>
__global__ void __launch_bounds__(256, OCFD_FACE_MINB) k_face_batch(BatchTab<FaceArgs<S>> b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) FaceArgs<S> sa;
  int bx, by, bz;
  const int q = batch_locate(b, blockIdx.x, bx, by, bz);
  const FaceArgs<S>& A = batch_args(b, q, &sa);
  // the member's own sweep variant, as its single-instance launch would choose
  // it (batched and single results are the same bits)
  if (OCFD_FEWER_DIVS && axis_aligned<DIR>(A.ph.metzero))
    face_body<DIR, CHAR, SCHEME, true, FaceTileV<DIR, V>::NP, FaceTileV<DIR, V>::TF, R, S, false,
              OCFD_FEWER_DIVS != 0>(A, bx, by, bz, reinterpret_cast<R*>(smem_raw));
  else
    face_body<DIR, CHAR, SCHEME, true, FaceTileV<DIR, V>::NP, FaceTileV<DIR, V>::TF, R, S>(
        A, bx, by, bz, reinterpret_cast<R*>(smem_raw));
}

// One block of a sweep with its input tiles staged by TMA (the arithmetic is
// that of k_face).  ALLIN: a periodic direction; otherwise the sweep includes
// the boundary closures, and tile points past the haloed array (read as zeros
// by the copy) are not used.
template <int DIR, bool CHAR, int SCHEME, typename R, typename S, bool AXS, bool ALLIN>
__device__ __forceinline__ void face_tma_block(const FaceArgs<S>& a, const FaceTmaMaps& tm, const int bx, const int by,
                                               const int bz, unsigned char* smem_raw) {
  using T = FaceTile<DIR, CHAR, SCHEME, R, ALLIN>;
  constexpr int NP = T::NP, TF = T::TF;
  using B = TmaBox<DIR, NP, TF, S, T::FPT>;
  __shared__ __align__(8) uint64_t bar;
  // TMA destinations start on 128-byte boundaries (128 bytes of the launch's
  // dynamic shared memory are reserved for this rounding)
  unsigned char* base = smem_raw + ((128 - (smem_u32(smem_raw) & 127u)) & 127u);
  using L = FaceTmaSmem<DIR, CHAR, SCHEME, NP, TF, R, S, AXS, T::FPT, ALLIN>;
  S* tile = reinterpret_cast<S*>(base);
  R* sm = reinterpret_cast<R*>(base + L::UNION);
  R* qbase = L::QUEUE ? reinterpret_cast<R*>(base) : nullptr;
  int* qcount = reinterpret_cast<int*>(base + L::COUNT_AT);
  const int g0 = a.fbeg + (DIR == 0 ? bx : by) * TF;  // first face; its stencil starts at g0 - 3
  const int pbase = (DIR == 0 ? by : bx) * NP;
  // haloed (0-based) coordinates of the tile's first element: index + LAP - 1
  const int x0 = DIR == 0 ? g0 : pbase + 4;
  const int toff = x0 % B::A;
  const int c0 = x0 - toff;
  const int c1 = DIR == 0 ? pbase + 4 : (DIR == 1 ? g0 : bz + 4);
  const int c2 = DIR == 2 ? g0 : bz + 4;
  // once a block of this instance has given up on its tile copies (error 4),
  // the launch's results are invalid: later blocks issue no copies and leave
  if (__syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile const int*>(a.err) == 4)) return;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int m0 = 13 + 3 * DIR;
    bool need[8];
    uint32_t bytes = 0;
    for (int q = 0; q < 8; q++) {
      need[q] = q < 5 || (AXS ? q == 5 + DIR : !((a.ph.metzero >> (m0 + q - 5)) & 1u));
      if (need[q]) bytes += B::BYTES;
    }
    mbar_arrive_expect_tx(&bar, bytes + (uint32_t)a.test_tx);
    if constexpr (sizeof(S) == 4) {
      // FP32: d, then u,v,w,T interleaved (one 4-D copy filling slots 1-4)
      tma_load_3d(tile, &tm.m[0], c0, c1, c2, &bar);
      tma_load_4d(tile + B::SLOT_ELEMS, &tm.m[1], 0, c0, c1, c2, &bar);
      for (int q = 5; q < 8; q++)
        if (need[q]) tma_load_3d(tile + (AXS ? 5 : q) * B::SLOT_ELEMS, &tm.m[q], c0, c1, c2, &bar);
    } else {
      for (int q = 0; q < 8; q++)
        if (need[q]) tma_load_3d(tile + (AXS && q > 5 ? 5 : q) * B::SLOT_ELEMS, &tm.m[q], c0, c1, c2, &bar);
    }
  }
  // bounded wait (about a second); a block that gives up records the error and
  // waits once more, again bounded, for its copies before leaving
  bool done = mbar_wait_bounded(&bar, 0, 1u << 20);
  if (__syncthreads_or(!done)) {
    if (threadIdx.x == 0) {
      atomicExch(a.err, 4);
      mbar_wait_bounded(&bar, 0, 1u << 20);
    }
    return;
  }
  face_body<DIR, CHAR, SCHEME, ALLIN, NP, TF, R, S, true, AXS, T::FPT>(a, bx, by, bz, sm, tile, toff, qbase, qcount);
}
template <int DIR, bool CHAR, int SCHEME, typename R, typename S, bool AXS = false, bool ALLIN = true>
__global__ void OCFD_FACE_BOUNDS k_face_tma(FaceArgs<S> a, const __grid_constant__ FaceTmaMaps tm) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  face_tma_block<DIR, CHAR, SCHEME, R, S, AXS, ALLIN>(a, tm, blockIdx.x, blockIdx.y, blockIdx.z, smem_raw);
}

// ---------------------------------------------------------------------------
template <int DIR, bool CHAR, int SCHEME, bool ALLIN, typename R, typename S, bool AXS = false>
static cudaError_t launch_face_t(const FaceArgs<S>& a, cudaStream_t st) {
  using T = FaceTile<DIR, CHAR, SCHEME, R, ALLIN>;
  constexpr int NP = T::NP, TF = T::TF;
  constexpr size_t smem = face_smem<DIR, CHAR, SCHEME, NP, TF, R, AXS, T::FPT, ALLIN>();
  auto kern = k_face<DIR, CHAR, SCHEME, ALLIN, R, S, AXS>;
  if (a.g.n == 0) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  kern<<<face_grid<DIR, NP, TF>(a), T::NT, smem, st>>>(a);
  return cudaGetLastError();
}

// Batched face sweep.  nblocks == 0 asks for the shared-memory attribute to be
// set instead of a launch; the host fills b from face_batch_dims().
template <int DIR, bool CHAR, int SCHEME, int V, typename R, typename S>
static cudaError_t launch_face_batch_t(const BatchTab<FaceArgs<S>>& b, int nblocks, cudaStream_t st) {
  constexpr int NP = FaceTileV<DIR, V>::NP, TF = FaceTileV<DIR, V>::TF;
  constexpr size_t smem = face_smem<DIR, CHAR, SCHEME, NP, TF, R>();
  auto kern = k_face_batch<DIR, CHAR, SCHEME, V, R, S>;
  if (nblocks == 0) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  kern<<<nblocks, NP * TF, smem, st>>>(b);
  return cudaGetLastError();
}

template <typename R, typename S>
cudaError_t launch_face_batch(int dir, bool chr, int scheme, int variant, const BatchTab<FaceArgs<S>>& b,
                              int nblocks, cudaStream_t st) {
#define OCFD_FB_CASE(D, C, SC)                                                     \
  if (dir == D && chr == C && scheme == SC)                                        \
    return variant ? launch_face_batch_t<D, C, SC, 1, R, S>(b, nblocks, st)        \
                   : launch_face_batch_t<D, C, SC, 0, R, S>(b, nblocks, st);
#define OCFD_FB_SCHEMES(D, C) \
  OCFD_FB_CASE(D, C, SCH_WENO5) \
  OCFD_FB_CASE(D, C, SCH_WENO7) \
  OCFD_FB_CASE(D, C, SCH_OMP6)  \
  OCFD_FB_CASE(D, C, SCH_UD7L)  \
  OCFD_FB_CASE(D, C, SCH_HYBRID)
  OCFD_FB_SCHEMES(0, false)
  OCFD_FB_SCHEMES(1, false)
  OCFD_FB_SCHEMES(2, false)
  OCFD_FB_SCHEMES(0, true)
  OCFD_FB_SCHEMES(1, true)
  OCFD_FB_SCHEMES(2, true)
#undef OCFD_FB_SCHEMES
#undef OCFD_FB_CASE
  return cudaErrorInvalidValue;
}

// Per-instance launch grid of a batched face sweep for tile variant V.
template <typename S>
dim3 face_batch_dims(int dir, int variant, const FaceArgs<S>& a) {
  if (dir == 0) return variant ? face_grid<0, 8, 32>(a) : face_grid<0, 4, 64>(a);
  if (dir == 1) return variant ? face_grid<1, 8, 32>(a) : face_grid<1, 16, 16>(a);
  return variant ? face_grid<2, 8, 32>(a) : face_grid<2, 16, 16>(a);
}

// ---- TMA path: tensor maps of the sweep's eight input arrays
bool face_tma_enabled();
bool face_tma32_enabled();
bool encode_tile_map(CUtensorMap* map, const void* base, bool f64, const Grid& g, int bx, int by, int bz);
// 4-D map of the interleaved FP32 u,v,w,T copy (4 floats a haloed point), box (4, bx, by, bz)
bool encode_tile_map4(CUtensorMap* map, const void* base, const Grid& g, int bx, int by, int bz);

template <typename S>
inline bool tma_strides_ok(const Grid& g) {
  return ((long long)g.nxh * sizeof(S)) % 16 == 0 && ((long long)g.nxh * g.nyh * sizeof(S)) % 16 == 0;
}

// tensor maps of a sweep's input arrays, boxes of B
template <typename B, typename S>
static bool face_tma_maps(const FaceArgs<S>& a, FaceTmaMaps& tm) {
  memset(&tm, 0, sizeof(tm));
  const S* arr[8] = {a.d, a.u, a.v, a.w, a.T, a.A1, a.A2, a.A3};
  for (int q = 0; q < 8; q++) {
    bool ok = true;
    if (sizeof(S) == 4 && q == 1)
      ok = encode_tile_map4(&tm.m[1], a.q4, a.g, B::BX, B::BY, B::BZ);
    else if (sizeof(S) == 8 || q == 0 || q >= 5)
      ok = encode_tile_map(&tm.m[q], arr[q], sizeof(S) == 8, a.g, B::BX, B::BY, B::BZ);
    if (!ok) return false;
  }
  return true;
}

template <int DIR, bool CHAR, int SCHEME, typename R, typename S, bool AXS = false, bool ALLIN = true>
static cudaError_t launch_face_tma_t(const FaceArgs<S>& a, cudaStream_t st) {
  using T = FaceTile<DIR, CHAR, SCHEME, R, ALLIN>;
  constexpr int NP = T::NP, TF = T::TF;
  using B = TmaBox<DIR, NP, TF, S, T::FPT>;
  constexpr size_t smem = FaceTmaSmem<DIR, CHAR, SCHEME, NP, TF, R, S, AXS, T::FPT, ALLIN>::BYTES;
  auto kern = k_face_tma<DIR, CHAR, SCHEME, R, S, AXS, ALLIN>;
  if (a.g.n == 0) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  FaceTmaMaps tm;
  if (!face_tma_maps<B>(a, tm)) return cudaErrorInvalidValue;
  kern<<<face_grid<DIR, NP, TF>(a), T::NT, smem, st>>>(a, tm);
  return cudaGetLastError();
}

// One (direction, form, scheme) combination: the TMA-staged sweep (FP64:
// periodic directions measured 1-3% faster at 256^3; FP32 with the four
// interleaved u,v,w,T floats of a point as the innermost dimension of a 4-D
// copy), the axis-aligned variant when the metric row allows it (production
// build).  An empty grid
// asks for the shared-memory attribute of every variant instead.
template <int D, bool C, int SC, typename R, typename S>
static cudaError_t launch_face_dc(const FaceArgs<S>& a, cudaStream_t st) {
  constexpr bool kAx = OCFD_FEWER_DIVS != 0;
  if (a.g.n == 0) {
    cudaError_t e = launch_face_t<D, C, SC, false, R, S>(a, st);
    if (e == cudaSuccess) e = launch_face_t<D, C, SC, true, R, S>(a, st);
    if (kAx && e == cudaSuccess) e = launch_face_t<D, C, SC, true, R, S, kAx>(a, st);
    if (e == cudaSuccess) e = launch_face_tma_t<D, C, SC, R, S>(a, st);
    if (kAx && e == cudaSuccess) e = launch_face_tma_t<D, C, SC, R, S, kAx>(a, st);
    if (e == cudaSuccess) e = launch_face_tma_t<D, C, SC, R, S, false, false>(a, st);
    return e;
  }
  const bool allin = a.ph.periodic[D] != 0;
  const bool tma = !a.no_tma && (sizeof(S) == 8 ? face_tma_enabled() : face_tma32_enabled()) && tma_strides_ok<S>(a.g);
  if (!allin) {
    if (tma) return launch_face_tma_t<D, C, SC, R, S, false, false>(a, st);
    return launch_face_t<D, C, SC, false, R, S>(a, st);
  }
  const bool ax = kAx && axis_aligned<D>(a.ph.metzero);
  if (tma) return ax ? launch_face_tma_t<D, C, SC, R, S, kAx>(a, st) : launch_face_tma_t<D, C, SC, R, S>(a, st);
  return ax ? launch_face_t<D, C, SC, true, R, S, kAx>(a, st) : launch_face_t<D, C, SC, true, R, S>(a, st);
}

template <typename R, typename S>
cudaError_t launch_face(int dir, bool chr, int scheme, const FaceArgs<S>& a, cudaStream_t st) {
#define OCFD_FACE_CASE(D, C, SC) \
  if (dir == D && chr == C && scheme == SC) return launch_face_dc<D, C, SC, R, S>(a, st);
#define OCFD_FACE_SCHEMES(D, C)         \
  OCFD_FACE_CASE(D, C, SCH_WENO5)       \
  OCFD_FACE_CASE(D, C, SCH_WENO7)       \
  OCFD_FACE_CASE(D, C, SCH_OMP6)        \
  OCFD_FACE_CASE(D, C, SCH_UD7L)        \
  OCFD_FACE_CASE(D, C, SCH_HYBRID)
  OCFD_FACE_SCHEMES(0, false)
  OCFD_FACE_SCHEMES(1, false)
  OCFD_FACE_SCHEMES(2, false)
  OCFD_FACE_SCHEMES(0, true)
  OCFD_FACE_SCHEMES(1, true)
  OCFD_FACE_SCHEMES(2, true)
#undef OCFD_FACE_SCHEMES
#undef OCFD_FACE_CASE
  return cudaErrorInvalidValue;
}

}  // namespace ocfd
