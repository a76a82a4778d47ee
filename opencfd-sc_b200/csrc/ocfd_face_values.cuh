// ocfd_face_values.cuh -- the mixed-precision hybrid's face fluxes (included by
// ocfd_face.cuh): the reference's splitting sums and schemes on stencil values.  Every
// other production sweep uses the shorter splittings and stencil differences.
//
// The hybrid's sensor is a hard threshold on the state: a last-bit change of an FP32
// flux moves faces beside a front from one scheme to the other, and two roundings of
// the same flux part by far more than they differ (isotropic turbulence with local
// Lax-Friedrichs splitting, 25 steps: 3e-5 in the 2-norm between this arithmetic and
// that of the differences, both within 6e-6 of the double-precision run).  Runs go on as
// they were begun only if the arithmetic stays as it is, so it is kept here, at the price
// of 5% of a step (192^3, ms per step: 3.18, on differences 3.03).  The splitting and the
// schemes are plain sums that the compiler contracts, so a change of this file, or of how
// it is inlined, is checked against stored digests (tests/test_gpu_mixed_hybrid.py).
#pragma once

namespace ocfd {

// The characteristic basis of one face: the rows of L = S and R = S^-1 of
// flux_charteric (OCFD_inviscous_character.f90:216-248) applied without forming the
// matrices.  AXS: the sweep's metric row has a single non-zero component, so
// n = s e_DIR with s its sign, and the general construction gives l = s e_y, m = e_z
// (DIR 0), l = -s e_x, m = e_z (DIR 1), l = -s e_x, m = -e_y (DIR 2): exact 0 and +-1
// entries, whose terms the projections and the back projection skip.
template <int DIR, bool AXS, typename R>
struct ValueBasis {
  static constexpr int LI = DIR == 0 ? 1 : 0;  // AXS: the velocity component along l
  static constexpr int MI = DIR == 2 ? 1 : 2;  // and along m
  R u, v, w, c;
  R n1, n2, n3, l1, l2, l3;  // AXS: n1 holds s, the others are unused

  __device__ __forceinline__ void init(R u1, R v1, R w1, R c1, R a1, R a2, R a3) {
    u = u1;
    v = v1;
    w = w1;
    c = c1;
    if constexpr (AXS) {
      n1 = copysign(R(1), DIR == 0 ? a1 : (DIR == 1 ? a2 : a3));
    } else {
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
  }
  __device__ __forceinline__ R vel(int q) const { return q == 0 ? u : (q == 1 ? v : w); }
  __device__ __forceinline__ R sl() const { return DIR == 0 ? n1 : -n1; }  // AXS: the non-zero entry of l
  // m = n x l
  __device__ __forceinline__ R m1() const { return xfma(n2, l3, -xmul(n3, l2)); }
  __device__ __forceinline__ R m2() const { return xfma(n3, l1, -xmul(n1, l3)); }
  __device__ __forceinline__ R m3() const { return xfma(n1, l2, -xmul(n2, l1)); }
  __device__ __forceinline__ R V2() const { return xmul(xfma(w, w, xfma(v, v, xmul(u, u))), R(0.5)); }
  __device__ __forceinline__ R un() const {
    return AXS ? xmul(n1, vel(DIR)) : xfma(w, n3, xfma(v, n2, xmul(u, n1)));
  }
  __device__ __forceinline__ R ul() const {
    return AXS ? xmul(sl(), vel(LI)) : xfma(w, l3, xfma(v, l2, xmul(u, l1)));
  }
  __device__ __forceinline__ R um() const {
    if constexpr (AXS) return DIR == 2 ? -v : w;
    return xfma(w, m3(), xfma(v, m2(), xmul(u, m1())));
  }
  // c = L f for one point (rows 0, 3, 4 through A = (V2,-u,-v,-w,1).f and
  // B = (un,-n).f: F0 - KK A and KK1 A +- X1 B)
  __device__ __forceinline__ void proj(R f0, R f1, R f2, R f3, R f4, R KK, R KK1, R X1, R V2_, R un_, R ul_,
                                       R um_, R* cc) const {
    const R A = xadd(xfma(-w, f3, xfma(-v, f2, xfma(-u, f1, xmul(V2_, f0)))), f4);
    cc[0] = xfma(-KK, A, f0);
    const R KA = xmul(KK1, A);
    if constexpr (AXS) {
      const R f[3] = {f1, f2, f3};
      const R B = xfma(-n1, f[DIR], xmul(un_, f0));
      cc[1] = xfma(-ul_, f0, xmul(sl(), f[LI]));
      cc[2] = xfma(-um_, f0, DIR == 2 ? -f[MI] : f[MI]);
      cc[3] = xfma(X1, B, KA);
      cc[4] = xfma(-X1, B, KA);
    } else {
      const R m1_ = m1(), m2_ = m2(), m3_ = m3();
      const R B = xfma(-n3, f3, xfma(-n2, f2, xfma(-n1, f1, xmul(un_, f0))));
      cc[1] = xfma(-ul_, f0, xfma(l3, f3, xfma(l2, f2, xmul(l1, f1))));
      cc[2] = xfma(-um_, f0, xfma(m3_, f3, xfma(m2_, f2, xmul(m1_, f1))));
      cc[3] = xfma(X1, B, KA);
      cc[4] = xfma(-X1, B, KA);
    }
  }
  // hh = R h0 (OCFD_inviscous_character.f90:284-288), H = V2 + c^2/(gamma-1)
  __device__ __forceinline__ void back(const R* h0, R* hh, R inv_gm1) const {
    const R V2_ = V2(), un_ = un(), ul_ = ul(), um_ = um();
    const R H = xfma(xmul(c, c), inv_gm1, V2_);
    hh[0] = xadd(xadd(h0[0], h0[3]), h0[4]);
    if constexpr (AXS) {
      const R cs = xmul(c, n1);
      R q[3];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const R vk = vel(k);
        if (k == DIR)
          q[k] = xfma(xadd(vk, cs), h0[4], xfma(xadd(vk, -cs), h0[3], xmul(vk, h0[0])));
        else if (k == LI)
          q[k] = xfma(vk, h0[4], xfma(vk, h0[3], xfma(sl(), h0[1], xmul(vk, h0[0]))));
        else
          q[k] = xfma(vk, h0[4], xfma(vk, h0[3], xadd(xmul(vk, h0[0]), DIR == 2 ? -h0[2] : h0[2])));
      }
      hh[1] = q[0];
      hh[2] = q[1];
      hh[3] = q[2];
    } else {
      const R m1_ = m1(), m2_ = m2(), m3_ = m3();
      hh[1] = xfma(xfma(c, n1, u), h0[4],
                   xfma(xfma(-c, n1, u), h0[3], xfma(m1_, h0[2], xfma(l1, h0[1], xmul(u, h0[0])))));
      hh[2] = xfma(xfma(c, n2, v), h0[4],
                   xfma(xfma(-c, n2, v), h0[3], xfma(m2_, h0[2], xfma(l2, h0[1], xmul(v, h0[0])))));
      hh[3] = xfma(xfma(c, n3, w), h0[4],
                   xfma(xfma(-c, n3, w), h0[3], xfma(m3_, h0[2], xfma(l3, h0[1], xmul(w, h0[0])))));
    }
    hh[4] = xfma(xfma(c, un_, H), h0[4],
                 xfma(xfma(-c, un_, H), h0[3], xfma(um_, h0[2], xfma(ul_, h0[1], xmul(V2_, h0[0])))));
  }
};

// One block of a sweep, one face per thread: face_body_main's arguments and shared-memory
// layout (in the characteristic form 17 values a point; the axis-aligned sweeps fill the
// ones they read).  Linear faces are finished at once; the WENO faces of the flux-vector
// form go through the block's list (FaceList), one (face, component) a thread.
template <int DIR, bool CHAR, bool ALLIN, int NP, int TF, typename R, typename S, bool TMA, bool AXS>
__device__ __forceinline__ void face_body_values(const FaceArgs<S>& a, const int bx, const int by, const int bz, R* sm,
                                                 const S* tile, int toff, R* qbase, int* qcount) {
  constexpr int SCHEME = SCH_HYBRID;
  constexpr int LT = TF + 7;
  constexpr int PS = face_ps<DIR, CHAR, R>();
  constexpr int GAP = PS > 1 ? 3 : 0;
  constexpr int VS = PS > 1 ? 1 : NP * LT;  // stride between variables
  auto PI = [](int l, int p) -> int { return DIR == 0 ? p * LT + l : l * NP + p; };  // point of the tile
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
  const R gam = R(ph.gamma);
  // the list and its two counts: after the staged points, or the caller's (see face_body_main)
  unsigned short* const ltag = reinterpret_cast<unsigned short*>(qbase ? qbase : sm + 10 * NP * LT);
  int* const ln = qbase ? qcount : reinterpret_cast<int*>(ltag + FaceList<NP * TF, false>::template bytes<R>() / 2);
  if (!CHAR && threadIdx.x < 2) ln[threadIdx.x] = 0;

  // ---- phase 1: split fluxes of the tile's points into shared memory
  for (int t = threadIdx.x; t < NP * LT; t += blockDim.x) {
    int l, p;
    if (DIR == 0) {
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
      using B = TmaBox<DIR, NP, TF, S>;
      const int e = DIR == 0 ? p * B::BX + l + toff : l * B::BX + p + toff;
      d = R(tile[e]);
      const float4 t = reinterpret_cast<const float4*>(tile + B::SLOT_ELEMS)[e];  // slots 1-4: u,v,w,T interleaved
      u = R(t.x);
      v = R(t.y);
      w = R(t.z);
      T = R(t.w);
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
      const float4 t = __ldg(reinterpret_cast<const float4*>(a.q4) + h);
      u = R(t.x);
      v = R(t.y);
      w = R(t.z);
      T = R(t.w);
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
    const R c = sqrt(T) * R(ph.inv_ma);
    R fp[5], fm[5];
    if constexpr (AXS) {
      const R Ad = DIR == 0 ? A1 : (DIR == 1 ? A2 : A3);
      if (a.split == 1)
        split_sw_axis_ref<DIR>(ph, gam, c, d, u, v, w, Ad, fp, fm);
      else
        split_llf_axis_ref<DIR>(ph, gam, c, d, u, v, w, Ad, fp, fm);
    } else {
      if (a.split == 1)
        split_sw_ref(ph, gam, c, d, u, v, w, A1, A2, A3, fp, fm);
      else
        split_llf_ref(ph, gam, c, d, u, v, w, A1, A2, A3, fp, fm);
    }
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
        // axis-aligned sweeps read only the direction's metric component
        if (!AXS || DIR == 0) sm[SI(14, l, p)] = A1;
        if (!AXS || DIR == 1) sm[SI(15, l, p)] = A2;
        if (!AXS || DIR == 2) sm[SI(16, l, p)] = A3;
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
  for (int t = threadIdx.x; t < NP * TF; t += blockDim.x) {
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
    // OCFD_inviscous.f90:76-81: Rhb0 = max(Rhybrid(g), Rhybrid(g+1))
    long long h = G.ih(i, j, k) + (long long)g * hs;
    double r0 = __ldg(a.rh + h), r1 = __ldg(a.rh + h + hs);
    const int ihy = hybrid_index(rmax(r0, r1), ph.hyb1, ph.hyb2);
    // the linear scheme of both sides, five components at a time: ud7lP and ud7lM as the
    // compiler contracts them, U0 f0 + (U1 f1) first
    auto linear = [&](R* h) {
      R x[5];
#pragma unroll
      for (int q = 1; q < 8; q++) {
        R fp[5], fm[5];
        W4(0, q, fp);
        fp[4] = W(4, q);
        W4(5, 7 - q, fm);
        fm[4] = W(9, 7 - q);
        if (q == 1) {
          R ep[5], em[5];
          W4(0, 0, ep);
          ep[4] = W(4, 0);
          W4(5, 7, em);
          em[4] = W(9, 7);
#pragma unroll
          for (int v = 0; v < 5; v++) {
            h[v] = xfma(U[0], ep[v], xmul(U[1], fp[v]));
            x[v] = xfma(U[0], em[v], xmul(U[1], fm[v]));
          }
        } else {
#pragma unroll
          for (int v = 0; v < 5; v++) {
            h[v] = xfma(U[q], fp[v], h[v]);
            x[v] = xfma(U[q], fm[v], x[v]);
          }
        }
      }
#pragma unroll
      for (int v = 0; v < 5; v++) h[v] = xadd(h[v], x[v]);
    };
    const int bi0 = ph.bi[2 * DIR], bi1 = ph.bi[2 * DIR + 1], sb0 = ph.sb[2 * DIR], sb1 = ph.sb[2 * DIR + 1];

    if (!CHAR) {
      // ---- flux-vector form: h1 (F+) and h2 (F-) per variable
      const int ib1 = (bi0 == 0 || sb0 == -1) ? 0 : -ph.ka1 + 1, ie1 = (bi1 == 0 || sb1 == -1) ? nn : nn - ph.kb1;
      const int ib2 = (bi0 == 0 || sb0 == -1) ? 0 : -ph.ka2 + 1, ie2 = (bi1 == 0 || sb1 == -1) ? nn : nn - ph.kb2;
      const bool inner = ALLIN || (g >= ib1 && g <= ie1 && g >= ib2 && g <= ie2);
      if (inner) {
        if (ihy != 1) {  // WENO7 faces from the front, WENO5 from the back
          const int n = atomicAdd(ln + (ihy == 2 ? 0 : 1), 1);
          ltag[ihy == 2 ? n : NP * TF - 1 - n] = (unsigned short)t;
          continue;
        }
        R hl[5];
        linear(hl);
        hf_store5(out, fo, a.fs, hl);
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
          out[hf_at(fo, a.fs, m)] = h1 + h2;
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
      if ((ALLIN || inner) && ihy == 1) {
        linear(hh);
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
        const R a1 = (AXS && DIR != 0) ? R(0) : mean(14);
        const R a2 = (AXS && DIR != 1) ? R(0) : mean(15);
        const R a3 = (AXS && DIR != 2) ? R(0) : mean(16);
        ValueBasis<DIR, AXS, R> cb;
        cb.init(u1, v1, w1, c1, a1, a2, a3);
        const R V2 = cb.V2(), un = cb.un(), ul = cb.ul(), um = cb.um();
        const R rc = R(1) / c1;
        const R KK = xmul(xadd(R(ph.gamma), R(-1)), xmul(rc, rc));
        const R KK1 = xmul(KK, R(0.5));
        const R X1 = xmul(R(0.5), rc);
        auto proj5 = [&](int vb, int q, R* c) {
          R f4[4];
          W4(vb, q, f4);
          cb.proj(f4[0], f4[1], f4[2], f4[3], W(vb + 4, q), KK, KK1, X1, V2, un, ul, um, c);
        };
        // F+ projected onto the characteristic variables (:254-261), reconstructed; then F- (:264-271)
        R h0[5];
        {
          R q[5][8];
#pragma unroll
          for (int s = 0; s < 8; s++) {
            R c[5];
            proj5(0, s, c);
#pragma unroll
            for (int r = 0; r < 5; r++) q[r][s] = c[r];
          }
          if (ALLIN || inner1) {
#pragma unroll
            for (int r = 0; r < 5; r++) h0[r] = schemeP<SCHEME>(q[r] + 3, U, ihy);
          } else {
#pragma unroll
            for (int r = 0; r < 5; r++) h0[r] = ch_flux1_bnd(q[r] + 3, g, nn, face_ends(ph, DIR));
          }
        }
        {
          R q[5][8];
#pragma unroll
          for (int s = 0; s < 8; s++) {
            R c[5];
            proj5(5, s, c);
#pragma unroll
            for (int r = 0; r < 5; r++) q[r][s] = c[r];
          }
          if (ALLIN || inner2) {
#pragma unroll
            for (int r = 0; r < 5; r++) h0[r] = h0[r] + schemeM<SCHEME>(q[r] + 3, U, ihy);
          } else {
#pragma unroll
            for (int r = 0; r < 5; r++) h0[r] = h0[r] + ch_flux2_bnd(q[r] + 3, g, nn, face_ends(ph, DIR));
          }
        }
        cb.back(h0, hh, R(ph.inv_gm1));  // back to physical space, hh = R h0 (:284-288)
      }
    }
    hf_store5(out, fo, a.fs, hh);
  }
  if constexpr (!CHAR) {
    __syncthreads();
    const int n7 = ln[0], nj = n7 + ln[1];
#pragma unroll 1
    for (int e = threadIdx.x; e < 5 * nj; e += NP * TF) {
      const int m = e / nj, x = e - m * nj;
      const int t = ltag[x < n7 ? x : NP * TF - 1 - (x - n7)];
      const int ihy = x < n7 ? 2 : 3;
      int f, p;
      if (DIR == 0) {
        f = t % TF;
        p = t / TF;
      } else {
        p = t % NP;
        f = t / NP;
      }
      int i, j, k;
      pencil(p, i, j, k);
      const int g = g0 + f;
      const R* wb = sm + PI(f, p) * PS;
      auto W = [&](int var, int q) -> R { return wb[var * VS + (var >= 5 ? GAP : 0) + q * QS]; };
      const long long fo = G.face(DIR, g, DIR == 0 ? g : i, DIR == 1 ? g : j, DIR == 2 ? g : k);
      R wv[8];
#pragma unroll
      for (int q = 0; q < 8; q++) wv[q] = W(m, q);
      const R h1 = schemeP<SCHEME>(wv + 3, U, ihy);
#pragma unroll
      for (int q = 0; q < 8; q++) wv[q] = W(5 + m, q);
      const R h2 = schemeM<SCHEME>(wv + 3, U, ihy);
      out[hf_at(fo, a.fs, m)] = h1 + h2;
    }
  }
}

}  // namespace ocfd
