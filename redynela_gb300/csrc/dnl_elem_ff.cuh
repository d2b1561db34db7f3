// The element pass in pairs of FP32 numbers (dnl_ff.cuh) for points whose increment is small, which
// is nearly every point of every step; included by dnl_elem.cu after the FP64 pass (elem_ip), whose
// phases, lane layout and error codes it shares.
//
// What bounds the FP64 pass is its ~900 FP64 instructions per hexahedral Gauss point at 64 cycles
// each.  Here FP64 is left where its 53 bits are the point: differences of nodal coordinates and
// displacements (exact, a few per lane) and the sums of increments into the stored state, the
// pressure, evp and evp^n -- 29 additions per hexahedral point in the middle of an impact.  Everything in
// between is formed as small quantities (F - I, C - I, ln U, R - I, stress increments, R X R^T - X).

// element types with the pair pass (the 10-node tetrahedron's tables make its Jacobian depend on
// absolute coordinates: FP64)
__host__ __device__ constexpr bool etype_fast(int et) { return et != DNL_ELTET10N3D; }

// weights dN/dxi of the quads' and the hexahedron's edges and N of the quads as pairs
struct ShapeFF {
  ff axN[3], axD[2], hxD[3];
  ff gpow[2][4];  // 3^(-c/2) / 4 (quads) and / 8 (hexahedron)
};
__constant__ ShapeFF c_shapeFF;
// the polar decomposition's stopping test as a pair, and whether the tolerances are within the pairs'
// reach (2^-52 to 2^-29 for the polar decomposition, whose dropped terms, up to the tolerance, go through
// single precision: at 1e-5 ln U would carry 9e-14; 2^-44 for the radial return; else every point is FP64's)
struct TolFF {
  ff polar;
  int ok;
};
__constant__ TolFF c_tolFF = {{(float)kPolarPrecision, (float)(kPolarPrecision - (double)(float)kPolarPrecision)}, 1};

__device__ __forceinline__ float2 f2(ff a) { return make_float2(a.h, a.l); }
__device__ __forceinline__ ff ff_from(float2 a) { return ff{a.x, a.y}; }
__device__ __forceinline__ ff ff_shfl(ff a, int mask)
{
  return ff{__shfl_xor_sync(0xffffffffu, a.h, mask), __shfl_xor_sync(0xffffffffu, a.l, mask)};
}
constexpr float hi_part(double x) { return (float)x; }
constexpr float lo_part(double x) { return (float)(x - (double)(float)x); }
#define FF_CONST(x) (ff{hi_part(x), lo_part(x)})

// |dN/dxi_c| of node k at point pt as a pair, and its sign (+1 or -1)
template <int ET> __device__ __forceinline__ ff dN_ff(int pt, int k, int c)
{
  ff w;
  int s;
  if constexpr (ET == DNL_ELHEX8N3D) {
    const int dx = sgx(k) ^ sgx(pt), dy = sgy(k) ^ sgy(pt), dz = sgz(k) ^ sgz(pt);
    const int d = c == 0 ? dy + dz : (c == 1 ? dx + dz : dx + dy);
    w = d == 0 ? c_shapeFF.hxD[0] : (d == 1 ? c_shapeFF.hxD[1] : c_shapeFF.hxD[2]);
    s = c == 0 ? sgx(k) : (c == 1 ? sgy(k) : sgz(k));
  } else {
    const int other = c == 0 ? (sgy(k) ^ sgy(pt)) : (sgx(k) ^ sgx(pt));
    w = other ? c_shapeFF.axD[1] : c_shapeFF.axD[0];
    s = c == 0 ? sgx(k) : sgy(k);
  }
  const uint32_t f = s ? 0u : 0x80000000u;
  return ff{bits_f(f_bits(w.h) ^ f), bits_f(f_bits(w.l) ^ f)};
}
__device__ __forceinline__ ff axN_ff(int pt, int k)
{
  const int d = (sgx(k) ^ sgx(pt)) + (sgy(k) ^ sgy(pt));
  return d == 0 ? c_shapeFF.axN[0] : (d == 1 ? c_shapeFF.axN[1] : c_shapeFF.axN[2]);
}

// Walsh transform of eight values, the first of them 0: after it, entry m is sum_b (-1)^popcount(m & b) v_b.
// Sums and differences with their rounding errors: on one grid for all eight values, two additions each
// instead of eight, the low parts lost 2^-44 of the largest value, and with them J and G_u
// (ln U at |G| = 2^-8: 1.6e-16 root mean square, now 1.8e-17, FP64 5.8e-17) and the hourglass forces (1.5e-13
// of themselves, now 8e-15; FP64 3e-14 at 5 to 60 edges from the origin, where its sums round).
__device__ __forceinline__ void walsh8(ff (&v)[8])
{
  v[0] = v[1];
  v[1] = ff_neg(v[1]);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1)
#pragma unroll
    for (int b = o == 1 ? 2 : 0; b < 8; b++)
      if (!(b & o)) {
        const ff p = v[b], q = v[b | o];
        v[b] = ff_add_raw(p, q);
        v[b | o] = ff_add_raw(p, ff_neg(q));
      }
}
// node k's place: bit 0, 1, 2 set where xi, eta, zeta = +1
__device__ __forceinline__ constexpr int sign_place(int k) { return ((k ^ (k >> 1)) & 1) | (k & 2) | (k & 4); }
// A nodal field relative to its value at the element's first node (d[0] = 0); the high word of the
// largest difference
__device__ __forceinline__ uint32_t rel_first(const double *f, const int (&nd)[8], double (&d)[8])
{
  const double f0 = f[nd[0]];
  uint32_t top = 0;
  d[0] = 0.;
#pragma unroll
  for (int k = 1; k < 8; k++) {
    d[k] = RSUB(f[nd[k]], f0);
    top = max(top, f64_mag(d[k]));
  }
  return top;
}
// The transform of such differences times 2^k (k20 = k << 20).  The sign product of the directions in m
// at node b is (-1)^|m| (-1)^popcount(m & b).
__device__ __forceinline__ void walsh_of(const double (&d)[8], int k20, ff (&w)[8])
{
#pragma unroll
  for (int k = 1; k < 8; k++) w[sign_place(k)] = ff_of(d[k], k20);
  walsh8(w);
#pragma unroll
  for (int k = 1; k < 8; k++) w[k] = ff_norm(w[k].h, w[k].l);
}
// hourglass coefficients of the coordinates (xi eta, eta zeta, zeta xi, xi eta zeta)
struct HourglassX {
  ff x[4][3];
};
// x^(2/3) of a positive pair within the float range: seed by the hardware exponential and logarithm
// base 2, two Newton steps of y^3 = x with the residual in pairs (one left 1e-13, the rounding of its
// correction of 1e-6)
__device__ __forceinline__ ff pow23_ff(ff x)
{
  ff y = {exp2f(log2f(x.h) * (1.f / 3.f)), 0.f};
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const ff y2 = ff_mul(y, y), r = ff_sub(x, ff_mul(y2, y));
    y = ff_norm(y.h, y.l + r.h * (f_rcp(y2.h) * (1.f / 3.f)));
  }
  return ff_mul(y, y);
}

// The first pivot of the polar decomposition (0: C01, 1: C02, 2: C12) from C in FP64 with the
// reference's rounding, for points where two off-diagonal entries are equal within the pairs' error
// (planes of symmetry of regular meshes: there the choice is the reference's rounding's, and the
// two choices differ at the stopping tolerance).  Warp-collective.
template <int ET>
__device__ __noinline__ int pivot_f64(const ElemArgs &a, int e, int pt, double *red)
{
  constexpr int NEN = Elem<ET>::NEN, DIM = Elem<ET>::DIM;
  int node[NEN];
#pragma unroll
  for (int k = 0; k < NEN; k++) node[k] = __ldg(a.conn + (long)k * a.E + e);
  double J[DIM][DIM], GU[DIM][DIM], Ji[DIM][DIM], F[3][3], f[3][3], Rad, vR, detJ;
  kinematics_f64<ET>(a, e, pt, node, red, J, GU, Rad, vR);
  inverse_f64(J, detJ, Ji);
  gradient_f64(GU, Ji, F);
  cauchy_f64<DIM == 2>(F, f);
  const bool q1 = abs_gt(f[0][1], f[0][2]);
  return abs_gt(q1 ? f[0][1] : f[0][2], f[1][2]) ? (q1 ? 0 : 1) : 2;
}

// The tabular law (hardening_law) with its stress and slope over 2^k as pairs; false past the table's
// end, on a vertical or nearly vertical segment (below 2^-60: a width below 2^-70 would be converted to 0) and
// outside the pairs' range (FP64 then).  The search compares the doubles' bits (x > 0).
__device__ __forceinline__ bool table_ff(const HardLaw &m, double x, int k20, ff &sig, ff &h)
{
  const double *X = m.tab, *Y = m.tab + m.tabN;
  const long long xb = __double_as_longlong(x);
  int lo = 1, hi = m.tabN;  // first i in [1, N) with X[i] >= x, else N
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__double_as_longlong(__ldg(X + mid)) >= xb)
      hi = mid;
    else
      lo = mid + 1;
  }
  if (lo >= m.tabN) return false;
  const double x0 = __ldg(X + lo - 1), y0 = __ldg(Y + lo - 1), x1 = __ldg(X + lo), y1 = __ldg(Y + lo);
  const uint32_t top = (uint32_t)((1023 + 50) << 20);
  if (f64_mag(x1 - x0) < (uint32_t)((1023 - 60) << 20) || max(f64_mag(x0), f64_mag(x1)) >= top || max(f64_mag(y0), f64_mag(y1)) >= top + (uint32_t)k20) return false;
  h = ff_mul(ff_of(y1 - y0, -k20), ff_rcp(ff_of(x1 - x0)));
  sig = ff_add(ff_of(y0, -k20), ff_mul(ff_of(x - x0), h));
  return true;
}

// Shared memory that holds a point's increments between the radial return and the rotation: entry i
// of the thread at hold[i HOLD], so that a warp's accesses are consecutive.
constexpr int HOLD = 32;
template <int ET> __host__ __device__ constexpr int hold_slots() { return 3 * Elem<ET>::NS; }

// One Gauss point in pairs.  Returns true when its element needs the FP64 pass instead (an increment
// above its limit, a badly shaped element, state or constants outside the pairs' range): then
// nothing of the element is stored or recorded.  Uniform over the element's lanes; depends on the
// element's own data only, so a warp's other elements do not matter.
template <int ET, bool TAPE, bool GENERAL>
__device__ __forceinline__ bool elem_fast(const ElemArgs &a, const Material &m, DevTime *tm, int e, int pt,
                                          bool valid, int lane, double *red, float2 *hold)
{
  using T = Elem<ET>;
  using Ly = IpLayout<ET>;
  using TL = TapeLayout<ET>;
  constexpr int NIP = T::NIP, NEN = T::NEN, DIM = T::DIM, NS = T::NS;
  constexpr bool AXI = ET == DNL_ELQUA4NAX;
  constexpr bool TWO_D = DIM == 2;
  constexpr bool EDGES = ET == DNL_ELHEX8N3D || ET == DNL_ELQUA4NAX || ET == DNL_ELQUA4N2D;
  const MatFF &mf = m.f;
  const long nIP = (long)a.E * NIP;
  const long ipx = (long)e * NIP + pt;
  float2 *const sh = reinterpret_cast<float2 *>(red);  // this element's shared memory
  const ff zero = {0.f, 0.f};

  // ---- J and G_u from differences of nodal values: FP64 differences, pairs from there on.  Lengths are
  // over 2^js, the power of two above the element's largest coordinate difference: one scale for the
  // element, as its lanes exchange products of their J, and taken before the conversion, so that the
  // unit of length does not matter (exact, and G is unchanged).
  ff J[DIM][DIM], GU[DIM][DIM];
  ff Rad = zero, vR = zero;
  uint32_t top = 0, topX = 0;  // largest high words: of the lane's other lengths, of the differences of x
  int js;
  float mJ[DIM];
  HourglassX hg;  // the one-point hexahedron's
  auto scale_of = [&]() {
#pragma unroll
    for (int o = 1; o < NIP; o <<= 1) topX = max(topX, __shfl_xor_sync(0xffffffffu, topX, o));
    js = (int)(topX >> 20) - 1022;
    return -js * (1 << 20);
  };
  if constexpr (EDGES) {
    using EG = Edges<ET>;
    constexpr int NE = EG::NE, PER = NE / DIM;
    float2 *ex = sh, *eu = sh + NE * DIM;
    double dx[DIM], du[DIM], dh[DIM];  // the lane's edge, and half of another
    {
      const int lo = __ldg(a.conn + (long)edge_node(EG::LO, pt) * a.E + e);
      const int hi = __ldg(a.conn + (long)edge_node(EG::HI, pt) * a.E + e);
#pragma unroll
      for (int r = 0; r < DIM; r++) {
        dx[r] = RSUB(a.x[r][hi], a.x[r][lo]);
        du[r] = RSUB(a.du[r][hi], a.du[r][lo]);
        topX = max(topX, f64_mag(dx[r]));
        top = max(top, f64_mag(du[r]));
      }
    }
    const int eg2 = NIP + (pt & (NIP / 2 - 1));
    const bool isx = pt < NIP / 2;
    if constexpr (NE > NIP) {  // the hexahedron's other four edges: x on one half of the lanes, u on the other
      static_assert(NE == NIP + NIP / 2, "edges per lane");
      const int lo = __ldg(a.conn + (long)edge_node(EG::LO, eg2) * a.E + e);
      const int hi = __ldg(a.conn + (long)edge_node(EG::HI, eg2) * a.E + e);
#pragma unroll
      for (int r = 0; r < DIM; r++) {
        const double *src = isx ? a.x[r] : a.du[r];
        dh[r] = RSUB(src[hi], src[lo]);
        const uint32_t t = f64_mag(dh[r]);
        topX = max(topX, isx ? t : 0u);
        top = max(top, isx ? 0u : t);
      }
    }
    const int j20 = scale_of();
#pragma unroll
    for (int r = 0; r < DIM; r++) {
      ex[pt * DIM + r] = f2(ff_of(dx[r], j20));
      eu[pt * DIM + r] = f2(ff_of(du[r], j20));
      if constexpr (NE > NIP) (isx ? ex : eu)[eg2 * DIM + r] = f2(ff_of(dh[r], j20));
    }
    if (AXI) {  // the nodes' radii and radial displacements
      const int nd = __ldg(a.conn + (long)pt * a.E + e);
      const double x0 = a.x[0][nd], u0 = a.du[0][nd];
      top = max(top, max(f64_mag(x0), f64_mag(u0)));
      sh[2 * NE * DIM + pt] = f2(ff_of(x0, j20));
      sh[2 * NE * DIM + NEN + pt] = f2(ff_of(u0, j20));
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < DIM; c++) {
      ff w[PER], dx[PER][DIM], du[PER][DIM];
#pragma unroll
      for (int q = 0; q < PER; q++) {
        const int eg = c * PER + q;
        w[q] = dN_ff<ET>(pt, edge_node(EG::HI, eg), c);
#pragma unroll
        for (int r = 0; r < DIM; r++) {
          dx[q][r] = ff_from(ex[eg * DIM + r]);
          du[q][r] = ff_from(eu[eg * DIM + r]);
        }
      }
      mJ[c] = 0.f;
#pragma unroll
      for (int r = 0; r < DIM; r++) {
        // both sums compensated: G_u on a grid of its edges' size cost ln U more than all that follows
        // (hexahedra, |G| = 2^-7: 1.1e-16 against 4.0e-17, FP64 5.6e-17)
        Dot sx(dx[0][r], w[0]), su(du[0][r], w[0]);
#pragma unroll
        for (int q = 1; q < PER; q++) {
          sx.mac(dx[q][r], w[q]);
          su.mac(du[q][r], w[q]);
        }
        J[r][c] = sx.get();
        GU[r][c] = su.get();
        mJ[c] = f_max(mJ[c], f_abs(J[r][c].h));
      }
    }
    if (AXI) {
      ff xr[NEN], ur[NEN];
#pragma unroll
      for (int k = 0; k < NEN; k++) {
        xr[k] = ff_from(sh[2 * NE * DIM + k]);
        ur[k] = ff_from(sh[2 * NE * DIM + NEN + k]);
      }
      Dot sx(xr[0], axN_ff(pt, 0)), su(ur[0], axN_ff(pt, 0));
#pragma unroll
      for (int k = 1; k < NEN; k++) {
        const ff n = axN_ff(pt, k);
        sx.mac(xr[k], n);
        su.mac(ur[k], n);
      }
      Rad = sx.get();
      vR = su.get();
    }
    __syncwarp();  // the force assembly reuses the buffer
  } else if constexpr (ET == DNL_ELTET4N3D) {
    int nd[4];
    double dx[3][3], du[3][3];  // [component][axis]
#pragma unroll
    for (int k = 0; k < 4; k++) nd[k] = __ldg(a.conn + (long)k * a.E + e);
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int r = 0; r < 3; r++) {
        dx[r][c] = RSUB(a.x[r][nd[c + 1]], a.x[r][nd[0]]);
        du[r][c] = RSUB(a.du[r][nd[c + 1]], a.du[r][nd[0]]);
        topX = max(topX, f64_mag(dx[r][c]));
        top = max(top, f64_mag(du[r][c]));
      }
    const int j20 = scale_of();
#pragma unroll
    for (int c = 0; c < 3; c++) {
      mJ[c] = 0.f;
#pragma unroll
      for (int r = 0; r < 3; r++) {
        J[r][c] = ff_of(dx[r][c], j20);
        GU[r][c] = ff_of(du[r][c], j20);
        mJ[c] = f_max(mJ[c], f_abs(J[r][c].h));
      }
    }
  } else {
    // the one-point hexahedron: values relative to node 0's (FP64), their Walsh transforms over the
    // node signs in pairs: J and G_u (1/8 of the linear coefficients), the hourglass coefficients of
    // x, all coefficients of v
    int nd[NEN];
    double dx[DIM][NEN];
#pragma unroll
    for (int k = 0; k < NEN; k++) nd[k] = __ldg(a.conn + (long)k * a.E + e);
#pragma unroll
    for (int r = 0; r < DIM; r++) topX = max(topX, rel_first(a.x[r], nd, dx[r]));
    const int j20 = scale_of();
#pragma unroll
    for (int c = 0; c < DIM; c++) mJ[c] = 0.f;
#pragma unroll
    for (int r = 0; r < DIM; r++) {
      ff w[NEN];
      double d[NEN];
      walsh_of(dx[r], j20, w);
      hg.x[0][r] = w[3];
      hg.x[1][r] = w[6];
      hg.x[2][r] = w[5];
      hg.x[3][r] = ff_neg(w[7]);
#pragma unroll
      for (int c = 0; c < DIM; c++) {
        J[r][c] = ff_scale(ff_neg(w[1 << c]), 0.125f);
        mJ[c] = f_max(mJ[c], f_abs(J[r][c].h));
      }
      top = max(top, rel_first(a.du[r], nd, d));
      walsh_of(d, j20, w);
#pragma unroll
      for (int c = 0; c < DIM; c++) {
        GU[r][c] = ff_scale(ff_neg(w[1 << c]), 0.125f);
      }
    }
  }
  // lengths within 2^-200 .. 2^200, none above 2^60 of the element's size (what is below 2^-70 of it is 0;
  // of displacements that is less than FP64 resolves in F)
  bool bad = !mf.ok || !c_tolFF.ok || js < -200 || js > 200 || (int)top >= (1022 + 60 + js) << 20;
  if constexpr (ET == DNL_ELHEX8N3D_1PT) {
    // the hourglass forces' factors: speeds below 2^39 (infinities and NaN are above it), rho c and the
    // coefficient within ranges whose product a float holds.  The state is stored before the forces are
    // formed, so this is looked at here.
    uint32_t topV = 0;
#pragma unroll
    for (int k = 0; k < NEN; k++) {
      const int n = __ldg(a.conn + (long)k * a.E + e);
#pragma unroll
      for (int r = 0; r < DIM; r++) topV = max(topV, f64_mag(a.v[r][n]));
    }
    const uint32_t c = f64_mag(a.hourglass), lo = (uint32_t)((1023 - 20) << 20);
    bad |= topV >= (uint32_t)((1023 + 39) << 20) || !mf.okHg || (c != 0u && c - lo >= (uint32_t)(40 << 20));
  }

  // ---- adjugate, determinant, G = G_u J^-1
  ff adj[DIM][DIM], det, rdet, G[3][3];
  float cols;
  deform_ff<DIM>(J, GU, mJ, adj, det, rdet, G, cols);
  bad |= !(f_abs(det.h) >= (TWO_D ? 0x1p-5f : 0x1p-6f) * cols);
  float mg = 0.f;
#pragma unroll
  for (int r = 0; r < DIM; r++)
#pragma unroll
    for (int c = 0; c < DIM; c++) mg = f_max(mg, f_abs(G[r][c].h));
  if (AXI) {
    G[2][2] = ff_mul(vR, ff_rcp(Rad));
    mg = f_max(mg, f_abs(G[2][2].h));
    bad |= !(Rad.h > 0x1p-60f);
  }
  bad |= !(mg <= kFastMax) || mg * cols > kShapeMax * kFastMax * f_abs(det.h);

  // all of the warp's elements for the FP64 form: the rest of this pass, three quarters of it, would be for
  // nothing (increments of 2^-5 throughout: 43,456 hexahedra 759 -> 715 us, the FP64 form alone 698; tetrahedra
  // 154 -> 121, 115)
  {
    const unsigned b = __ballot_sync(0xffffffffu, bad), mine = NIP > 1 ? ((1u << NIP) - 1u) << (lane - pt) : 1u << lane;
    if (__all_sync(0xffffffffu, (b & mine) != 0u || !valid)) return true;
  }

  // ---- ln U and R - I
  ff E[6];
  const float mge = green_ff<TWO_D>(G, E);
  int first = -1;
  if constexpr (!TWO_D) {
    const bool tie = valid && !bad && pivot_tie(E, mge, c_tolFF.polar.h);
    if (__any_sync(0xffffffffu, tie)) {
      const int k = pivot_f64<ET>(a, e, pt, red);
      __syncwarp();
      if (tie) first = k;
    }
  }
  ff Ln[6], Q[3][3];
  bool conv;
  if constexpr (TAPE) {
    ff V[3][3], lam[3], H[6];
    conv = strain_ff<TWO_D, true>(G, E, mge, c_tolFF.polar, c_caps[0], first, Ln, Q, V, lam, H);
    auto tape = [&](int slot, double v) {
      if (valid && !bad) a.tape[(long)slot * nIP + ipx] = v;
    };
    const int j20 = js * (1 << 20);
#pragma unroll
    for (int l = 0; l < DIM; l++)
#pragma unroll
      for (int c = 0; c < DIM; c++) {
        tape(TL::JI + l * DIM + c, f64_of(ff_mul(adj[l][c], rdet), -j20));
        tape(TL::GU + l * DIM + c, f64_of(GU[l][c], j20));
      }
    tape(TL::DETJ, f64_of(det, DIM * j20));
    tape(TL::RAD, AXI ? f64_of(Rad, j20) : 0.);
    tape(TL::VRR, AXI ? f64_of(G[2][2]) : 0.);
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const int i = k / 3, j = k % 3;
      const double d = i == j ? 1. : 0.;
      const bool out = TWO_D && (i == 2) != (j == 2);  // outside the plane case's blocks: 0
      tape(TL::F + k, out ? 0. : f64_add(d, G[i][j]));
      tape(TL::R + k, out ? 0. : f64_add(d, Q[i][j]));
      tape(TL::V + k, f64_of(V[i][j]));
    }
    // divided differences of ln(l)/2 and l^-1/2 (Daleckii-Krein factors), l = 1 + lam; the second is
    // -1 / (sqrt(li lj) (sqrt(li) + sqrt(lj))).  Between the plane case's blocks they multiply zeros.  In FP64,
    // with divisions and logarithms, they and the sums that are 0 took a quarter of this pass on 4,000
    // axisymmetric elements (its adjoint of 150 steps: 13.3 -> 12.5 ms).
    ff il[3], sq[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const ff y = ff_add(ff{1.f, 0.f}, lam[k]);
      il[k] = ff_add(ff{1.f, 0.f}, rsqrt1p_ff(lam[k]));
      sq[k] = ff_mul(y, il[k]);
    }
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const int i = sym_i(k), j = sym_j(k);
      const bool out = TWO_D && k > 3;
      ff g = zero, hh = zero;
      if (i == j) {
        const ff h = ff_scale(ff_mul(il[i], il[i]), 0.5f);
        g = h;
        hh = ff_neg(ff_mul(h, il[i]));
      } else if (!out) {
        g = half_log_slope_ff(lam[i], lam[j]);
        hh = ff_neg(ff_mul(ff_mul(il[i], il[j]), ff_rcp(ff_add(sq[i], sq[j]))));
      }
      tape(TL::GD + k, f64_of(g));
      tape(TL::HD + k, f64_of(hh));
      tape(TL::UI + k, out ? 0. : f64_add(i == j ? 1. : 0., H[k]));
    }
  } else {
    conv = strain_ff<TWO_D, false>(G, E, mge, c_tolFF.polar, c_caps[0], first, Ln, Q);
  }

  // ---- strain increment's trace; element-mean pressure increment (butterfly: the sum of a pair is
  // symmetric in its arguments, so every lane gets the same)
  const ff trace = ff_add(ff_add(Ln[0], Ln[1]), Ln[2]);
  ff pinc = trace;
#pragma unroll
  for (int o = 1; o < NIP; o <<= 1) pinc = ff_add(pinc, ff_shfl(pinc, o));
  pinc = ff_mul(mf.K, ff_scale(pinc, 1.f / NIP));

  // ---- trial stress, J2 radial return (Element.C:245-345), stresses over 2^k
  const int k20 = mf.k20;
  const double pd = a.ip[Ly::P * nIP + ipx];
  ff St[6], inc[6];
#pragma unroll
  for (int k = 0; k < 6; k++) St[k] = inc[k] = zero;
  {
    uint32_t topS = 0;
#pragma unroll
    for (int k = 0; k < NS; k++) {
      const double Sd = a.ip[(Ly::S + k) * nIP + ipx];
      topS = max(topS, f64_mag(Sd));
      St[k] = ff_of(Sd, -k20);
    }
    topS = max(topS, f64_mag(pd));
    bad |= topS >= (uint32_t)(((1023 + 50) << 20) + k20);
    // Eps and EpsPlas are read further down, when parts of the element may be stored: their high words here
    uint32_t topE = 0;
#pragma unroll
    for (int k = 0; k < NS; k++)
      topE = max(topE, max(f64_mag_at(a.ip + (Ly::EPS + k) * nIP + ipx), f64_mag_at(a.ip + (Ly::EPSP + k) * nIP + ipx)));
    bad |= topE >= (uint32_t)((1023 + 100) << 20);
    const ff tr3 = ff_mul(trace, FF_CONST(1. / 3.));
#pragma unroll
    for (int k = 0; k < NS; k++) {
      inc[k] = ff_mul(mf.g2, k < 3 ? ff_sub(Ln[k], tr3) : Ln[k]);
      St[k] = ff_add(St[k], inc[k]);
    }
  }
  double evp = a.ip[Ly::EVP * nIP + ipx];
  double evpn = a.ip[Ly::EVPN * nIP + ipx];
  bool plastic = false, rr_ok = true;
  ff gi = zero;  // gamma / |S|
  {
    Dot s(St[0], St[0]);
#pragma unroll
    for (int k = 1; k < NS; k++) s.mac(k < 3 ? St[k] : ff_scale(St[k], 2.f), St[k]);
    const ff ss = s.get();
    const bool some = ss.h > 0x1p-100f;
    const ff inv = some ? ff_rsqrt(ss) : zero;
    const ff normS = some ? ff_sqrt(ss, inv.h) : zero;
    const ff Strial = ff_mul(FF_CONST(kSqrt32), normS);
    const bool power = !GENERAL || m.hard.law == DNL_HARD_POWER;
    const bool table = GENERAL && m.hard.law == DNL_HARD_TABULAR;
    if (TAPE && valid && !bad) {
#pragma unroll
      for (int k = 0; k < NS; k++)
        a.tape[(long)(TL::STR + k) * nIP + ipx] = f64_add(a.ip[(Ly::S + k) * nIP + ipx], inc[k], k20);
      a.tape[(long)TL::NORMS * nIP + ipx] = f64_of(normS, k20);
    }
    double gam_d = 0., lxv = 0.;
    if (power || table) {
      bad |= f64_mag(evp) - (uint32_t)((1023 - 60) << 20) >= (uint32_t)(120 << 20);  // 2^-60 .. 2^60
      const ff one = {1.f, 0.f};
      ff evF = zero, Bx = zero, revp = zero, Sig0, h0;
      if (power) {
        bad |= f64_mag(evpn) >= (uint32_t)((1023 + 30) << 20);
        evF = ff_of(evp);
        Bx = ff_mul(mf.B, ff_of(evpn));
        revp = ff_rcp(evF);
        Sig0 = ff_add(mf.A, Bx);
        h0 = ff_mul(ff_mul(mf.n, Bx), revp);  // n B evp^(n-1)
      } else {
        bad |= !table_ff(m.hard, evp, k20, Sig0, h0);
      }
      // evp^n below the pairs' range matters only where it is to grow: FP64 then
      if (power && ff_gt(Strial, Sig0)) bad |= f64_mag(evpn) < (uint32_t)((1023 - 60) << 20);
      if (ff_gt(Strial, Sig0) && !bad) {
        plastic = true;
        ff gamma = ff_mul(ff_sub(normS, ff_mul(FF_CONST(kSqrt23), Sig0)),
                          ff_rcp(ff_mul(mf.g2, ff_add(one, ff_mul(h0, mf.rG3)))));
        const float tol = (float)c_returnTol;
        ff Tn = zero;
        int iteration = 0;
        for (;;) {
          const ff dv = ff_mul(FF_CONST(kSqrt23), gamma);  // xv = evp + dv
          ff Sigv, h;
          if (power) {
            // (xv / evp)^n - 1 from q = dv / evp: the binomial series while q <= 2^-6 (all but a point's
            // first steps), else by logarithm and exponential
            const ff q = ff_mul(dv, revp), q1 = ff_add(one, q);
            if (q.h <= (float)kSeriesMax && f_abs(mf.n.h) <= 2.f)
              Tn = pow1p_ff(mf, q);
            else
              Tn = powq_ff(mf.n, mf.n3, q);
            Sigv = ff_add(Sig0, ff_mul(Bx, Tn));
            h = ff_mul(h0, ff_mul(ff_add(one, Tn), ff_rcp(q1)));
            if (!(q.h >= 0.f && q.h < 0x1p60f && mf.n.h * __log2f(q1.h) < 58.f && mf.n.h >= 0.f)) {
              bad = true;  // FP64 instead
              break;
            }
          } else if (!table_ff(m.hard, f64_add(evp, dv), k20, Sigv, h)) {
            bad = true;
            break;
          }
          // f = sqrt(3/2) 2 G gamma - Strial + sigma_y (the reference's terms in h cancel)
          const ff fun = ff_add(ff_sub(ff_mul(mf.dfun0, gamma), Strial), Sigv);
          // the residual carries some 2^-46 of the trial stress, 1e-6 of the tolerance: where that decides, FP64 does
          const float af = f_abs(fun.h), lim = tol * f_abs(Sigv.h);
          if (f_abs(af - lim) <= 0x1p-44f * Strial.h) {
            bad = true;
            break;
          }
          if (af > lim) {
            ff dg = ff_neg(ff_mul(fun, ff_rcp(ff_add(mf.dfun0, ff_mul(FF_CONST(kSqrt23), h)))));
            if (dg.h < 0.f && f_abs(dg.h) > gamma.h) dg = ff_mul(gamma, FF_CONST(-0.9));
            gamma = ff_add(gamma, dg);
          } else {
            break;
          }
          iteration++;
          if (iteration > c_caps[1]) {
            rr_ok = false;
            break;
          }
        }
        bad |= !(f_abs(gamma.h) < 0x1p30f);  // no root: a table whose slope cancels 3 G
        gi = ff_mul(gamma, inv);
        const double xv = f64_add(evp, ff_mul(FF_CONST(kSqrt23), gamma));
        if (TAPE) {
          gam_d = f64_of(gamma);
          lxv = log(xv);
        }
        evp = xv;
        if (power) evpn = f64_add(evpn, ff_mul(ff_of(evpn), Tn));
      }
    } else if (GENERAL) {
      const double nS = f64_of(normS, k20), Str = kSqrt32 * nS;
      double Sigv0, hl = 0.;
      if (m.hard.law != DNL_HARD_ELASTIC) {
        hardening_law(m.hard, evp, Sigv0, hl);
        if (Str > Sigv0 && some) {
          plastic = true;
          double gamma = (nS - kSqrt23 * Sigv0) / (m.G2 * (1.0 + hl / m.G3));
          int iteration = 0;
          for (;;) {
            double Sigv, h;
            hardening_law(m.hard, RADD(evp, RMUL(kSqrt23, gamma)), Sigv, h);
            const double dfun = kSqrt32 * m.G2 + kSqrt23 * h;
            const double fun = dfun * gamma - (Str - Sigv + h * kSqrt23 * gamma);
            if (fabs(fun / Sigv) > c_returnTol) {
              double dgamma = -fun / dfun;
              if (dgamma < 0 && fabs(dgamma) > gamma) dgamma = -gamma * 0.9;
              gamma += dgamma;
            } else {
              break;
            }
            iteration++;
            if (iteration > c_caps[1]) {
              rr_ok = false;
              break;
            }
          }
          evp = RADD(evp, RMUL(kSqrt23, gamma));
          bad |= f64_mag(gamma) >= (uint32_t)((1023 + 30) << 20);
          gi = ff_mul(ff_of(gamma), inv);
        }
      }
    }
    if (TAPE && valid && !bad) {
      a.tape[(long)TL::GAM * nIP + ipx] = gam_d;
      a.tape[(long)TL::XV * nIP + ipx] = evp;
      a.tape[(long)TL::XN * nIP + ipx] = evpn;
      a.tape[(long)TL::LXV * nIP + ipx] = lxv;
    }
  }

  // ---- the element's lanes decide together
  if constexpr (NIP > 1) {
    const unsigned mask = ((1u << NIP) - 1u) << (lane - pt);
    bad = (__ballot_sync(0xffffffffu, bad) & mask) != 0u;
  }
  const bool put = valid && !bad;
  if (put) {
    if (TWO_D && det.h < 0.f) record_error(tm, DNL_ERR_NEG_DETJ, a.eBase + e);
    if (!conv) record_error(tm, DNL_ERR_JACOBI_NOCONV, a.eBase + e);
    if (!rr_ok) record_error(tm, DNL_ERR_RR_NOCONV, a.eBase + e);
  }

  // ---- RFI: X <- R X R^T for S, Eps, EpsPlas (Element.C:386-388) as increments of the stored state
  float mq = 0.f;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      if (!TWO_D || (i == 2) == (j == 2)) mq = f_max(mq, f_abs(Q[i][j].h));
  // Increments of EpsPlas (gamma n), Eps (ln U) and S (2 G dev ln U - 2 G gamma n) before the rotation
  // wait in shared memory; one loop body then serves the three tensors (unrolled, the pass is bound by
  // fetching its instructions).  S last: its rotated value is what the forces need.
  {
    if (plastic) {
      const ff cc = ff_mul(mf.g2, gi);
#pragma unroll
      for (int k = 0; k < NS; k++) {
        hold[(0 * NS + k) * HOLD] = f2(ff_mul(gi, St[k]));
        inc[k] = ff_sub(inc[k], ff_mul(cc, St[k]));
      }
    }
#pragma unroll
    for (int k = 0; k < NS; k++) {
      hold[(1 * NS + k) * HOLD] = f2(Ln[k]);
      hold[(2 * NS + k) * HOLD] = f2(inc[k]);
    }
  }
  ff Sn[6];  // the rotated tensor; after the loop the new stress over 2^k
#pragma unroll
  for (int k = 0; k < 6; k++) Sn[k] = zero;
#pragma unroll 1
  for (int t = 0; t < 3; t++) {
    double *const X = a.ip + (long)(t == 2 ? Ly::S : (t == 1 ? Ly::EPS : Ly::EPSP)) * nIP + ipx;
    const int kt = t == 2 ? k20 : 0;
    double Xd[NS];
    uint32_t nz = 0;
#pragma unroll
    for (int k = 0; k < NS; k++) {
      Xd[k] = X[k * nIP];
      nz |= f64_mag(Xd[k]) | (uint32_t)d_bits(Xd[k]);
    }
    if (t > 0 || nz || plastic) {  // a point that never yielded has EpsPlas = 0 exactly
      ff D[6], in[6];
#pragma unroll
      for (int k = 0; k < NS; k++) {
        in[k] = t > 0 || plastic ? ff_from(hold[(t * NS + k) * HOLD]) : zero;
        Sn[k] = ff_add(ff_of(Xd[k], -kt), in[k]);
      }
      rfi_ff<TWO_D>(Q, mq, Sn, D);
#pragma unroll
      for (int k = 0; k < NS; k++) {
        if (put) X[k * nIP] = f64_add(Xd[k], ff_add(in[k], D[k]), kt);
        Sn[k] = ff_add(Sn[k], D[k]);
      }
    }
  }
  const ff pn = ff_add(ff_of(pd, -k20), pinc);
  if (put) {
    a.ip[Ly::P * nIP + ipx] = f64_add(pd, pinc, k20);
    if (plastic) {
      a.ip[Ly::EVP * nIP + ipx] = evp;
      a.ip[Ly::EVPN * nIP + ipx] = evpn;
    }
    if (a.stepT) {
#pragma unroll
      for (int k = 0; k < 9; k++) {
        a.stepT[k * nIP + ipx] = f64_of(Ln[sym_of(k / 3, k % 3)]);
        a.stepT[(9 + k) * nIP + ipx] = f64_add(k % 4 == 0 ? 1. : 0., Q[k / 3][k % 3]);
      }
      a.detJ[ipx] = f64_of(det, DIM * js * (1 << 20));
    }
  }

  // ---- forces: M = J^-1 Sig W = adj(J) Sig times the weight (and 2 pi R); J's scale goes to the end
  ff M[DIM][DIM], hoop = zero;
#pragma unroll
  for (int i = 0; i < 3; i++) Sn[i] = ff_add(Sn[i], pn);
#pragma unroll
  for (int l = 0; l < DIM; l++)
#pragma unroll
    for (int i = 0; i < DIM; i++) {
      Dot s(adj[l][0], Sn[sym_of(0, i)]);
#pragma unroll
      for (int j = 1; j < DIM; j++) s.mac(adj[l][j], Sn[sym_of(j, i)]);
      M[l][i] = s.get();
    }
  if (AXI) {
    const ff twoPiR = ff_mul(FF_CONST(kDeuxPi), Rad);
#pragma unroll
    for (int l = 0; l < DIM; l++)
#pragma unroll
      for (int i = 0; i < DIM; i++) M[l][i] = ff_mul(M[l][i], twoPiR);
    hoop = ff_mul(ff_mul(Sn[2], det), FF_CONST(kDeuxPi));  // sigma_tt / R x W, W = detJ 2 pi R
  }
  const int f20 = k20 + (DIM - 1 + (AXI ? 1 : 0)) * js * (1 << 20);  // forces' exponent: stress x length^(DIM-1)
  if constexpr (NEN == NIP) {
    // Node k's force is sum_q sum_l dN_k,l(q) M_q[l] (+ N_k(q) hoop_q).  With s_b(k) the sign of node
    // k's (and Gauss point k's) coordinate b and g = 1/sqrt(3), dN_k,l(q) = s_l(k) / 2^DIM prod_(b != l)
    // (1 + g s_b(k) s_b(q)), so over sets m of directions, with s_m the product of their signs,
    //   f_k = sum_m s_m(k) [sum_(l in m) g^(|m|-1) / 2^DIM T_l(m - l) + g^|m| / 2^DIM T_hoop(m)],
    //   T(m) = sum_q s_m(q) M_q:
    // a sign transform over the element's lanes (lane of place b <-> set b), one weight, and the
    // transform back: DIM shuffled sums each way instead of NIP DIM multiply-adds per component.
    const int place = sign_place(pt);
    auto partner = [lane, pt, place](int bit) {  // lane of the place with one bit flipped
      const int b = place ^ bit;
      return lane - pt + (b ^ ((b >> 1) & 1));
    };
    int to[DIM];
#pragma unroll
    for (int d = 0; d < DIM; d++) to[d] = partner(1 << d);
    auto get = [](ff v, int from) {
      return ff{__shfl_sync(0xffffffffu, v.h, from), __shfl_sync(0xffffffffu, v.l, from)};
    };
    // at each direction the + place takes (+) - (-), the - place their sum: entry m is T(m)
    auto transform = [&](ff v) {
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        const ff o = get(v, to[d]);
        const uint32_t f = (place >> d & 1) ? 0x80000000u : 0u;
        v = ff_add_raw(v, ff{bits_f(f_bits(o.h) ^ f), bits_f(f_bits(o.l) ^ f)});
      }
      return ff_norm(v.h, v.l);
    };
    const int pop = __popc(place);
    const ff w = c_shapeFF.gpow[DIM == 3 ? 1 : 0][pop];
    ff F[DIM];
#pragma unroll
    for (int i = 0; i < DIM; i++) F[i] = zero;
#pragma unroll
    for (int l = 0; l < DIM; l++)
#pragma unroll
      for (int i = 0; i < DIM; i++) {
        // weighted where it is formed (its set lacks l, so the target's |m| - 1 is its own count)
        const ff o = get(ff_mul(transform(M[l][i]), w), to[l]);
        const bool in = place >> l & 1;
        F[i] = ff_add_raw(F[i], in ? o : zero);
      }
    if (AXI) F[0] = ff_add_raw(F[0], ff_mul(transform(hoop), w));
    // back: f_k = sum_m s_m(k) F(m); s_d(k) = +1 at the places with bit d
#pragma unroll
    for (int i = 0; i < DIM; i++) {
      ff v = ff_norm(F[i].h, F[i].l);
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        const ff o = get(v, to[d]);
        // (without d) + s_d (with d): + places hold "with", - places "without"
        const uint32_t f = (place >> d & 1) ? 0u : 0x80000000u;
        v = ff_add_raw(ff{v.h, v.l}, ff{bits_f(f_bits(o.h) ^ f), bits_f(f_bits(o.l) ^ f)});
      }
      if (put) a.fe[(long)i * a.feStride + (long)e * NEN + pt] = f64_of(ff_neg(ff_norm(v.h, v.l)), f20);
    }
  } else if constexpr (ET == DNL_ELTET4N3D) {
    // dN/dxi of the nodes 1, 2, 3 are the unit vectors, of node 0 minus their sum; weight 1/6
#pragma unroll
    for (int i = 0; i < 3; i++) {
      ff m[3];
#pragma unroll
      for (int l = 0; l < 3; l++) m[l] = ff_mul(M[l][i], FF_CONST(1. / 6.));
      if (put) {
#pragma unroll
        for (int l = 0; l < 3; l++) a.fe[(long)i * a.feStride + (long)e * NEN + l + 1] = f64_of(ff_neg(m[l]), f20);
        a.fe[(long)i * a.feStride + (long)e * NEN] = f64_of(ff_add(ff_add(m[0], m[1]), m[2]), f20);
      }
    }
  } else {
    // the one-point hexahedron: weight 8 and dN/dxi = +-1/8, so node k's internal force is
    // sum_l xi_l(k) M[l].  Hourglass control (see elem_ip): with h_a the node signs' products, hx_a and
    // hv_a their sums over x and v, g_ak = h_ak - hx_a . b_k and b_k = J^-T xi(k) / 8,
    //   q_a = g_a . v = hv_a - (grad v) hx_a,
    //   sum_a g_ak q_a = sum_a h_ak q_a - sum_l xi_l(k) / 8 (J^-1 P)_l,  P = sum_a hx_a (x) q_a:
    // all of it coefficients of one inverse transform over the nodes.  Lengths over 2^js.
    int nd[8];
#pragma unroll
    for (int k = 0; k < 8; k++) nd[k] = __ldg(a.conn + (long)k * a.E + e);
    ff q[4][3], gv[3][3];
    int jv[3];  // velocities' component r is over 2^jv[r]
#pragma unroll
    for (int r = 0; r < 3; r++) {
      ff w[8];
      double d[8];
      jv[r] = (int)(rel_first(a.v[r], nd, d) >> 20) - 1023;
      walsh_of(d, -jv[r] * (1 << 20), w);
      q[0][r] = w[3];
      q[1][r] = w[6];
      q[2][r] = w[5];
      q[3][r] = ff_neg(w[7]);
#pragma unroll
      for (int c = 0; c < 3; c++) gv[r][c] = ff_scale(ff_neg(w[1 << c]), 0.125f);
    }
    // grad v = gv J^-1 (times 2^-js), q_a = hv_a - grad v hx_a
    ff Ji[3][3];
#pragma unroll
    for (int l = 0; l < 3; l++)
#pragma unroll
      for (int c = 0; c < 3; c++) Ji[l][c] = ff_mul(adj[l][c], rdet);
#pragma unroll
    for (int r = 0; r < 3; r++) {
      ff g[3];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        ff t = ff_mul(gv[r][0], Ji[0][i]);
        t = ff_add(t, ff_mul(gv[r][1], Ji[1][i]));
        g[i] = ff_add(t, ff_mul(gv[r][2], Ji[2][i]));
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        ff t = ff_mul(g[0], hg.x[k][0]);
        t = ff_add(t, ff_mul(g[1], hg.x[k][1]));
        t = ff_add(t, ff_mul(g[2], hg.x[k][2]));
        q[k][r] = ff_sub(q[k][r], t);
      }
    }
    // a_h = coefficient rho c V^(2/3) / 4 over 2^k, V = 8 detJ; the volume's sign does not matter
    // (an element that is turned inside out or numbered the other way round is no error in 3D)
    const ff vol = ff_scale(det.h < 0.f ? ff_neg(det) : det, 8.f);
    const ff ah0 = ff_mul(ff_mul(mf.rhoCs4, ff_of(a.hourglass)), pow23_ff(vol));
#pragma unroll
    for (int r = 0; r < 3; r++) {
      // M and the hourglass part are added over 2^ef, the larger one's power of two, so that either alone
      // keeps its precision however small it is against 2^k
      ff P[3], F[8];
      const float mM = f_max(f_abs(M[0][r].h), f_max(f_abs(M[1][r].h), f_abs(M[2][r].h)));
      const int ef = max((int)(f_bits(mM) >> 23) - 127, jv[r]);
      const float sM = bits_f((uint32_t)(127 - ef) << 23), sv = jv[r] - ef < -100 ? 0.f : bits_f((uint32_t)(127 + jv[r] - ef) << 23);
      const ff ah = ff_scale(ah0, sv);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        ff t = ff_mul(hg.x[0][i], q[0][r]);
#pragma unroll
        for (int k = 1; k < 4; k++) t = ff_add(t, ff_mul(hg.x[k][i], q[k][r]));
        P[i] = t;
      }
#pragma unroll
      for (int l = 0; l < 3; l++) {
        ff t = ff_mul(Ji[l][0], P[0]);
        t = ff_add(t, ff_mul(Ji[l][1], P[1]));
        t = ff_add(t, ff_mul(Ji[l][2], P[2]));
        F[1 << l] = ff_neg(ff_sub(ff_scale(M[l][r], sM), ff_scale(ff_mul(ah, t), 0.125f)));
      }
      F[3] = ff_mul(ah, q[0][r]);
      F[6] = ff_mul(ah, q[1][r]);
      F[5] = ff_mul(ah, q[2][r]);
      F[7] = ff_neg(ff_mul(ah, q[3][r]));
      walsh8(F);
      if (put) {
#pragma unroll
        for (int k = 0; k < 8; k++) a.fe[(long)r * a.feStride + (long)e * NEN + k] = f64_of(ff_neg(ff_norm(F[sign_place(k)].h, F[sign_place(k)].l)), f20 + ef * (1 << 20));
      }
    }
  }
  return bad;
}

static void set_tables_ff(const double (&axN)[3], const double (&axD)[2], const double (&hxD)[3])
{
  ShapeFF f;
  for (int i = 0; i < 3; i++) f.axN[i] = ff_host(axN[i]);
  for (int i = 0; i < 2; i++) f.axD[i] = ff_host(axD[i]);
  for (int i = 0; i < 3; i++) f.hxD[i] = ff_host(hxD[i]);
  for (int c = 0; c < 4; c++) {
    f.gpow[0][c] = ff_host(0.25 * pow(3.0, -0.5 * c));
    f.gpow[1][c] = ff_host(0.125 * pow(3.0, -0.5 * c));
  }
  cudaMemcpyToSymbol(c_shapeFF, &f, sizeof f);
}

static bool set_tolerances_ff(double polar, double radial)
{
  TolFF t;
  t.polar = ff_host(polar);
  t.ok = polar >= 0x1p-52 && polar <= 0x1p-29 && radial >= 0x1p-44;
  return cudaMemcpyToSymbol(c_tolFF, &t, sizeof t) == cudaSuccess;
}
