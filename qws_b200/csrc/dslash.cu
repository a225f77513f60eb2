// Wilson-clover hopping kernels for the DD solver (FP64, FP32, and FP16
// storage with FP32 arithmetic).
//
// One templated kernel covers every operator the reference spreads over
// ddd_in_*, ddd_out_pre/pos_*, jinv_ddd_in_s_ and the SAP update loops:
//   SEL  which hops:  inner (stay inside the SAP block; ddd_in, open block
//        faces, ddd_in_d.cc:91-190), outer (cross a block face; the
//        reference's halo path ddd_out_*), or all (ddd_d_/ddd_s_).
//   EPI  what is done with acc = A^-1 * (sum of selected hops):
//        EPI_D    out = src - kappa*acc                (ddd_in / D)
//        EPI_ADD  out += coef*acc                      (ddd_out_pos, factor coef)
//        EPI_JINV out = aux + kappa*acc                (one Richardson step
//                 x <- b + kappa A^-1 H_blk x, algebraically the reference's
//                 x + (b - D_blk x), static_solver.cc:77-139)
//        EPI_SAPE out = out + (aux - (src - kappa*acc)) (s_e += in_e - D_blk a_e,
//                 qws.cc:815-818 with the ddd_in result kept in registers; with
//                 all hops also s_e += kappa A^-1 H_face a, see sap_t)
//   T    storage format (float, double, H16); arithmetic in Arith<T>::R.
// Faces are not packed: a face hop reads the neighbouring block's site of
// the source field directly from HBM (the whole lattice is resident).
#include <type_traits>

#include "kernels.h"
#include "lattice.cuh"

namespace qwsg {

// How a thread's values map to memory.  Scalar: one (site, RHS) entry per
// thread in the storage format's own layout.  Pair (FP16 multi-RHS fields):
// two RHS of one site per thread as F2 lanes, IOP layout.
template <typename T>
struct OneRhs {
  using V = typename Arith<T>::R;
  using S = typename Store<T>::type;
  __device__ __forceinline__ static int lanes_log(const Geom& G) { return G.lgnr; }
  __device__ __forceinline__ static int pad(const Geom& G) { return spad(G); }
  __device__ __forceinline__ static int entry(const Geom& G, int g, int lane) { return sentry(G, g, lane); }
  __device__ __forceinline__ static void load_raw(const S* p, int pd, int e, V v[24], V& s) {
    IO<T>::load_spinor_raw(p, pd, e, v, s);
  }
  __device__ __forceinline__ static void load_half_raw(const S* p, int pd, int e, int up, V v[24], V& s) {
    IO<T>::load_half_raw(p, pd, e, up, v, s);
  }
  __device__ __forceinline__ static void load(const S* p, int pd, int e, V v[24]) {
    IO<T>::load_spinor(p, pd, e, v);
  }
  __device__ __forceinline__ static void store(S* p, int pd, int e, const V v[24]) {
    IO<T>::store_spinor(p, pd, e, v);
  }
  // A^-1 v with the site's clover, or the entry's (PRK: per-RHS kappa)
  template <bool PRK>
  __device__ __forceinline__ static void clover(const HopArgs<T>& a, int g, int lane, V v[24]) {
    if constexpr (PRK)
      clover_apply<T, V>(a.Cr, spad(a.G), sentry(a.G, g, lane), v);
    else
      clover_apply<T, V>(a.C, a.G.pad, g, v);
  }
  template <bool PRK>
  __device__ __forceinline__ static V coef(const HopArgs<T>& a, int lane) {
    if constexpr (PRK) return copysign(a.kap[lane], a.coef);
    return a.coef;
  }
};
struct TwoRhs {
  using V = F2;
  using S = __half;
  __device__ __forceinline__ static int lanes_log(const Geom& G) { return G.lgnr - 1; }
  __device__ __forceinline__ static int pad(const Geom& G) { return spad(G) >> 1; }
  __device__ __forceinline__ static int entry(const Geom& G, int g, int lane) {
    return (g << (G.lgnr - 1)) + lane;
  }
  __device__ __forceinline__ static void load_raw(const S* p, int pd, int e, V v[24], V& s) {
    IOP::load_spinor_raw(p, pd, e, v, s);
  }
  __device__ __forceinline__ static void load_half_raw(const S* p, int pd, int e, int up, V v[24], V& s) {
    IOP::load_half_raw(p, pd, e, up, v, s);
  }
  __device__ __forceinline__ static void load(const S* p, int pd, int e, V v[24]) {
    IOP::load_spinor(p, pd, e, v);
  }
  __device__ __forceinline__ static void store(S* p, int pd, int e, const V v[24]) {
    IOP::store_spinor(p, pd, e, v);
  }
  // the site's clover for both lanes, or each lane's own (PRK: per-RHS kappa)
  template <bool PRK>
  __device__ __forceinline__ static void clover(const HopArgs<H16>& a, int g, int lane, V v[24]) {
    if constexpr (PRK) {
      const int sp = spad(a.G), e0 = sentry(a.G, g, 2 * lane);
      clover_apply_with<F2>(
          [&](int i, F2 c[36]) {
            float s0[36], s1[36];
            IO<H16>::load_clover_block(a.Cr, sp, e0, i, s0);
            IO<H16>::load_clover_block(a.Cr, sp, e0 + 1, i, s1);
#pragma unroll
            for (int k = 0; k < 36; k++) c[k] = F2{s0[k], s1[k]};
          },
          v);
    } else {
      clover_apply<H16, F2>(a.C, a.G.pad, g, v);
    }
  }
  template <bool PRK>
  __device__ __forceinline__ static V coef(const HopArgs<H16>& a, int lane) {
    if constexpr (PRK)
      return F2{copysignf(a.kap[2 * lane], a.coef), copysignf(a.kap[2 * lane + 1], a.coef)};
    return Lanes<F2>::bcast(a.coef);
  }
};

template <typename T, typename P, int SEL, int MU, int DIR, typename V = typename P::V>
__device__ __forceinline__ void do_hop(const HopArgs<T>& a, const Site& s, int g, int lane,
                                       V acc[24]) {
  using R = typename Arith<T>::R;
  const bool face = DIR > 0 ? (s.lc[MU] == a.G.B[MU] - 1) : (s.lc[MU] == 0);
  if (face) {
    if (!(SEL & HOP_OUTER)) return;
  } else {
    if (!(SEL & HOP_INNER)) return;
  }
  int gn;
  if (!face) {
    gn = g + rot_step(a.G, MU, s.lc[MU], DIR);
  } else {
    int ncol;
    gn = nbr_across(a.G, s, MU, DIR, &ncol);
    if (ncol == a.zero_col) return;  // that colour's source is defined as zero
  }
  V v[24], sc;
  const int pd = P::pad(a.G), en = P::entry(a.G, gn, lane);
  // the projection and the link product are linear: the source's scale
  // (FP16 storage) is applied once, in the reconstruction
  if (MU == 3)
    P::load_half_raw(a.src, pd, en, DIR > 0, v, sc);
  else
    P::load_raw(a.src, pd, en, v, sc);
  V h[12], r[12], ul[18];
  project<V, MU, DIR>(v, h);
  {
    R u[18];
    if constexpr (std::is_same<T, float>::value) {
      if (a.U12)
        load_link12(a.U12, a.G.pad, MU, DIR > 0 ? g : gn, u);
      else
        IO<T>::load_link(a.U, a.G.pad, MU, DIR > 0 ? g : gn, u);
    } else {
      IO<T>::load_link(a.U, a.G.pad, MU, DIR > 0 ? g : gn, u);
    }
#pragma unroll
    for (int e = 0; e < 18; e++) ul[e] = Lanes<V>::bcast(u[e]);
  }
  if (DIR > 0)
    link_mul<V, false>(ul, h, r);
  else
    link_mul<V, true>(ul, h, r);
  V f = sc;
  if (MU == 3) {
    f = Lanes<V>::bcast((R)2) * sc;
    if (face && (DIR > 0 ? s.bc[3] == a.G.NB[3] - 1 : s.bc[3] == 0))
      f = Lanes<V>::bcast((R)(2 * a.G.tbc)) * sc;
  }
  reconstruct<V, MU, DIR>(r, acc, f);
}

// The FP32 block and face kernels and the FP16 block kernels are held to
// 64 registers (4 CTAs of 256 or 8 of 128 threads per SM): more warps in
// flight hide more of the neighbour-load latency that bounds them (FP32
// Richardson step 7% faster, FP16 SAP 4-8%); the full-lattice FP32
// operator and the FP16 face kernel spill at that bound and keep theirs.
template <typename T, int SEL>
struct MinCtas {
  static constexpr int value =
      ((std::is_same<T, float>::value && SEL != HOP_ALL) || (std::is_same<T, H16>::value && SEL == HOP_INNER))
          ? 4
          : 1;
};

template <typename T, typename P, int SEL, int EPI, bool PRK>
__device__ __forceinline__ void hop_site_at(const HopArgs<T>& a, const int i) {
  using V = typename P::V;
  const int ll = P::lanes_log(a.G);
  if (i >= (a.nsites << ll)) return;
  // consecutive threads: the right-hand sides (or RHS pairs) of one site,
  // then the next site
  const int si = i >> ll, lane = i & ((1 << ll) - 1);
  const int g = a.list ? __ldg(a.list + si) : a.site0 + si;
  Site s;
  decode_site(a.G, g, s);
  if (a.dom >= 0 && (s.bc[0] & 1) != a.dom) return;
  if (SEL == HOP_OUTER) {
    bool face = false;
#pragma unroll
    for (int mu = 0; mu < 4; mu++) face |= (s.lc[mu] == 0) | (s.lc[mu] == a.G.B[mu] - 1);
    if (!face) return;
  }
  V acc[24];
#pragma unroll
  for (int j = 0; j < 24; j++) acc[j] = Lanes<V>::bcast((typename Arith<T>::R)0);
  do_hop<T, P, SEL, 0, +1>(a, s, g, lane, acc);
  do_hop<T, P, SEL, 0, -1>(a, s, g, lane, acc);
  do_hop<T, P, SEL, 1, +1>(a, s, g, lane, acc);
  do_hop<T, P, SEL, 1, -1>(a, s, g, lane, acc);
  do_hop<T, P, SEL, 2, +1>(a, s, g, lane, acc);
  do_hop<T, P, SEL, 2, -1>(a, s, g, lane, acc);
  do_hop<T, P, SEL, 3, +1>(a, s, g, lane, acc);
  do_hop<T, P, SEL, 3, -1>(a, s, g, lane, acc);
  P::template clover<PRK>(a, g, lane, acc);
  const int pd = P::pad(a.G), e = P::entry(a.G, g, lane);
  const V coef = P::template coef<PRK>(a, lane);
  V o[24];
  if (EPI == EPI_D) {
    P::load(a.src, pd, e, o);
#pragma unroll
    for (int j = 0; j < 24; j++) o[j] = madd(coef, acc[j], o[j]);
  } else if (EPI == EPI_ADD) {
    P::load(a.out, pd, e, o);
#pragma unroll
    for (int j = 0; j < 24; j++) o[j] = madd(coef, acc[j], o[j]);
  } else if (EPI == EPI_JINV) {
    P::load(a.aux, pd, e, o);
#pragma unroll
    for (int j = 0; j < 24; j++) o[j] = madd(coef, acc[j], o[j]);
  } else {  // EPI_SAPE: coef = -kappa
    V in[24], av[24];
    P::load(a.sin ? a.sin : a.out, pd, e, o);
    P::load(a.aux, pd, e, in);
    P::load(a.src, pd, e, av);
#pragma unroll
    for (int j = 0; j < 24; j++) o[j] = o[j] + (in[j] - madd(coef, acc[j], av[j]));
  }
  P::store(a.out, pd, e, o);
}

template <typename T, typename P, int SEL, int EPI, bool PRK>
__device__ __forceinline__ void hop_site(const HopArgs<T>& a) {
  hop_site_at<T, P, SEL, EPI, PRK>(a, blockIdx.x * blockDim.x + threadIdx.x);
}

// the same body with and without the 64-register bound (an explicit
// minimum of one CTA per SM would let the compiler spend every register)
// PRK: per-RHS kappa (clover planes and kappa per RHS, multi-RHS handles only)
template <typename T, int SEL, int EPI, bool PRK>
__global__ void __launch_bounds__(256) k_hop(const HopArgs<T> a) {
  hop_site<T, OneRhs<T>, SEL, EPI, PRK>(a);
}
template <typename T, int SEL, int EPI, bool PRK>
__global__ void __launch_bounds__(256, 4) k_hop_r64(const HopArgs<T> a) {
  hop_site<T, OneRhs<T>, SEL, EPI, PRK>(a);
}
// The full-lattice operators at a register bound of their own: FP64 at 128
// registers (4 CTAs of 128 threads per SM instead of 3; 56 bytes spill) and
// FP32 at 72 with CTAs of 128 (7 CTAs instead of 6): 13 % and 3 % faster
// at 32^3x64; the FP16 face kernel at 72 too (7 instead of 6, ~5 % faster).
// Bit for bit the same results.  (The FP16 block kernels at 56 registers,
// 9 CTAs, ran 5 % slower than at 64.)
template <typename T, int SEL, int EPI, bool PRK>
__global__ void __launch_bounds__(256, 2) k_hop_r128(const HopArgs<T> a) {
  hop_site<T, OneRhs<T>, SEL, EPI, PRK>(a);
}
template <typename T, int SEL, int EPI, bool PRK>
__global__ void __launch_bounds__(128, 7) k_hop_r73(const HopArgs<T> a) {
  hop_site<T, OneRhs<T>, SEL, EPI, PRK>(a);
}
// FP16 fields with two or more RHS: two RHS per thread in packed FP32x2
// arithmetic (the link and clover of the site serve both lanes)
template <int SEL, int EPI, bool PRK>
__global__ void __launch_bounds__(256) k_hop_pair(const HopArgs<H16> a) {
  hop_site<H16, TwoRhs, SEL, EPI, PRK>(a);
}

// ---------------------------------------------------------------------------
// Four threads per site (one RHS; FP32 and FP16): a CTA of four warps handles
// 32 sites.  Warp w first computes the two hops along direction w (projection
// and link product), then owns spin w: it adds the eight hops' contributions
// to that spin, makes three rows of A^-1 x and writes the spin's six reals.
// What the warps exchange goes through shared memory.  Every sum runs in the
// order of hop_site_at, so the results are bit for bit the same.
//
// For launches that leave the chip underfilled, where the time is one thread's
// chain of loads and its ~1,900 instructions: a quarter of the chain per
// thread and four times the warps.
// ---------------------------------------------------------------------------
// Most sites of such a launch.  Measured per SAP application (one thread ->
// four threads a site): FP32 at 2,048 sites a launch 188 -> 98 us, 20,736:
// 224 -> 173, 27,440: 242 -> 213, 38,416: 265 -> 281 (D alone at 30,240 sites
// 10.2 -> 9.0, at 38,416 10.4 -> 12.2); FP16 (more instructions
// a site, so an SM fills earlier) 150 -> 102, 190 -> 172, 198 -> 207,
// 222 -> 268.
template <typename T>
constexpr int kSplitSites = std::is_same<T, H16>::value ? 148 * 144 : 148 * 216;
struct SplitShared {
  float2 r[8][6][32];   // hop 2 mu + (dir < 0): link product, [2 colour + k]
  float f[8][32];       // and its factor (0: the hop does not count)
  float2 x[4][3][32];   // summed spins, [spin][colour]
  float2 y[2][6][32];   // A^-1 x of the two chiral blocks
  float m[4][32];       // FP16 storage: largest component of each spin
};

// link product of one hop into shared memory
template <typename T, int SEL, int MU, int DIR>
__device__ __forceinline__ void split_hop(const HopArgs<T>& a, const Site& s, int g, bool live,
                                          int lane, SplitShared& sh) {
  constexpr int k = 2 * MU + (DIR < 0);
  const bool face = DIR > 0 ? (s.lc[MU] == a.G.B[MU] - 1) : (s.lc[MU] == 0);
  bool on = live && (face ? (SEL & HOP_OUTER) != 0 : (SEL & HOP_INNER) != 0);
  int gn = g;
  if (on) {
    if (!face) {
      gn = g + rot_step(a.G, MU, s.lc[MU], DIR);
    } else {
      int ncol;
      gn = nbr_across(a.G, s, MU, DIR, &ncol);
      on = ncol != a.zero_col;
    }
  }
  float r[12], f = 0;
  if (on) {
    float v[24], sc, h[12], u[18];
    if (MU == 3)
      IO<T>::load_half_raw(a.src, a.G.pad, gn, DIR > 0, v, sc);
    else
      IO<T>::load_spinor_raw(a.src, a.G.pad, gn, v, sc);
    if constexpr (std::is_same<T, float>::value) {
      if (a.U12)
        load_link12(a.U12, a.G.pad, MU, DIR > 0 ? g : gn, u);
      else
        IO<T>::load_link(a.U, a.G.pad, MU, DIR > 0 ? g : gn, u);
    } else {
      IO<T>::load_link(a.U, a.G.pad, MU, DIR > 0 ? g : gn, u);
    }
    project<float, MU, DIR>(v, h);
    if (DIR > 0)
      link_mul<float, false>(u, h, r);
    else
      link_mul<float, true>(u, h, r);
    f = sc;
    if (MU == 3) {
      f = 2.0f * sc;
      if (face && (DIR > 0 ? s.bc[3] == a.G.NB[3] - 1 : s.bc[3] == 0))
        f = (float)(2 * a.G.tbc) * sc;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 12; j++) r[j] = 0;
  }
#pragma unroll
  for (int j = 0; j < 6; j++) sh.r[k][j][lane] = make_float2(r[2 * j], r[2 * j + 1]);
  sh.f[k][lane] = f;
}

// the contribution of hop (MU, DIR) to spin SPIN (the rows of reconstruct)
template <int SPIN, int MU, int DIR>
__device__ __forceinline__ void split_add(const SplitShared& sh, int lane, float acc[6]) {
  if (MU == 3 && (DIR > 0 ? SPIN < 2 : SPIN >= 2)) return;
  constexpr int hop = 2 * MU + (DIR < 0);
  // which of the two projected spins, and as it is (+-1) or times +-i
  constexpr int k = SPIN < 2 || MU == 3 ? SPIN & 1 : MU == 2 ? SPIN - 2 : 3 - SPIN;
  constexpr bool times_i = SPIN >= 2 && (MU == 0 || MU == 2);
  constexpr int up = DIR > 0 ? 1 : -1;
  constexpr int sgn = SPIN < 2 || MU == 3 ? 1
                      : MU == 0           ? up
                      : MU == 1           ? (SPIN == 2 ? up : -up)
                                          : (SPIN == 2 ? up : -up);
  const float f = sh.f[hop][lane], p = sgn > 0 ? f : -f;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const float2 r = sh.r[hop][2 * c + k][lane];
    if (times_i) {
      acc[2 * c] = madd(-p, r.y, acc[2 * c]);
      acc[2 * c + 1] = madd(p, r.x, acc[2 * c + 1]);
    } else {
      acc[2 * c] = madd(p, r.x, acc[2 * c]);
      acc[2 * c + 1] = madd(p, r.y, acc[2 * c + 1]);
    }
  }
}
template <int SPIN>
__device__ __forceinline__ void split_sum(const SplitShared& sh, int lane, float acc[6]) {
#pragma unroll
  for (int j = 0; j < 6; j++) acc[j] = 0;
  split_add<SPIN, 0, +1>(sh, lane, acc);
  split_add<SPIN, 0, -1>(sh, lane, acc);
  split_add<SPIN, 1, +1>(sh, lane, acc);
  split_add<SPIN, 1, -1>(sh, lane, acc);
  split_add<SPIN, 2, +1>(sh, lane, acc);
  split_add<SPIN, 2, -1>(sh, lane, acc);
  split_add<SPIN, 3, +1>(sh, lane, acc);
  split_add<SPIN, 3, -1>(sh, lane, acc);
}

// rows 3 H .. 3 H + 2 of A x, A the Hermitian block a (clover_apply_with's
// order: for row j the columns 0 .. 5 but j, after the diagonal)
template <int H>
__device__ __forceinline__ void split_clover(const float a[36], const float2 x[6], float2 y[3]) {
#pragma unroll
  for (int q = 0; q < 3; q++) {
    constexpr int kFirst = 3 * H;
    const int j = kFirst + q;
    float yr = a[j] * x[j].x, yi = a[j] * x[j].y;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      if (k == j) continue;
      const int lo = k < j ? k : j, hi = k < j ? j : k;
      const int n = lo * 5 - lo * (lo - 1) / 2 + (hi - lo - 1);  // pair (lo, hi)
      const float mr = a[6 + 2 * n], mi = a[7 + 2 * n], nmi = -a[7 + 2 * n];
      yr = madd(mr, x[k].x, yr);
      yr = madd(k < j ? mi : nmi, x[k].y, yr);
      yi = madd(mr, x[k].y, yi);
      yi = madd(k < j ? nmi : mi, x[k].x, yi);
    }
    y[q] = make_float2(yr, yi);
  }
}

// the six reals of one spin of an FP32 or FP16 spinor, as stored, and the
// site's scale
template <typename T>
struct SpinIO;
template <>
struct SpinIO<float> {
  __device__ __forceinline__ static void load(const float* p, int pad, int g, int spin, float v[6],
                                              float& s) {
    s = 1.0f;
    const float2* q = reinterpret_cast<const float2*>(p);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float2 t = __ldg(q + 2 * ((size_t)(2 * c + (spin >> 1)) * pad + g) + (spin & 1));
      v[2 * c] = t.x;
      v[2 * c + 1] = t.y;
    }
  }
};
template <>
struct SpinIO<H16> {
  // 4-byte word of (colour, spin) of site g in the IO<H16> planes
  __device__ __forceinline__ static size_t word(int pad, int g, int spin, int c) {
    return c < 2 ? 4 * ((size_t)(spin >> 1) * pad + g) + 2 * c + (spin & 1)
                 : 4 * ((size_t)2 * pad + g) + spin;
  }
  __device__ __forceinline__ static void load(const __half* p, int pad, int g, int spin, float v[6],
                                              float& s) {
    s = IO<H16>::scale(p, pad, g);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const unsigned w = __ldg(reinterpret_cast<const unsigned*>(p) + word(pad, g, spin, c));
      __half2 h;
      memcpy(&h, &w, 4);
      const float2 t = __half22float2(h);
      v[2 * c] = t.x;
      v[2 * c + 1] = t.y;
    }
  }
};

template <typename T, int SEL, int EPI>
__global__ void __launch_bounds__(128) k_hop_split(const HopArgs<T> a) {
  __shared__ SplitShared sh;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  bool live = i < a.nsites;
  const int ii = live ? i : a.nsites - 1;  // (a valid site for the idle lanes)
  const int g = a.list ? __ldg(a.list + ii) : a.site0 + ii;
  const int pad = a.G.pad;
  Site s;
  decode_site(a.G, g, s);
  if (a.dom >= 0 && (s.bc[0] & 1) != a.dom) live = false;
  if (SEL == HOP_OUTER) {
    bool face = false;
#pragma unroll
    for (int mu = 0; mu < 4; mu++) face |= (s.lc[mu] == 0) | (s.lc[mu] == a.G.B[mu] - 1);
    live = live && face;
  }
  switch (w) {
    case 0:
      split_hop<T, SEL, 0, +1>(a, s, g, live, lane, sh);
      split_hop<T, SEL, 0, -1>(a, s, g, live, lane, sh);
      break;
    case 1:
      split_hop<T, SEL, 1, +1>(a, s, g, live, lane, sh);
      split_hop<T, SEL, 1, -1>(a, s, g, live, lane, sh);
      break;
    case 2:
      split_hop<T, SEL, 2, +1>(a, s, g, live, lane, sh);
      split_hop<T, SEL, 2, -1>(a, s, g, live, lane, sh);
      break;
    default:
      split_hop<T, SEL, 3, +1>(a, s, g, live, lane, sh);
      split_hop<T, SEL, 3, -1>(a, s, g, live, lane, sh);
  }
  // this warp's chiral block and the epilogue's operands, while the others hop
  const int blk = w >> 1;
  float cl[36], o[6], in[6], av[6], so, si, sa;
  if (blk == 0)
    IO<T>::load_clover_block(a.C, pad, g, 0, cl);
  else
    IO<T>::load_clover_block(a.C, pad, g, 1, cl);
  SpinIO<T>::load(EPI == EPI_D ? a.src : EPI == EPI_JINV ? a.aux : EPI == EPI_SAPE && a.sin ? a.sin
                                                                                        : a.out,
                  pad, g, w, o, so);
  if (EPI == EPI_SAPE) {
    SpinIO<T>::load(a.aux, pad, g, w, in, si);
    SpinIO<T>::load(a.src, pad, g, w, av, sa);
  }
  __syncthreads();
  float acc[6];
  switch (w) {
    case 0: split_sum<0>(sh, lane, acc); break;
    case 1: split_sum<1>(sh, lane, acc); break;
    case 2: split_sum<2>(sh, lane, acc); break;
    default: split_sum<3>(sh, lane, acc);
  }
#pragma unroll
  for (int c = 0; c < 3; c++) sh.x[w][c][lane] = make_float2(acc[2 * c], acc[2 * c + 1]);
  __syncthreads();
  float2 x[6], y[3];
#pragma unroll
  for (int j = 0; j < 6; j++) {  // rows 0-2: s0 +- s2, rows 3-5: s1 +- s3
    const float2 p = sh.x[j / 3][j % 3][lane], q = sh.x[2 + j / 3][j % 3][lane];
    x[j] = blk == 0 ? make_float2(p.x + q.x, p.y + q.y) : make_float2(p.x - q.x, p.y - q.y);
  }
  if ((w & 1) == 0)
    split_clover<0>(cl, x, y);
  else
    split_clover<1>(cl, x, y);
#pragma unroll
  for (int c = 0; c < 3; c++) sh.y[blk][3 * (w & 1) + c][lane] = y[c];
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const float2 p = sh.y[1 - blk][3 * (w & 1) + c][lane];
    acc[2 * c] = blk == 0 ? y[c].x + p.x : p.x - y[c].x;
    acc[2 * c + 1] = blk == 0 ? y[c].y + p.y : p.y - y[c].y;
  }
#pragma unroll
  for (int j = 0; j < 6; j++) {
    if (EPI == EPI_SAPE) {  // (the roundings hop_site_at's expression comes out with)
      const float m = madd(a.coef, acc[j], __fmul_rn(av[j], sa));
      o[j] = __fmaf_rn(o[j], so, __fmaf_rn(in[j], si, -m));
    } else {
      o[j] = madd(a.coef, acc[j], __fmul_rn(o[j], so));
    }
  }
  if constexpr (std::is_same<T, float>::value) {
    if (!live) return;
    float2* q = reinterpret_cast<float2*>(a.out);
#pragma unroll
    for (int c = 0; c < 3; c++)
      q[2 * ((size_t)(2 * c + blk) * pad + g) + (w & 1)] = make_float2(o[2 * c], o[2 * c + 1]);
  } else {  // IO<H16>::store_spinor
    float n = 0;
#pragma unroll
    for (int j = 0; j < 6; j++) n = fmaxf(n, fabsf(o[j]));
    sh.m[w][lane] = n;
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int k = 0; k < 4; k++) n = fmaxf(n, sh.m[k][lane]);
    const bool keep = n >= 1e-30f;
    const float inv = keep ? 1.0f / n : 0.0f;
    unsigned* q = reinterpret_cast<unsigned*>(a.out);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const __half2 h = __floats2half2_rn(o[2 * c] * inv, o[2 * c + 1] * inv);
      unsigned t;
      memcpy(&t, &h, 4);
      q[SpinIO<H16>::word(pad, g, w, c)] = t;
    }
    if (w == 0)
      reinterpret_cast<float*>(reinterpret_cast<uint4*>(a.out) + (size_t)3 * pad)[g] = keep ? n : 0.0f;
  }
}

// Several lattices in one launch (a group solve; one right-hand side each):
// block b runs threads [(b - starts[l]) * blockDim, ...) of member l's own
// launch, with l's arguments copied into shared memory first.  Every member's
// result is bit for bit that of its own launch: the same body, or, where its
// own launch is small enough for k_hop_split, that kernel's sums in the same
// order (a group's launch is large where its members' are small, so here one
// thread takes a site).
template <typename T, int SEL, int EPI>
__device__ __forceinline__ void hop_multi_body(const HopArgs<T>* __restrict__ args,
                                               const int* __restrict__ starts, int n) {
  __shared__ HopArgs<T> sa;
  const int l = group_member(starts, n, blockIdx.x);
  group_load_args(sa, args + l);
  hop_site_at<T, OneRhs<T>, SEL, EPI, false>(sa, (blockIdx.x - starts[l]) * blockDim.x +
                                                     threadIdx.x);
}
template <typename T, int SEL, int EPI>
__global__ void __launch_bounds__(256) k_hop_multi(const HopArgs<T>* __restrict__ args,
                                                   const int* __restrict__ starts, int n) {
  hop_multi_body<T, SEL, EPI>(args, starts, n);
}
template <typename T, int SEL, int EPI>
__global__ void __launch_bounds__(256, 4) k_hop_multi_r64(const HopArgs<T>* __restrict__ args,
                                                          const int* __restrict__ starts, int n) {
  hop_multi_body<T, SEL, EPI>(args, starts, n);
}

template <typename T, int SEL, int EPI, bool PRK>
static void launch_v(const HopArgs<T>& a, cudaStream_t st) {
  const int threads = a.G.hop_threads;
  if constexpr (std::is_same<T, H16>::value) {
    if (a.G.nr >= 2) {
      const int blocks = ((a.nsites << (a.G.lgnr - 1)) + threads - 1) / threads;
      k_hop_pair<SEL, EPI, PRK><<<blocks, threads, 0, st>>>(a);
      return;
    }
  }
  if constexpr (!PRK && !std::is_same<T, double>::value) {
    if (a.G.nr == 1 && a.nsites <= kSplitSites<T>) {
      k_hop_split<T, SEL, EPI><<<(a.nsites + 31) / 32, 128, 0, st>>>(a);
      return;
    }
  }
  const int blocks = ((a.nsites << a.G.lgnr) + threads - 1) / threads;
  if constexpr (SEL == HOP_ALL && !PRK && std::is_same<T, double>::value) {
    k_hop_r128<T, SEL, EPI, PRK><<<blocks, threads, 0, st>>>(a);
    return;
  }
  if constexpr (!PRK && ((SEL == HOP_ALL && std::is_same<T, float>::value) ||
                         (SEL != HOP_INNER && std::is_same<T, H16>::value))) {
    if (threads == 128) {  // (the bound assumes CTAs of at most 128 threads)
      k_hop_r73<T, SEL, EPI, PRK><<<blocks, threads, 0, st>>>(a);
      return;
    }
  }
  // (the FP32 update with all hops and a kappa per RHS lands in k_hop, at 104
  // registers; M_SAP with four kappas 5.28 -> 5.15 ms at 24^3x48 and 1.22 ->
  // 1.15 at 16^3x32 against the bounded update and face passes it replaces)
  if constexpr (MinCtas<T, SEL>::value == 4)
    k_hop_r64<T, SEL, EPI, PRK><<<blocks, threads, 0, st>>>(a);
  else
    k_hop<T, SEL, EPI, PRK><<<blocks, threads, 0, st>>>(a);
}

template <typename T, int SEL, int EPI>
static void launch(const HopArgs<T>& a, cudaStream_t st) {
  if (a.nsites <= 0) return;
  count_launch();
  if (a.Cr && a.kap)
    launch_v<T, SEL, EPI, true>(a, st);
  else
    launch_v<T, SEL, EPI, false>(a, st);
}

// merge one hop launch of each group member: 128-thread blocks (a thread's
// work does not depend on the CTA size), each member's sites in its own
// blocks; the FP16 block kernels keep their 64-register bound (the FP32
// block kernels and the full-lattice operators would spill under the bounds
// of their one-lattice forms, where the arguments sit in kernel parameters).
// The FP16 update with all hops is unbounded, at 101 registers; beside the
// update at 64 and the face pass at 80 that it replaces, the group's time on
// the GPU fell: 38.3 -> 35.4 ms for 48 lattices of 8^4 and 12^3x24, 28.0 -> 26.7
// for eight of 16^3x32, 69.4 -> 68.1 for four of 24^3x48.
template <typename T, int SEL, int EPI>
static void merge_hop(const GroupRec* const* recs, int n, GroupBatch& b) {
  constexpr int threads = 128;
  std::vector<HopArgs<T>> args(n);
  std::vector<int> starts(n + 1);
  int blocks = 0;
  for (int l = 0; l < n; l++) {
    args[l] = group_arg<HopArgs<T>>(recs[l]);
    starts[l] = blocks;
    blocks += args[l].nsites > 0 ? (args[l].nsites + threads - 1) / threads : 0;
  }
  starts[n] = blocks;
  if (blocks == 0) return;
  const size_t oa = b.put(args.data(), sizeof(HopArgs<T>) * n), os = b.put_starts(starts);
  b.launches.push_back([=](const unsigned char* dev, cudaStream_t st) {
    count_launch();
    const auto* A = reinterpret_cast<const HopArgs<T>*>(dev + oa);
    const auto* S = reinterpret_cast<const int*>(dev + os);
    if constexpr (std::is_same<T, H16>::value && MinCtas<T, SEL>::value == 4)
      k_hop_multi_r64<T, SEL, EPI><<<blocks, threads, 0, st>>>(A, S, n);
    else
      k_hop_multi<T, SEL, EPI><<<blocks, threads, 0, st>>>(A, S, n);
  });
}

template <typename T>
void launch_hop(int sel, int epi, const HopArgs<T>& a, cudaStream_t st) {
  if (g_group_rec) {  // a group solve: one right-hand side, one kappa per lattice
    if (a.G.nr != 1 || (a.Cr && a.kap)) group_unrecorded_launch();
#define QWSG_CASE(S, E)                           \
  if (sel == S && epi == E) {                     \
    group_record(&merge_hop<T, S, E>, a);         \
    return;                                       \
  }
    QWSG_CASE(HOP_ALL, EPI_D)
    QWSG_CASE(HOP_INNER, EPI_D)
    QWSG_CASE(HOP_OUTER, EPI_ADD)
    QWSG_CASE(HOP_INNER, EPI_JINV)
    QWSG_CASE(HOP_INNER, EPI_SAPE)
    if constexpr (!std::is_same<T, double>::value) {
      QWSG_CASE(HOP_ALL, EPI_SAPE)
    }
#undef QWSG_CASE
  }
#define QWSG_CASE(S, E)              \
  if (sel == S && epi == E) {        \
    launch<T, S, E>(a, st);          \
    return;                          \
  }
  QWSG_CASE(HOP_ALL, EPI_D)
  QWSG_CASE(HOP_INNER, EPI_D)
  QWSG_CASE(HOP_OUTER, EPI_ADD)
  QWSG_CASE(HOP_INNER, EPI_JINV)
  QWSG_CASE(HOP_INNER, EPI_SAPE)
  if constexpr (!std::is_same<T, double>::value) {
    QWSG_CASE(HOP_ALL, EPI_SAPE)
  }
#undef QWSG_CASE
}

template void launch_hop<float>(int, int, const HopArgs<float>&, cudaStream_t);
template void launch_hop<double>(int, int, const HopArgs<double>&, cudaStream_t);
template void launch_hop<H16>(int, int, const HopArgs<H16>&, cudaStream_t);

}  // namespace qwsg
