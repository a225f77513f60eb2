// Even-odd (site parity) hopping kernels: the deo_* family of the reference
// (deo_in_d.cc:65-445, deo_out_d.cc:88-286, deo_dag_in.cc, deo_dag_out.cc and
// the FP32 deo_in_s.cc / deo_out_s.cc).
//
// Sites of parity pe = (x+y+z+t) % 2 receive the hops from the other parity:
//   WHICH  1 = hops inside the rank box (deo_in_*), 2 = hops across its faces
//          (deo_out_pre/pos_*), 3 = both;
//   DAG    the adjoint hopping H^dagger (projectors 1 + gamma_mu forward,
//          1 - gamma_mu backward, deo_dag_*);
//   CLOV   multiply by the parity's A^-1 (dee_*);
//   MODE   0 out = acc (__store_sc), 1 out += coef acc (__store_add_sc),
//          2 out = in0 + coef acc (one_minus_*).
//
// Two forms.  The Schur operators and solvers work on
// vectors and fields of one parity each, stored compactly in the order
// e = x/2 + Lx/2 (y + Ly (z + Lz t)).  On the full lattice's planes the two
// parities alternate along a row, so one parity's 16-byte entries use half of
// every 32-byte sector; compact, every byte fetched is used (FP64 normal
// operator at 24^3x48: 2.6 ms on full planes walked in x order, 0.67 ms
// compact).  Full-plane vectors of the API are gathered and scattered by
// eo_gather / eo_scatter, the fields once per load.  A single hop operator of
// the API reads and writes the full planes as they are (k_eo_planes).
//
// A y/z/t hop reads the other parity's site at the same compressed index x/2
// of the neighbouring row, also across a boundary, as the reference's face
// packers do (deo_out_d.cc:88-153); this is the geometric neighbour when the
// wrapped extent is even.
#include "kernels.h"
#include "lattice.cuh"

namespace qwsg {

struct EoSite {
  int xh, y, z, t;
  int odd;  // x = 2 xh + odd
};
template <typename T>
__device__ __forceinline__ EoSite eo_site(const EoArgs<T>& a, int e) {
  EoSite s;
  int k = fdiv(e, a.dxh);
  s.xh = e - k * (a.G.L[0] >> 1);
  int q = fdiv(k, a.dy);
  s.y = k - q * a.G.L[1];
  s.t = fdiv(q, a.dz);
  s.z = q - s.t * a.G.L[2];
  s.odd = (a.pe + s.y + s.z + s.t) & 1;
  return s;
}

// (the products are written out here and in eo_hop_planes: shared through a
// function they came out with other register spills, mtilde in FP32 at 24^3x48
// 169 -> 182 us)
template <typename T, int DAG, int MU, int DIR, typename R = typename Arith<T>::R>
__device__ __forceinline__ void eo_hop(const EoArgs<T>& a, const EoSite& s, int e, R acc[24]) {
  const int c = MU == 0 ? 2 * s.xh + s.odd : MU == 1 ? s.y : MU == 2 ? s.z : s.t;
  const int en = eo_step(a.G, e, MU, DIR, c, s.xh, s.odd);
  constexpr int PD = DAG ? -DIR : DIR;  // projector / reconstruction of this hop
  R v[24];
  if (MU == 3)
    IO<T>::load_half(a.src, a.pad, en, PD > 0, v);
  else
    IO<T>::load_spinor(a.src, a.pad, en, v);
  R h[12], r[12], u[18];
  project<R, MU, PD>(v, h);
  // forward: this parity's own link, backward: the other parity's
  IO<T>::load_link(DIR > 0 ? a.U[0] : a.U[1], a.pad, MU, DIR > 0 ? e : en, u);
  if (DIR > 0)
    link_mul<R, false>(u, h, r);
  else
    link_mul<R, true>(u, h, r);
  R f = 1;
  if (MU == 3) {
    f = 2;
    if (DIR > 0 ? s.t == a.G.L[3] - 1 : s.t == 0) f = (R)(2 * a.G.tbc);
  }
  reconstruct<R, MU, PD>(r, acc, f);
}

// Memory bound: per output site 8 links (1152 bytes in FP64, each link of the
// lattice once per launch), A^-1, the source once and the result: 2112 bytes
// in FP64, 118 us at 24^3x48, 0.91 of the measured copy rate.
template <typename T, int DAG, int CLOV, int MODE>
__device__ __forceinline__ void eo_body(const EoArgs<T>& a) {
  using R = typename Arith<T>::R;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.G.Vh) return;
  const EoSite s = eo_site(a, e);
  R acc[24];
#pragma unroll
  for (int j = 0; j < 24; j++) acc[j] = 0;
  eo_hop<T, DAG, 0, +1>(a, s, e, acc);
  eo_hop<T, DAG, 0, -1>(a, s, e, acc);
  eo_hop<T, DAG, 1, +1>(a, s, e, acc);
  eo_hop<T, DAG, 1, -1>(a, s, e, acc);
  eo_hop<T, DAG, 2, +1>(a, s, e, acc);
  eo_hop<T, DAG, 2, -1>(a, s, e, acc);
  eo_hop<T, DAG, 3, +1>(a, s, e, acc);
  eo_hop<T, DAG, 3, -1>(a, s, e, acc);
  if (CLOV) clover_apply<T>(a.C, a.pad, e, acc);
  if (MODE == 2) {
    R o[24];
    IO<T>::load_spinor(a.in0, a.pad, e, o);
#pragma unroll
    for (int j = 0; j < 24; j++) acc[j] = o[j] + acc[j] * a.coef;
  }
  IO<T>::store_spinor(a.out, a.pad, e, acc);
}
// FP64 at 128 registers (4 CTAs of 128 threads an SM), FP32 at 80 (6)
template <typename T, int DAG, int CLOV, int MODE>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 4 : 6) k_eo(const EoArgs<T> a) {
  eo_body<T, DAG, CLOV, MODE>(a);
}

// The same on the full planes.  Thread i takes the sites of parity pe among 2i
// and 2i + 1 of the planes' order: one, where the two are neighbours along an
// even row, so that a warp reads runs of the planes.  Half of every sector is
// still the other parity's, but the neighbouring warps' hops use it from L2.
// Time of one operator at 24^3x48 (hops alone / with A^-1), against threads in
// x order and against a gather, k_eo on copies that exist, and a scatter:
// FP64 164 / 215 us (373 / 562; 203 / 227), FP32 75 / 105 (230 / 286; 98 / 109);
// at 8^3x16 10 us (19 / 21; 17).
template <typename T, int WHICH, int DAG, int MU, int DIR, typename R = typename Arith<T>::R>
__device__ __forceinline__ void eo_hop_planes(const EoArgs<T>& a, const int x[4], int g, R acc[24]) {
  if (WHICH != 3) {
    const int box = a.box[MU], in_box = x[MU] % box;
    const bool inner = DIR > 0 ? in_box != box - 1 : in_box != 0;
    if (inner ? !(WHICH & 1) : !(WHICH & 2)) return;
  }
  int xn[4];
  eo_neighbour<MU, DIR>(a.G, x, a.pe, xn);
  const int gn = dd_index(a.G, xn);
  constexpr int PD = DAG ? -DIR : DIR;
  R v[24], u[18];
  if (MU == 3)
    IO<T>::load_half(a.src, a.G.pad, gn, PD > 0, v);
  else
    IO<T>::load_spinor(a.src, a.G.pad, gn, v);
  IO<T>::load_link(a.U[0], a.G.pad, MU, DIR > 0 ? g : gn, u);
  R h[12], r[12];
  project<R, MU, PD>(v, h);
  if (DIR > 0)
    link_mul<R, false>(u, h, r);
  else
    link_mul<R, true>(u, h, r);
  R f = 1;
  if (MU == 3) {
    f = 2;
    if (DIR > 0 ? x[3] == a.G.L[3] - 1 : x[3] == 0) f = (R)(2 * a.G.tbc);
  }
  reconstruct<R, MU, PD>(r, acc, f);
}
template <typename T, int WHICH, int DAG, int CLOV, int MODE>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 4 : 6) k_eo_planes(const EoArgs<T> a) {
  using R = typename Arith<T>::R;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (2 * i >= a.G.V) return;
  int x[4], x1[4];
  site_coords(a.G, 2 * i, x);
  site_coords(a.G, 2 * i + 1, x1);
  bool second;
  int g = eo_first(x, x1, a.pe, second);
  if (g < 0) return;
  g += 2 * i;
  for (;;) {
    R acc[24];
#pragma unroll
    for (int j = 0; j < 24; j++) acc[j] = 0;
    eo_hop_planes<T, WHICH, DAG, 0, +1>(a, x, g, acc);
    eo_hop_planes<T, WHICH, DAG, 0, -1>(a, x, g, acc);
    eo_hop_planes<T, WHICH, DAG, 1, +1>(a, x, g, acc);
    eo_hop_planes<T, WHICH, DAG, 1, -1>(a, x, g, acc);
    eo_hop_planes<T, WHICH, DAG, 2, +1>(a, x, g, acc);
    eo_hop_planes<T, WHICH, DAG, 2, -1>(a, x, g, acc);
    eo_hop_planes<T, WHICH, DAG, 3, +1>(a, x, g, acc);
    eo_hop_planes<T, WHICH, DAG, 3, -1>(a, x, g, acc);
    if (CLOV) clover_apply<T>(a.C, a.G.pad, g, acc);
    if (MODE != 0) {
      R o[24];
      IO<T>::load_spinor(MODE == 1 ? a.out : a.in0, a.G.pad, g, o);
#pragma unroll
      for (int j = 0; j < 24; j++) acc[j] = o[j] + acc[j] * a.coef;
    }
    IO<T>::store_spinor(a.out, a.G.pad, g, acc);
    if (!second) return;
    second = false;  // (rows of odd length)
    g++;
    site_coords(a.G, g, x);
  }
}

// out = A^-1 in on compact vectors (as an epilogue of the operator before it,
// a second A^-1 in one kernel spilled: 76 us against 25 + 11 at 16^3x32)
template <typename T>
__global__ void __launch_bounds__(128) k_eo_clv(const EoArgs<T> a) {
  using R = typename Arith<T>::R;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.G.Vh) return;
  R v[24];
  IO<T>::load_spinor(a.src, a.pad, e, v);
  clover_apply<T>(a.C, a.pad, e, v);
  IO<T>::store_spinor(a.out, a.pad, e, v);
}

// parity-pe clover multiplication on full planes (clvd_vm_/clv_s_,
// qws.cc:390-425), walked in the planes' order
template <typename T>
__global__ void __launch_bounds__(128) k_clv(Geom G, T* out, const T* __restrict__ in,
                                             const T* __restrict__ C, int pe) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= G.V) return;
  int x[4];
  site_coords(G, g, x);
  if (((x[0] + x[1] + x[2] + x[3]) & 1) != pe) return;
  T v[24];
  IO<T>::load_spinor(in, G.pad, g, v);
  clover_apply<T>(C, G.pad, g, v);
  IO<T>::store_spinor(out, G.pad, g, v);
}

// Conversions walk the order of what they write: a scattered 16-byte read costs
// a sector, a scattered write a partly written one (FP64 at 24^3x48: gather
// 38 us so, 69 in the planes' order; scatter 57, 129 in compact order).
// full planes -> compact vector of parity pe
template <typename T>
__global__ void __launch_bounds__(128) k_eo_gather(Geom G, T* __restrict__ dst, int pad,
                                                   const T* __restrict__ src, int pe) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= G.Vh) return;
  int x[4];
  eo_coords(G, e, pe, x);
  T v[24];
  IO<T>::load_spinor(src, G.pad, dd_index(G, x), v);
  IO<T>::store_spinor(dst, pad, e, v);
}
// compact vector -> parity pe of full planes; ZERO: the other parity becomes
// zero (else untouched)
template <typename T, bool ZERO>
__global__ void __launch_bounds__(128) k_eo_scatter(Geom G, T* out, const T* __restrict__ v, int pad,
                                                    int pe) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= G.V) return;
  int x[4];
  site_coords(G, g, x);
  T o[24];
  if (((x[0] + x[1] + x[2] + x[3]) & 1) != pe) {
    if (!ZERO) return;
#pragma unroll
    for (int j = 0; j < 24; j++) o[j] = 0;
  } else {
    IO<T>::load_spinor(v, pad, eo_index(G, x), o);
  }
  IO<T>::store_spinor(out, G.pad, g, o);
}

// full field planes -> the two parities' compact planes (parity p at
// p * 72 * pad reals)
template <typename T>
__global__ void __launch_bounds__(128) k_eo_links(Geom G, T* __restrict__ dst, int pad,
                                                  const T* __restrict__ U) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.z;
  if (e >= G.Vh) return;
  int x[4];
  eo_coords(G, e, p, x);
  const int g = dd_index(G, x);
  T u[18];
  IO<T>::load_link(U, G.pad, blockIdx.y, g, u);
  store_link<T>(dst + (size_t)72 * pad * p, pad, blockIdx.y, e, u);
}
template <typename T>
__global__ void __launch_bounds__(128) k_eo_clover(Geom G, T* __restrict__ dst, int pad,
                                                   const T* __restrict__ C) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.z;
  if (e >= G.Vh) return;
  int x[4];
  eo_coords(G, e, p, x);
  const int g = dd_index(G, x);
  // one chiral block's 16-byte planes
  constexpr int n = 36 * sizeof(T) / 16;
  const uint4* s = reinterpret_cast<const uint4*>(C) + (size_t)n * blockIdx.y * G.pad + g;
  uint4* d = reinterpret_cast<uint4*>(dst + (size_t)72 * pad * p) + (size_t)n * blockIdx.y * pad + e;
#pragma unroll
  for (int j = 0; j < n; j++) d[(size_t)j * pad] = __ldg(s + (size_t)j * G.pad);
}

template <typename T>
void eo_fields(const Geom& G, T* Ue, T* Ce, int pad, const T* U, const T* C, cudaStream_t st) {
  const int nb = (G.Vh + 127) / 128;
  count_launch();
  k_eo_links<T><<<dim3(nb, 4, 2), 128, 0, st>>>(G, Ue, pad, U);
  count_launch();
  k_eo_clover<T><<<dim3(nb, 2, 2), 128, 0, st>>>(G, Ce, pad, C);
}
template <typename T>
void eo_gather(const Geom& G, T* dst, int pad, const T* src, int pe, cudaStream_t st) {
  count_launch();
  k_eo_gather<T><<<(G.Vh + 127) / 128, 128, 0, st>>>(G, dst, pad, src, pe);
}
template <typename T>
void eo_scatter(const Geom& G, T* out, const T* v, int pad, int pe, bool zero_other,
                cudaStream_t st) {
  const int nb = (G.V + 127) / 128;
  count_launch();
  if (zero_other)
    k_eo_scatter<T, true><<<nb, 128, 0, st>>>(G, out, v, pad, pe);
  else
    k_eo_scatter<T, false><<<nb, 128, 0, st>>>(G, out, v, pad, pe);
}
template <typename T>
void launch_clv(const Geom& G, T* out, const T* in, const T* C, int pe, cudaStream_t st) {
  count_launch();
  k_clv<T><<<(G.V + 127) / 128, 128, 0, st>>>(G, out, in, C, pe);
}
template <typename T>
void launch_eo_clv(const EoArgs<T>& a, cudaStream_t st) {
  count_launch();
  k_eo_clv<T><<<(a.G.Vh + 127) / 128, 128, 0, st>>>(a);
}

template <typename T>
void launch_eo(int dag, int clov, int mode, const EoArgs<T>& a, cudaStream_t st) {
#define QWSG_EO(D, C, M)                                     \
  if (dag == D && clov == C && mode == M) {                  \
    count_launch();                                          \
    k_eo<T, D, C, M><<<(a.G.Vh + 127) / 128, 128, 0, st>>>(a); \
    return;                                                  \
  }
  QWSG_EO(0, 1, 0) QWSG_EO(1, 1, 0) QWSG_EO(0, 1, 2) QWSG_EO(1, 0, 2)
#undef QWSG_EO
  throw_unsupported_eo();
}

template <typename T>
void launch_eo_planes(int which, int dag, int clov, int mode, const EoArgs<T>& a, cudaStream_t st) {
  // every combination the reference uses (12 FP64, 5 FP32 entry points); as
  // many pairs of sites as sites of a parity
#define QWSG_EO(W, D, C, M)                                               \
  if (which == W && dag == D && clov == C && mode == M) {                 \
    count_launch();                                                       \
    k_eo_planes<T, W, D, C, M><<<(a.G.Vh + 127) / 128, 128, 0, st>>>(a);  \
    return;                                                               \
  }
  QWSG_EO(1, 0, 0, 0) QWSG_EO(1, 0, 1, 0) QWSG_EO(1, 1, 0, 0) QWSG_EO(1, 1, 1, 0)
  QWSG_EO(1, 0, 1, 2) QWSG_EO(1, 1, 0, 2)
  QWSG_EO(2, 0, 0, 1) QWSG_EO(2, 1, 0, 1) QWSG_EO(2, 0, 1, 1) QWSG_EO(2, 1, 1, 1)
  QWSG_EO(3, 0, 0, 0) QWSG_EO(3, 0, 1, 0) QWSG_EO(3, 1, 0, 0) QWSG_EO(3, 1, 1, 0)
  QWSG_EO(3, 0, 1, 2) QWSG_EO(3, 1, 0, 2) QWSG_EO(3, 0, 0, 1) QWSG_EO(3, 0, 1, 1)
#undef QWSG_EO
  throw_unsupported_eo();
}

#define QWSG_INST(T)                                                                          \
  template void launch_eo<T>(int, int, int, const EoArgs<T>&, cudaStream_t);                  \
  template void launch_eo_planes<T>(int, int, int, int, const EoArgs<T>&, cudaStream_t);      \
  template void launch_eo_clv<T>(const EoArgs<T>&, cudaStream_t);                             \
  template void launch_clv<T>(const Geom&, T*, const T*, const T*, int, cudaStream_t);        \
  template void eo_fields<T>(const Geom&, T*, T*, int, const T*, const T*, cudaStream_t);     \
  template void eo_gather<T>(const Geom&, T*, int, const T*, int, cudaStream_t);              \
  template void eo_scatter<T>(const Geom&, T*, const T*, int, int, bool, cudaStream_t);
QWSG_INST(float)
QWSG_INST(double)
#undef QWSG_INST

}  // namespace qwsg
