// On-device clover term: the clover-leaf field strength of the resident FP64
// gauge field and the packed inverse chiral blocks the DD kernels read.
//
// No counterpart in the reference: QWS loads a clover term that BQCD built
// and inverted (qws_bqcd.cc:284-382).  The conventions are those of the host
// generator (fields.cu), so the two agree to rounding:
//   F_{mu nu} = (Q - Q^dag) / (8i), traceless, Q the four-leaf sum;
//   T = 1 - csw*kappa * sum_{mu<nu} sigma_{mu nu} F_{mu nu};
//   stored: the two 6x6 chiral blocks M_i = (P T P^T / 2)_i^-1 / 2 in the
//   reference's packing (clover_def.h:88-284, diagonal then pairs j<k).
// In the chiral basis sigma_{mu nu} is block diagonal, so each block is built
// directly: (P T P^T / 2)_i = 1 - csw*kappa * sum S_{mu nu,i} (x) F_{mu nu},
// S the 2x2 spin tables of clover_chiral_tables().
//
// Two kernels.  k_field_strength: one thread per (site, plane) writes the
// Hermitian F (9 reals) into the FP64 planes the clover term will fill.
// k_clover_blocks: one thread per (site, chirality, right-hand side) reads F,
// forms its 6x6 Hermitian block and inverts it in registers (L D L^+).  F does
// not depend on kappa, so a handle with a kappa per RHS computes it once.
#include <algorithm>
#include <cmath>

#include <type_traits>

#include "ctx.h"

namespace qwsg {

double clover_chiral_tables(double S[6][2][2][2][2]);

namespace {

struct Cx {
  double r, i;
};
__device__ __forceinline__ Cx cmul(Cx a, Cx b) { return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }
__device__ __forceinline__ Cx cadd(Cx a, Cx b) { return {a.r + b.r, a.i + b.i}; }
__device__ __forceinline__ Cx csub(Cx a, Cx b) { return {a.r - b.r, a.i - b.i}; }
__device__ __forceinline__ Cx conj(Cx a) { return {a.r, -a.i}; }
__device__ __forceinline__ double cabs2(Cx a) { return a.r * a.r + a.i * a.i; }

struct Mat {
  Cx a[3][3];
};

// one row of a link: U_mu(g)[i][0..2]
__device__ __forceinline__ void load_row(const double* __restrict__ U, int pad, int mu, int g,
                                         int i, Cx r[3]) {
  const double2* q = reinterpret_cast<const double2*>(U) + (size_t)(9 * mu + 3 * i) * pad + g;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double2 t = __ldg(q + (size_t)k * pad);
    r[k] = {t.x, t.y};
  }
}
__device__ __forceinline__ void fma_to(Cx& s, Cx a, Cx b) { s = cadd(s, cmul(a, b)); }

// Products with a link read from memory row by row (three complex at a time
// instead of a whole matrix in registers).
// C = U
__device__ __forceinline__ void load_mat(const double* U, int pad, int mu, int g, Mat& C) {
#pragma unroll
  for (int i = 0; i < 3; i++) load_row(U, pad, mu, g, i, C.a[i]);
}
// C = U^dag
__device__ __forceinline__ void load_dag(const double* U, int pad, int mu, int g, Mat& C) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    Cx r[3];
    load_row(U, pad, mu, g, i, r);
#pragma unroll
    for (int k = 0; k < 3; k++) C.a[k][i] = conj(r[k]);
  }
}
// C = A U^dag
__device__ __forceinline__ void mul_dag(const Mat& A, const double* U, int pad, int mu, int g,
                                        Mat& C) {
#pragma unroll
  for (int j = 0; j < 3; j++) {
    Cx r[3];
    load_row(U, pad, mu, g, j, r);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      Cx s = cmul(A.a[i][0], conj(r[0]));
      fma_to(s, A.a[i][1], conj(r[1]));
      fma_to(s, A.a[i][2], conj(r[2]));
      C.a[i][j] = s;
    }
  }
}
// C += f A U   (f = 1 or -1)
__device__ __forceinline__ void mul_add(const Mat& A, const double* U, int pad, int mu, int g,
                                        double f, Mat& C) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    Cx r[3];
    load_row(U, pad, mu, g, k, r);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const Cx x = {f * A.a[i][k].r, f * A.a[i][k].i};
#pragma unroll
      for (int j = 0; j < 3; j++) fma_to(C.a[i][j], x, r[j]);
    }
  }
}
// C += U A
__device__ __forceinline__ void left_add(const double* U, int pad, int mu, int g, const Mat& A,
                                         Mat& C) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    Cx r[3];
    load_row(U, pad, mu, g, i, r);
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
      for (int k = 0; k < 3; k++) fma_to(C.a[i][j], r[k], A.a[k][j]);
  }
}
__device__ __forceinline__ void clear(Mat& C) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) C.a[i][j] = {0, 0};
}

__device__ __forceinline__ int wrap(int v, int L) { return v < 0 ? v + L : (v >= L ? v - L : v); }
// the site x + d e_a + e e_b
__device__ __forceinline__ int shifted(const Geom& G, const int x[4], int a, int d, int b, int e) {
  int y[4];
#pragma unroll
  for (int k = 0; k < 4; k++)  // (a, b are not compile-time: no indexed writes)
    y[k] = wrap(x[k] + (k == a ? d : 0) + (k == b ? e : 0), G.L[k]);
  return dd_index(G, y);
}

// W_ab(x) = the upper minus the lower staple of the link U_a(x) in the plane
// (a, b):  U_b(x+a) U_a(x+b)^dag U_b(x)^dag - U_b(x+a-b)^dag U_a(x-b)^dag U_b(x-b)
__device__ __forceinline__ void staples(const Geom& G, const double* U, const int x[4], int g,
                                        int a, int b, Mat& W) {
  Mat P, Q;
  const int xmb = shifted(G, x, b, -1, a, 0);
  load_dag(U, G.pad, b, shifted(G, x, a, 1, b, -1), P);
  mul_dag(P, U, G.pad, a, xmb, Q);
  clear(W);
  mul_add(Q, U, G.pad, b, xmb, -1.0, W);
  load_mat(U, G.pad, b, shifted(G, x, a, 1, b, 0), P);
  mul_dag(P, U, G.pad, a, shifted(G, x, b, 1, a, 0), Q);
#pragma unroll
  for (int j = 0; j < 3; j++) {  // W += Q U_b(x)^dag
    Cx r[3];
    load_row(U, G.pad, b, g, j, r);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int k = 0; k < 3; k++) fma_to(W.a[i][j], Q.a[i][k], conj(r[k]));
  }
}

// in-place inverse of a 6x6 complex matrix (Gauss-Jordan, partial pivoting on
// the modulus); returns false for a singular block
__device__ bool invert6(Cx a[6][6]) {
  Cx inv[6][6];
  for (int i = 0; i < 6; i++)
    for (int j = 0; j < 6; j++) inv[i][j] = {i == j ? 1.0 : 0.0, 0.0};
  for (int c = 0; c < 6; c++) {
    int p = c;
    for (int r = c + 1; r < 6; r++)
      if (cabs2(a[r][c]) > cabs2(a[p][c])) p = r;
    if (cabs2(a[p][c]) == 0) return false;
    if (p != c)
      for (int k = 0; k < 6; k++) {
        Cx t = a[p][k];
        a[p][k] = a[c][k];
        a[c][k] = t;
        t = inv[p][k];
        inv[p][k] = inv[c][k];
        inv[c][k] = t;
      }
    const double n = cabs2(a[c][c]);
    const Cx d = {a[c][c].r / n, -a[c][c].i / n};
    for (int k = 0; k < 6; k++) {
      a[c][k] = cmul(a[c][k], d);
      inv[c][k] = cmul(inv[c][k], d);
    }
    for (int r = 0; r < 6; r++) {
      if (r == c) continue;
      const Cx f = a[r][c];
      if (f.r == 0 && f.i == 0) continue;
      for (int k = 0; k < 6; k++) {
        a[r][k] = csub(a[r][k], cmul(f, a[c][k]));
        inv[r][k] = csub(inv[r][k], cmul(f, inv[c][k]));
      }
    }
  }
  for (int i = 0; i < 6; i++)
    for (int j = 0; j < 6; j++) a[i][j] = inv[i][j];
  return true;
}

// F_{mu nu} = (Q - Q^dag) / (8i), traceless: the Hermitian matrix as 9 reals
// (diagonal; 01, 02, 12 complex) in five 16-byte planes, plane set p at planes
// 5p .. 5p+4 of `F` (entry g << oshift, stride ostride).
//
// Of the four leaves only Q - Q^dag enters, so a leaf may be replaced by minus
// its adjoint; with W the staple difference above
//   Q - Q^dag = [U_a(x) W(x) + W(x-a) U_a(x-a)] - h.c.,
// and W(x) serves x and x + a: a thread walks `seg` sites along a, 6 + 4/seg
// matrix products a site and plane instead of the leaves' 12.  Bound by FP64
// issue at the 12 warps its registers leave an SM (52 % of the FP64 pipe at
// 24^3x48: 0.47 ms, where one thread per site and plane with whole matrices
// in registers took 0.76 ms).  a is the one of mu, nu that is not the fastest
// direction in memory, so that a warp reads runs of neighbouring sites.
__global__ void __launch_bounds__(128, 3) k_field_strength(Geom G, const double* __restrict__ U,
                                                           double* F, int oshift, int ostride,
                                                           int seg) {
  // planes of the same sites are neighbours in the grid (shared links)
  const int p = blockIdx.x % 6;
  const int mu = p < 3 ? 0 : (p < 5 ? 1 : 2), nu = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
  const bool swap = mu == G.rot;
  const int a = swap ? nu : mu, b = swap ? mu : nu;
  // thread -> first site of its walk: the fastest direction first, then the
  // others, direction a in steps of seg
  int t = (blockIdx.x / 6) * 128 + threadIdx.x;
  int x[4];
  {
    const int n = G.L[G.rot];
    const int q = t / n;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k == G.rot) x[k] = t - q * n;
    t = q;
  }
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (k == G.rot) continue;
    const int n = k == a ? (G.L[k] + seg - 1) / seg : G.L[k];
    const int q = t / n;
    x[k] = (t - q * n) * (k == a ? seg : 1);
    t = q;
  }
  if (t > 0) return;
  const double sign = swap ? -1.0 : 1.0;  // F_ba = -F_ab
  int left = 0;  // sites of this walk
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (k == a) left = min(seg, G.L[k] - x[k]);
  Mat Q, W;
  int g;
  {
    int y[4];
#pragma unroll
    for (int k = 0; k < 4; k++) y[k] = k == a ? wrap(x[k] - 1, G.L[k]) : x[k];
    g = dd_index(G, y);
    staples(G, U, y, g, a, b, W);
  }
  for (; left > 0; left--) {
    clear(Q);
    mul_add(W, U, G.pad, a, g, 1.0, Q);  // W(x-a) U_a(x-a)
    g = dd_index(G, x);
    staples(G, U, x, g, a, b, W);
    left_add(U, G.pad, a, g, W, Q);  // U_a(x) W(x)
    double f[10];
    // (Q - Q^dag)/(8i): entry ij is (Im(d)/8, -Re(d)/8) of d = Q_ij - conj(Q_ji)
#pragma unroll
    for (int i = 0; i < 3; i++) f[i] = 2.0 * Q.a[i][i].i / 8.0;
    const double tr = (f[0] + f[1] + f[2]) / 3.0;
#pragma unroll
    for (int i = 0; i < 3; i++) f[i] -= tr;
    int n = 3;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = i + 1; j < 3; j++, n += 2) {
        const Cx d = csub(Q.a[i][j], conj(Q.a[j][i]));
        f[n] = d.i / 8.0;
        f[n + 1] = -d.r / 8.0;
      }
    f[9] = 0;
    double2* q = reinterpret_cast<double2*>(F) + (size_t)5 * p * ostride + ((size_t)g << oshift);
#pragma unroll
    for (int k = 0; k < 5; k++)
      q[(size_t)k * ostride] = make_double2(sign * f[2 * k], sign * f[2 * k + 1]);
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k == a) x[k]++;
  }
}

// spin tables of one launch: per plane and chirality the 2x2 Hermitian S
struct SpinTab {
  double s00[2][6], s11[2][6], s01r[2][6], s01i[2][6];
};
struct CsKappa {
  double v[Ctx::kMaxRhs];  // csw * kappa of each right-hand side
};

// upper triangle of one chirality block of T = 1 - ck sum S (x) F: diagonal d,
// pairs j < k in order
struct Herm6 {
  double d[6];
  Cx o[15];
};
__host__ __device__ constexpr int pair6(int j, int k) {  // index of (j, k), j < k
  return j * 5 - j * (j - 1) / 2 + (k - j - 1);
}

// h = L D L^+ without pivoting, all in registers: di = D^-1 and the unit
// lower X = L^-1 as l[pair6(j, i)] = X_ij.  Stable while every pivot stays
// positive and not small beside the unit diagonal of T; returns false
// otherwise.
__device__ __forceinline__ bool factor_ldl(const Herm6& h, double di[6], Cx l[15]) {
  double d[6];
#pragma unroll
  for (int j = 0; j < 6; j++) d[j] = h.d[j];
#pragma unroll
  for (int j = 0; j < 15; j++) l[j] = conj(h.o[j]);
  bool ok = true;
  // (constant trip counts throughout: a loop left rolled would put the
  // arrays into local memory)
#pragma unroll
  for (int k = 0; k < 6; k++) {
    ok = ok && d[k] > 1e-3;
    di[k] = 1.0 / d[k];
#pragma unroll
    for (int j = 0; j < 6; j++) {
      if (j <= k) continue;
      const Cx ljk = {l[pair6(k, j)].r * di[k], l[pair6(k, j)].i * di[k]};
      d[j] -= cabs2(l[pair6(k, j)]) * di[k];
#pragma unroll
      for (int i = 0; i < 6; i++)
        if (i > j) l[pair6(j, i)] = csub(l[pair6(j, i)], cmul(l[pair6(k, i)], conj(ljk)));
    }
#pragma unroll
    for (int j = 0; j < 6; j++)
      if (j > k) l[pair6(k, j)] = {l[pair6(k, j)].r * di[k], l[pair6(k, j)].i * di[k]};
  }
  if (!ok) return false;
  // X = L^-1 (unit lower), in place of L: X_ij = -(L_ij + sum_{j<k<i} X_ik L_kj)
#pragma unroll
  for (int jj = 0; jj < 5; jj++)
#pragma unroll
    for (int ii = 0; ii < 5; ii++) {
      const int j = 4 - jj, i = 5 - ii;
      if (i <= j) continue;
      Cx s = l[pair6(j, i)];
#pragma unroll
      for (int k = 0; k < 6; k++)
        if (k > j && k < i) s = cadd(s, cmul(l[pair6(k, i)], l[pair6(j, k)]));
      l[pair6(j, i)] = {-s.r, -s.i};
    }
  return true;
}
// row j of the inverse X^+ D^-1 X: its diagonal entry, and entry (j, k) for k > j
__device__ __forceinline__ double inverse_diag(const double di[6], const Cx x[15], int j) {
  double s = di[j];
#pragma unroll
  for (int m = 0; m < 6; m++)
    if (m > j) s += di[m] * cabs2(x[pair6(j, m)]);
  return s;
}
__device__ __forceinline__ Cx inverse_pair(const double di[6], const Cx x[15], int j, int k) {
  const Cx xkj = x[pair6(j, k)];
  Cx o = {xkj.r * di[k], -xkj.i * di[k]};
#pragma unroll
  for (int m = 0; m < 6; m++) {
    if (m <= k) continue;
    const Cx v = {x[pair6(k, m)].r * di[m], x[pair6(k, m)].i * di[m]};
    o = cadd(o, cmul(conj(x[pair6(j, m)]), v));
  }
  return o;
}

// writes one chirality block: FP64 and FP32 planes, and FP16 planes when Ch,
// at entry (g << lgnr) + r with plane stride ostride.  Thread = (RHS, site,
// chirality), RHS fastest, the two chiralities of a CTA's sites in its two
// halves; F is read from the FP64 planes (entry g << lgnr) before any thread
// of the CTA writes there.  Bound by memory: 480 bytes read and 864 written a
// site take 0.155 ms at 24^3x48 (0.88 of the measured copy rate), at three
// blocks an SM (two: 0.199; four spill: 0.183); field strength and inverse in
// one thread per site, with indexed arrays in local memory, took 4.3 ms.
__global__ void __launch_bounds__(128, 3) k_clover_blocks(Geom G, double* Cd, float* Cs, __half* Ch,
                                                       const __grid_constant__ SpinTab S,
                                                       const __grid_constant__ CsKappa ck,
                                                       unsigned* left, int lgnr, int ostride) {
  const int per = 64 >> lgnr;  // sites of this CTA
  const int r = threadIdx.x & ((1 << lgnr) - 1);
  const int b = threadIdx.x >> 6;
  const int g = blockIdx.x * per + ((threadIdx.x & 63) >> lgnr);
  const bool live = g < G.V;
  Herm6 h;
#pragma unroll
  for (int j = 0; j < 6; j++) h.d[j] = 1;
#pragma unroll
  for (int j = 0; j < 15; j++) h.o[j] = {0, 0};
  if (live) {
    const double c = ck.v[r];
    const double2* q = reinterpret_cast<const double2*>(Cd) + ((size_t)g << lgnr);
#pragma unroll
    for (int p = 0; p < 6; p++) {
      double f[10];
#pragma unroll
      for (int k = 0; k < 5; k++) {
        const double2 t = q[(size_t)(5 * p + k) * ostride];
        f[2 * k] = t.x;
        f[2 * k + 1] = t.y;
      }
      const double s00 = S.s00[b][p] * c, s11 = S.s11[b][p] * c;
      const Cx s01 = {S.s01r[b][p] * c, S.s01i[b][p] * c};
      const Cx o[3] = {{f[3], f[4]}, {f[5], f[6]}, {f[7], f[8]}};  // 01, 02, 12
      // (of s00, s11 and s01 one kind is zero for every plane; a branch on it
      // would keep the next plane's loads back)
#pragma unroll
      for (int i = 0; i < 3; i++) {
        h.d[i] -= s00 * f[i];
        h.d[3 + i] -= s11 * f[i];
      }
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
          if (j <= i) continue;
          const Cx m = o[i + j - 1];
          Cx& u = h.o[pair6(i, j)];
          u = csub(u, {s00 * m.r, s00 * m.i});
          Cx& w = h.o[pair6(3 + i, 3 + j)];
          w = csub(w, {s11 * m.r, s11 * m.i});
        }
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
          const Cx m = i == j ? Cx{f[i], 0} : (i < j ? o[i + j - 1] : conj(o[i + j - 1]));
          Cx& u = h.o[pair6(i, 3 + j)];
          u = csub(u, cmul(s01, m));
        }
    }
  }
  __syncthreads();  // every F of this CTA's sites has been read
  if (!live) return;
  // entries leave as they are made (the FP32 copies wait in registers)
  const size_t e = ((size_t)g << lgnr) + r;
  double2* qd = reinterpret_cast<double2*>(Cd) + (size_t)18 * b * ostride + e;
  float fs[36];
  auto put = [&](int j, double x, double y) {  // reals 2j, 2j+1 of the packed block
    qd[(size_t)j * ostride] = make_double2(x, y);
    fs[2 * j] = (float)x;
    fs[2 * j + 1] = (float)y;
  };
  double di[6];
  Cx x[15];
  if (factor_ldl(h, di, x)) {
#pragma unroll
    for (int j = 0; j < 3; j++)
      put(j, 0.5 * inverse_diag(di, x, 2 * j), 0.5 * inverse_diag(di, x, 2 * j + 1));
#pragma unroll
    for (int j = 0; j < 6; j++)
#pragma unroll
      for (int k = 0; k < 6; k++) {
        if (k <= j) continue;
        const Cx o = inverse_pair(di, x, j, k);
        put(3 + pair6(j, k), 0.5 * o.r, 0.5 * o.i);
      }
  } else {  // the block itself, marked by its first FP32 real: k_clover_pivoted
    atomicAdd(left, 1u);
#pragma unroll
    for (int j = 0; j < 3; j++) put(j, h.d[2 * j], h.d[2 * j + 1]);
#pragma unroll
    for (int n = 0; n < 15; n++) put(3 + n, h.o[n].r, h.o[n].i);
    fs[0] = __int_as_float(0x7fc00000);
  }
  float4* qs = reinterpret_cast<float4*>(Cs) + (size_t)9 * b * ostride + e;
#pragma unroll
  for (int j = 0; j < 9; j++)
    qs[(size_t)j * ostride] = make_float4(fs[4 * j], fs[4 * j + 1], fs[4 * j + 2], fs[4 * j + 3]);
  if (Ch) {  // (a constant block index keeps fs in registers)
    if (b == 0)
      IO<H16>::store_clover_block(Ch, ostride, (int)e, 0, fs);
    else
      IO<H16>::store_clover_block(Ch, ostride, (int)e, 1, fs);
  }
}

// the blocks k_clover_blocks left (rare: none on fields smooth enough for a
// positive clover term): pivoted elimination; a kernel of its own, because its
// indexed arrays live in local memory.  A singular block becomes zero and
// counts in `bad`.
__global__ void k_clover_pivoted(double* Cd, float* Cs, __half* Ch, unsigned* bad, int entries,
                                 int ostride) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= entries) return;
  for (int b = 0; b < 2; b++) {
    double2* qd = reinterpret_cast<double2*>(Cd) + (size_t)18 * b * ostride + e;
    float4* qs = reinterpret_cast<float4*>(Cs) + (size_t)9 * b * ostride + e;
    if (!isnan(qs[0].x)) continue;
    double out[36];
    for (int j = 0; j < 18; j++) {
      out[2 * j] = qd[(size_t)j * ostride].x;
      out[2 * j + 1] = qd[(size_t)j * ostride].y;
    }
    Cx a[6][6];
    int n = 0;
    for (int j = 0; j < 6; j++) {
      a[j][j] = {out[j], 0};
      for (int k = j + 1; k < 6; k++, n++) {
        a[j][k] = {out[6 + 2 * n], out[7 + 2 * n]};
        a[k][j] = conj(a[j][k]);
      }
    }
    const bool ok = invert6(a);
    if (!ok) atomicAdd(bad, 1u);
    n = 0;
    for (int j = 0; j < 6; j++) {
      out[j] = ok ? 0.5 * a[j][j].r : 0;
      for (int k = j + 1; k < 6; k++, n++) {
        out[6 + 2 * n] = ok ? 0.5 * a[j][k].r : 0;
        out[7 + 2 * n] = ok ? 0.5 * a[j][k].i : 0;
      }
    }
    float fs[36];
    for (int j = 0; j < 36; j++) fs[j] = (float)out[j];
    for (int j = 0; j < 18; j++) qd[(size_t)j * ostride] = make_double2(out[2 * j], out[2 * j + 1]);
    for (int j = 0; j < 9; j++)
      qs[(size_t)j * ostride] = make_float4(fs[4 * j], fs[4 * j + 1], fs[4 * j + 2], fs[4 * j + 3]);
    if (Ch) IO<H16>::store_clover_block(Ch, ostride, e, b, fs);
  }
}

}  // namespace

static const double (*chiral_tables())[2][2][2][2] {
  struct Tables {
    double S[6][2][2][2][2];
    double off;
    Tables() { off = clover_chiral_tables(S); }
  };
  static const Tables tab;  // built once, thread-safe
  if (tab.off > 1e-14) throw Error(3, "sigma_{mu nu} is not block diagonal in the chiral basis");
  return tab.S;
}

// the clover terms for csw * kappa = ck[r] on c's stream into (Cd, Cs, Ch) at
// entries (g << lgnr) + r, plane stride ostride
static void build_into(Ctx& c, const double* Ud, double* Cd, float* Cs, __half* Ch,
                       const CsKappa& ck, int lgnr, int ostride) {
  const auto* tab = chiral_tables();
  SpinTab S;
  for (int b = 0; b < 2; b++)
    for (int p = 0; p < 6; p++) {
      S.s00[b][p] = tab[p][b][0][0][0];
      S.s11[b][p] = tab[p][b][1][1][0];
      S.s01r[b][p] = tab[p][b][0][1][0];
      S.s01i[b][p] = tab[p][b][0][1][1];
    }
  unsigned* count = c.rb.counter + 1;  // a spare counter slot
  QWSG_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned), c.st));
  // walks of 4 sites once that still leaves every SM a few waves of blocks
  const int seg = c.G.V >= (1 << 17) ? 4 : 1;
  long walks = 0;  // the most over the directions a walk may take
  for (int mu = 0; mu < 4; mu++)
    walks = std::max(walks, (long)(c.G.V / c.G.L[mu]) * ((c.G.L[mu] + seg - 1) / seg));
  count_launch();
  k_field_strength<<<(unsigned)(6 * ((walks + 127) / 128)), 128, 0, c.st>>>(c.G, Ud, Cd, lgnr,
                                                                           ostride, seg);
  const int per = 64 >> lgnr;
  count_launch();
  k_clover_blocks<<<(c.G.V + per - 1) / per, 128, 0, c.st>>>(c.G, Cd, Cs, Ch, S, ck, count, lgnr,
                                                             ostride);
  c.check_launch("build_clover");
  unsigned n = 0;
  auto read = [&] {
    QWSG_CUDA(cudaMemcpyAsync(&n, count, sizeof(unsigned), cudaMemcpyDeviceToHost, c.st));
    QWSG_CUDA(cudaStreamSynchronize(c.st));
  };
  read();
  if (n == 0) return;
  QWSG_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned), c.st));
  const int entries = c.G.V << lgnr;
  count_launch();
  k_clover_pivoted<<<(entries + 127) / 128, 128, 0, c.st>>>(Cd, Cs, Ch, count, entries, ostride);
  c.check_launch("build_clover (pivoted)");
  read();
  if (n) throw Error(2, "clover term singular on " + std::to_string(n) + " blocks");
}

// clover term of the resident FP64 gauge field for this context's kappa:
// writes the FP64 and FP32 clover planes (the FP16 copies follow on demand)
void build_clover(Ctx& c, double csw) {
  if (!c.Ud) throw Error(4, "gauge field not loaded");
  if (c.parent) throw Error(1, "build the clover term on the parent lattice");
  c.ensure_fields_d();
  const bool links12 = c.Us && c.links12_valid;  // the links stay as they are
  c.ensure_fields_s();
  c.links12_valid = links12;
  CsKappa ck{};
  ck.v[0] = csw * c.kappa;
  build_into(c, c.Ud, c.Cd, c.Cs, nullptr, ck, 0, c.G.pad);
}

// per-RHS kappa on a multi-RHS handle: the clover term of the parent's gauge
// field for kappas[r], into the handle's per-RHS planes (FP64, FP32 and the
// FP16 copy), and the kappa tables the Dirac kernels read
void set_rhs_kappas(Ctx& c, const double* kappas, double csw) {
  if (!c.parent) throw Error(1, "per-RHS kappa needs a multi-RHS handle");
  c.sync_from_parent(false);
  if (!c.Ud) throw Error(4, "gauge field not loaded");
  const size_t n = (size_t)72 * spad(c.G);
  if (c.rhs_kappas.empty()) {  // graphs captured before read the parent's clover
    QWSG_CUDA(cudaStreamSynchronize(c.st));
    c.clear_graphs();
  }
  // each plane set on its own: one that failed to allocate is retried by the
  // next call, and no launch below runs before all of them exist
  auto want = [&](auto** p, size_t bytes) {
    if (*p) return;
    void* q = nullptr;
    QWSG_CUDA(cudaMalloc(&q, bytes));
    c.owned.push_back(q);
    *p = static_cast<std::remove_reference_t<decltype(**p)>*>(q);
  };
  want(&c.Cdr, sizeof(double) * n);
  want(&c.Csr, sizeof(float) * n);
  want(&c.Chr, sizeof(__half) * n);
  want(&c.kap_d, sizeof(double) * Ctx::kMaxRhs);
  want(&c.kap_s, sizeof(float) * Ctx::kMaxRhs);
  CsKappa ck{};
  for (int r = 0; r < c.G.nr; r++) ck.v[r] = csw * kappas[r];
  build_into(c, c.Ud, c.Cdr, c.Csr, c.Chr, ck, c.G.lgnr, spad(c.G));
  double kd[Ctx::kMaxRhs];
  float ks[Ctx::kMaxRhs];
  for (int r = 0; r < c.G.nr; r++) {
    kd[r] = kappas[r];
    ks[r] = (float)kappas[r];
  }
  QWSG_CUDA(cudaMemcpyAsync(c.kap_d, kd, sizeof(double) * c.G.nr, cudaMemcpyHostToDevice, c.st));
  QWSG_CUDA(cudaMemcpyAsync(c.kap_s, ks, sizeof(float) * c.G.nr, cudaMemcpyHostToDevice, c.st));
  QWSG_CUDA(cudaStreamSynchronize(c.st));
  c.rhs_kappas.assign(kappas, kappas + c.G.nr);
}

}  // namespace qwsg
