// real.cu - determinants over real orbitals (real_det.cuh) between the pair
// passes and the evaluation's end: orbitals, inverse and F matrices of every
// (walker, spin), then the sums over its Jacobian blocks.
//
// F_a = D^-1 d_a D with D(o, j) the orbitals sqrt(2) cos(g.q_j),
// sqrt(2) sin(g.q_j) of the pairs +-g and the constant (paho_orbitals,
// reptation.f:10268; zgefa/zgedi :9227, :9338; slater_excitations
// :10189-10200). Orbital o < n - 1 is the cosine (even) or sine (odd) of
// pair o / 2, whose wave vector is gvec row o | 1; orbital n - 1 is the
// constant 1. The derivative of a cosine is -g times its sine, of a sine g
// times its cosine, so
//   F_a(l, j) = sum_o Dinv(l, o) s_o g_a D(o ^ 1, j), s_o = -1 for a cosine.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "real_det.cuh"

namespace q2d {

namespace {

// The pivot key of |x|: the top word of the double with its low byte
// replaced by 255 - r, so ties within 2^-12 go to the lowest row; every
// unused row's key is nonzero, a zero or NaN column included.
__device__ __forceinline__ unsigned pivot_key(double x, int r, bool on) {
  return on ? ((unsigned)__double2hiint(fabs(x)) & ~0xFFu) | (unsigned)(255 - r) : 0u;
}

constexpr double kSqrt2 = 1.4142135623730951;

__host__ __device__ inline int odd4(int c) {  // smallest odd multiple of 4 that holds c
  return ((c + 3) / 4 | 1) * 4;
}

// (s_o g_x, s_o g_y) of orbital o of n.
__device__ __forceinline__ double2 orbital_g(const double *gvec, int o, int n) {
  if (o >= n - 1) return make_double2(0.0, 0.0);
  const double s = o & 1 ? 1.0 : -1.0;
  return make_double2(s * __ldg(gvec + 2 * (o | 1)), s * __ldg(gvec + 2 * (o | 1) + 1));
}

// Orbital rows of a spin (row o at at(o, j)) by threads t, t + nthr, ...: one
// sincos for the two rows of a pair.
template <class At>
__device__ __forceinline__ void orbital_rows(const RealArgs &a, const double *q, int n, int t,
                                             int nthr, At at) {
  for (int e = t; e < (n - 1) / 2 * n; e += nthr) {
    const int p = e / n, j = e - p * n;
    const double2 x = *reinterpret_cast<const double2 *>(q + 2 * j);
    double sv, cv;
    sincos(x.x * __ldg(a.gvec + 4 * p + 2) + x.y * __ldg(a.gvec + 4 * p + 3), &sv, &cv);
    at(2 * p, j) = kSqrt2 * cv;
    at(2 * p + 1, j) = kSqrt2 * sv;
  }
  // (NaN where the coordinates are not finite, as exp(i 0.q) is)
  for (int j = t; j < n; j += nthr) at(n - 1, j) = fma(0.0, q[2 * j], fma(0.0, q[2 * j + 1], 1.0));
}

// F_x and F_y of kR row tiles (from l0) and kT column tiles (from j0) of 8 x 8
// entries on the FP64 tensor cores (mma.m8n8k4): the A fragment is
// Dinv(l, o) s_o g_a, the B fragment D(o ^ 1, j). wt(o, l) and b(o, j) read the
// transposed inverse and the orbitals, sg[o] the scaled wave vectors (zeros
// from orbital n - 1 on). Entries outside n x n are computed from whatever
// finite values stand there and not stored.
template <int kR, int kT, class Wt, class Bm>
__device__ __forceinline__ void f_products(double (&acc)[kR][kT][2][2], int n, int l0, int j0,
                                           const double2 *sg, Wt wt, Bm b) {
  const int lane = threadIdx.x & 31, lg = lane >> 2, lt = lane & 3;
#pragma unroll 2
  for (int ob = 0; ob < n; ob += 4) {
    const int o = ob + lt;
    const double2 g = sg[o];
    double ax[kR], ay[kR];
#pragma unroll
    for (int r = 0; r < kR; r++) {
      const double w = wt(o, l0 + 8 * r + lg);
      ax[r] = w * g.x;
      ay[r] = w * g.y;
    }
#pragma unroll
    for (int t = 0; t < kT; t++) {
      const double v = b(o ^ 1, j0 + 8 * t + lg);
#pragma unroll
      for (int r = 0; r < kR; r++) {
        dmma_m8n8k4(acc[r][t][0], ax[r], v);
        dmma_m8n8k4(acc[r][t][1], ay[r], v);
      }
    }
  }
}
template <int kR, int kT>
__device__ __forceinline__ void f_store(const double (&acc)[kR][kT][2][2], double *F, int n,
                                        int l0, int j0) {
  const int lane = threadIdx.x & 31, lg = lane >> 2, lt = lane & 3;
#pragma unroll
  for (int r = 0; r < kR; r++)
#pragma unroll
    for (int t = 0; t < kT; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int l = l0 + 8 * r + lg, j = j0 + 8 * t + 2 * lt + e;
        if (l < n && j < n) {
          F[l + j * n] = acc[r][t][0][e];
          F[n * n + l + j * n] = acc[r][t][1][e];
        }
      }
}

// ------------------------------------------------ spins of at most 32 orbitals
// One warp per (walker, spin), as orb_inv_kernel: lane r holds row r of the
// Gauss-Jordan matrix, rotated so that the pivot column is always register 0
// and the step loop stays rolled; the pivot row reaches the other lanes
// through shared memory. The inverse then goes to shared memory and F comes
// from the FP64 tensor cores: 450 instructions per matrix of 29 where lanes
// holding a row of the inverse and 8 columns of F took 3200. 0.15 ms per 4096
// walkers at 29 + 29, bound by the chains of 12 warps per SM. Both matrices have rows of LD doubles, columns
// XOR-swizzled by 4 (row mod 4): the fragments' half-warp reads (four rows,
// four columns) and the lanes' column writes fall on distinct banks.
constexpr int kRealWarps = 4;
__host__ __device__ constexpr int real_ld(int nm) { return nm <= 16 ? 16 : 32; }
__host__ __device__ constexpr size_t real_warp_doubles(int nm) {
  // orbitals, transposed inverse, two pivot rows, (s g) and pivots per orbital
  return (size_t)2 * nm * real_ld(nm) + 2 * 32 + 2 * 36 + 16;
}

template <int NM>
__global__ void __launch_bounds__(32 * kRealWarps) real_det_warp_kernel(RealArgs a, int nw) {
  static_assert(NM <= 32, "one lane per row");
  extern __shared__ __align__(16) char smem[];
  pdl_wait();
  constexpr int LD = real_ld(NM), TT = (NM + 7) / 8;
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int item = blockIdx.x * kRealWarps + wl;
  const int w = a.nt > 1 ? item >> 1 : item, spn = a.nt > 1 ? item & 1 : 0;
  const int n = spn ? a.np[1] : a.np[0], r = lane;
  if (w >= nw || n > NM || !real_on(a, w)) return;  // whole warps; nothing below waits on other warps
  double *Bs = reinterpret_cast<double *>(smem) + wl * real_warp_doubles(NM);
  double *Wt = Bs + NM * LD, *prow = Wt + NM * LD;
  double2 *sg = reinterpret_cast<double2 *>(prow + 64);
  int *perm = reinterpret_cast<int *>(sg + 36);
  auto at = [](double *m, int o, int j) -> double & { return m[o * LD + (j ^ (4 * (o & 3)))]; };
  double *F = real_base(a, w) + (spn ? a.f[1] : a.f[0]);
  // finite values wherever the tiles' padding reads
  for (int e = lane; e < (NM - n + 1) * LD; e += 32) {
    const int k = n - 1 + e / LD;
    Bs[k * LD + e % LD] = 0.0;
    Wt[k * LD + e % LD] = 0.0;
  }
  for (int e = lane; e < n * (LD - n); e += 32) {
    const int k = e / (LD - n), j = n + e - k * (LD - n);
    at(Bs, k, j) = 0.0;
    at(Wt, k, j) = 0.0;
  }
  prow[lane] = prow[32 + lane] = 0.0;
  for (int o = lane; o < 36; o += 32) sg[o] = orbital_g(a.gvec, o, n);
  __syncwarp();
  orbital_rows(a, a.scr + w * a.stride + a.l_q + 2 * (spn ? a.f0[1] : a.f0[0]), n, lane, 32,
               [&](int o, int j) -> double & { return at(Bs, o, j); });
  __syncwarp();
  double v[NM];
#pragma unroll
  for (int j = 0; j < NM; j++) v[j] = r < n && j < n ? at(Bs, r, j) : (r == j ? 1.0 : 0.0);
  bool used = r >= n;
  double my_inv = 1.0, my_d = 1.0;
  int my_l = r, sing = 0;
#pragma unroll 1
  for (int k = 0; k < NM; k++) {
    int p = k;  // an identity row's own step
    if (k < n) {
      const unsigned best = __reduce_max_sync(0xffffffffu, pivot_key(v[0], r, !used));
      p = 255 - (int)(best & 0xFFu);
      sing |= (best >> 8) == 0u;
    }
    double2 *pr = reinterpret_cast<double2 *>(prow + (k & 1) * 32);
    if (r == p)
#pragma unroll
      for (int c = 0; c < NM; c += 2) pr[c / 2] = make_double2(v[c], c + 1 < NM ? v[c + 1] : 0.0);
    __syncwarp();
    const double2 b0 = pr[0];
    const double inv = rcp_newton(b0.x);
    const bool isp = r == p;
    used = used || isp;
    if (isp) {
      my_inv = inv;
      my_d = fabs(b0.x);
      my_l = k;
    }
    const double fac = isp || r >= n ? 0.0 : v[0] * inv;
    v[0] = fma(-fac, b0.y, v[1]);
#pragma unroll
    for (int j = 2; j < NM; j += 2) {
      const double2 b = pr[j / 2];
      v[j - 1] = fma(-fac, b.x, v[j]);
      if (j + 1 < NM) v[j] = fma(-fac, b.y, v[j + 1]);
    }
    v[NM - 1] = isp ? 1.0 : -fac;
  }
  // step c's pivot row is the orbital of the inverse's column c
  if (r < n) perm[my_l] = r;
  double ld = r < n ? log(my_d) : 0.0;
#pragma unroll
  for (int q = 16; q > 0; q >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, q);
  // where a spin has more than 32 orbitals a NaN pivot counts as none, as in
  // real_inv_cta_kernel
  if (max(a.np[0], a.np[1]) > 32) sing |= __any_sync(0xffffffffu, r < n && my_d != my_d);
  __syncwarp();
  if (r < n)
#pragma unroll
    for (int c = 0; c < NM; c++)
      if (c < n) at(Wt, perm[c], my_l) = v[c] * my_inv;
  __syncwarp();
  // D2_l = -sum_o Dinv(l, o) g_a g_b D(o, l)
  if (r < n) {
    double xx = 0.0, xy = 0.0, yy = 0.0;
    for (int o = 0; o < n - 1; o++) {
      const double t = at(Wt, o, r) * at(Bs, o, r);
      const double2 g = sg[o];
      xx -= t * (g.x * g.x);
      xy -= t * (g.x * g.y);
      yy -= t * (g.y * g.y);
    }
    double *d2 = F + 2 * n * n + 2;
    d2[3 * r] = xx;
    d2[3 * r + 1] = xy;
    d2[3 * r + 2] = yy;
  }
#pragma unroll 1
  for (int lt2 = 0; lt2 < TT; lt2 += 2) {
    if (8 * lt2 >= n) break;
    double acc[2][TT][2][2] = {};
    f_products<2, TT>(acc, n, 8 * lt2, 0, sg,
                      [&](int o, int l) { return at(Wt, min(o, NM - 1), min(l, LD - 1)); },
                      [&](int o, int j) { return at(Bs, min(o, NM - 1), j); });
    f_store<2, TT>(acc, F, n, 8 * lt2, 0);
  }
  if (lane == 0) {
    F[2 * n * n] = ld;
    F[2 * n * n + 1] = (double)sing;
  }
}

// ------------------------------------------------- spins above 32 orbitals
// One CTA per (walker, spin), the whole Gauss-Jordan matrix in registers: kL
// lanes share kR rows, lane s holding their columns kL j + s in kC registers
// per row, rotated by one every kL steps so that the pivot column of step k
// is register 0 of lane k mod kL. As gj_invert_reg a step is
// one barrier: before it every warp publishes its best candidate row (key,
// reciprocal, columns), after it every thread takes the best key's row. Bound
// by shared-memory wavefronts and the step's latency chain: a pivot-row value
// read once serves kR rows: 2.19 ms for 768 matrices of 161, 0.73 for 768 of
// 113, where one row per four lanes with every value used once (shared-memory
// pipe 61%, FP64 pipe 15% busy) took 3.53 and 1.94.
// Above 128 orbitals the last kS columns of a lane, which the registers of
// one SM cannot hold, live in shared memory as a ring that the rotation
// feeds from. When both spins have at most kRealFused orbitals the
// transposed inverse and the orbitals then share the CTA's memory and F
// comes from the FP64 tensor cores here; else both go to device memory for
// real_f_kernel.
// doubles between the lanes' columns in a published row: twice an odd number,
// so the lanes' 16-byte reads fall on distinct banks
__host__ __device__ constexpr int gjc_stride(int c) { return ((c + 1) / 2 | 1) * 2; }
__host__ __device__ constexpr int gjc_slot(int l, int c) { return l * gjc_stride(c) + 2; }
__host__ __device__ inline int gjc_warps(int n, int l, int rows) {
  const int r = 32 / l * rows;  // rows per warp
  return (n + r - 1) / r;
}
inline size_t inv_cta_doubles(int n, int l, int rows, int c, int ring, bool fused) {
  // candidate rows and ring; fused: the transposed inverse in their place (there
  // is no ring), the orbitals, the scaled wave vectors
  const size_t g = gjc_warps(n, l, rows), gj = 2 * g * gjc_slot(l, c) + (size_t)ring * rows * 32 * g;
  if (!fused) return gj;
  const size_t m = (size_t)(n + 3) * odd4(n);
  return std::max(gj, m) + m + 2 * (n + 8);
}

template <int kL, int kR, int kC, int kS, int kMaxT, int kMB, bool kFused>
__global__ void __launch_bounds__(kMaxT, kMB) real_inv_cta_kernel(RealArgs a, int nw) {
  constexpr int CR = kC - kS, LS = gjc_stride(kC), SL = gjc_slot(kL, kC), RW = 32 / kL * kR;
  static_assert(!kFused || kS == 0, "the ring would share its place");
  static_assert(kC > 1, "the next pivot column is register 1 at a rotation");
  __shared__ unsigned keys[2][32];
  __shared__ double red[32], rinv[176], dk[176];
  __shared__ int perm[176], rowl[176];
  __shared__ int singular;
  extern __shared__ __align__(16) char smem[];
  pdl_wait();
  const int w = a.nt > 1 ? blockIdx.x >> 1 : blockIdx.x, spn = a.nt > 1 ? blockIdx.x & 1 : 0;
  const int n = spn ? a.np[1] : a.np[0];
  if (w >= nw || n <= 32 || !real_on(a, w)) return;  // whole CTAs
  const int t = threadIdx.x, nthr = blockDim.x, G = nthr >> 5, lane = t & 31, wp = t >> 5;
  const int s = lane & (kL - 1), r0 = wp * RW + lane / kL * kR;  // first of its rows
  double *slots = reinterpret_cast<double *>(smem);                  // [2][G][SL]
  // logical column CR + i of row q at xs[(((hd + i) mod kS) kR + q) nthr]
  double *xs = slots + 2 * G * SL + t;
  int hd = 0;
  auto xcol = [&](int i, int q) -> double & {
    const int h = hd + i;
    return xs[((h >= kS ? h - kS : h) * kR + q) * nthr];
  };
  double *base = real_base(a, w);
  const int ldw = spn ? a.ldw[1] : a.ldw[0], ld = odd4(n);
  double *Wg = base + (spn ? a.w[1] : a.w[0]), *Bg = Wg + n * ldw;  // !kFused
  double *F = base + (spn ? a.f[1] : a.f[0]);
  // kFused: the inverse over the candidate rows, the orbitals behind it
  const int gj = 2 * G * SL, mat = (n + 3) * ld;
  double *Wt = slots, *Bs = slots + max(gj, mat);
  double2 *sg = reinterpret_cast<double2 *>(Bs + mat);
  auto bat = [&](int o, int j) -> double & {
    return kFused ? Bs[o * ld + j] : Bg[o * ldw + j];
  };
  if (t == 0) singular = 0;
  if (t < 64) keys[t >> 5][t & 31] = 0u;
  orbital_rows(a, a.scr + w * a.stride + a.l_q + 2 * (spn ? a.f0[1] : a.f0[0]), n, t, nthr, bat);
  if (kFused) {
    for (int o = t; o < n + 8; o += nthr) sg[o] = orbital_g(a.gvec, o, n);
    for (int e = t; e < 3 * ld; e += nthr) Bs[n * ld + e] = 0.0;  // read past the last row
    for (int e = t; e < n * (ld - n); e += nthr) {
      const int k = e / (ld - n);
      Bs[k * ld + n + e - k * (ld - n)] = 0.0;
    }
  }
  __syncthreads();
  auto first = [&](int q, int j) {
    return r0 + q < n && kL * j + s < n ? bat(r0 + q, kL * j + s) : 0.0;
  };
  double v[kR][CR];
#pragma unroll
  for (int q = 0; q < kR; q++) {
#pragma unroll
    for (int j = 0; j < CR; j++) v[q][j] = first(q, j);
#pragma unroll
    for (int i = 0; i < kS; i++) xcol(i, q) = first(q, CR + i);
  }
  unsigned used = 0;
#pragma unroll
  for (int q = 0; q < kR; q++) used |= (r0 + q < n ? 0u : 1u) << q;
  // a column's best candidate among this thread's rows x[q]
  auto best_key = [&](const double (&x)[kR], bool own) -> unsigned {
    unsigned b = 0u;
#pragma unroll
    for (int q = 0; q < kR; q++)
      b = max(b, pivot_key(x[q], r0 + q, own && !((used >> q) & 1u)));
    return b;
  };
  auto pick = [&](const double (&x)[kR], int i) -> double {
    double y = x[0];
#pragma unroll
    for (int q = 1; q < kR; q++) y = i == q ? x[q] : y;
    return y;
  };
  // step k's candidate of this warp, whose column k is x in the lanes own
  auto publish = [&](int k, unsigned wk, bool own, const double (&x)[kR]) {
    double *sl = slots + ((k & 1) * G + wp) * SL;
    const int i = 255 - (int)(wk & 0xFFu) - r0;
    if (wk != 0u && i >= 0 && i < kR) {
#pragma unroll
      for (int q = 0; q < kR; q++)
        if (i == q) {
#pragma unroll
          for (int j = 0; j < CR; j += 2)
            *reinterpret_cast<double2 *>(sl + s * LS + j) =
                make_double2(v[q][j], j + 1 < CR ? v[q][j + 1] : 0.0);
        }
#pragma unroll
      for (int c = 0; c < kS; c++) sl[s * LS + CR + c] = xcol(c, i);
      if (own) {
        const double y = pick(x, i);
        *reinterpret_cast<double2 *>(sl + kL * LS) = make_double2(rcp_newton(y), fabs(y));
      }
    }
    if (lane == 0) keys[k & 1][wp] = wk;
  };
  double f[kR];  // the rows' entries of the pivot column
  {
    double x[kR];
#pragma unroll
    for (int q = 0; q < kR; q++) x[q] = v[q][0];
    const bool own = s == 0;
    publish(0, __reduce_max_sync(0xffffffffu, best_key(x, own)), own, x);
#pragma unroll
    for (int q = 0; q < kR; q++) f[q] = __shfl_sync(0xffffffffu, x[q], 0, kL);
  }
  // one step; kRot: the last of kL, which rotates the columns
  auto step = [&](int k, int u, auto rot) {
    constexpr bool kRot = decltype(rot)::value;
    __syncthreads();
    const unsigned best = __reduce_max_sync(0xffffffffu, keys[k & 1][lane]);
    const int p = 255 - (int)(best & 0xFFu);
    const double *ps = slots + ((k & 1) * G + p / RW) * SL;
    const double inv = ps[kL * LS];
    if (t == 0) {
      perm[k] = p;
      rowl[p] = k;
      rinv[p] = inv;
      dk[k] = ps[kL * LS + 1];
      if ((best >> 8) == 0u) singular = 1;
    }
    double fac[kR];
#pragma unroll
    for (int q = 0; q < kR; q++) fac[q] = r0 + q == p ? 0.0 : f[q] * inv;
    if (p >= r0 && p < r0 + kR) used |= 1u << (p - r0);
    const double *pc = ps + s * LS;
    // the registers of column k + 1 first: the next key needs them
    constexpr int jn = kRot ? 1 : 0;  // before the rotation
    const bool ownn = s == (kRot ? 0 : u + 1);
    double x[kR];
    {
      const double b = pc[jn];
#pragma unroll
      for (int q = 0; q < kR; q++) x[q] = fma(-fac[q], b, v[q][jn < CR ? jn : 0]);
    }
    const unsigned wk = __reduce_max_sync(0xffffffffu, best_key(x, ownn));
    double done[kR];  // the eliminated column
#pragma unroll
    for (int q = 0; q < kR; q++) done[q] = r0 + q == p ? 1.0 : -fac[q];
    const bool own = s == u;
    if (!kRot) {
#pragma unroll
      for (int j = 0; j < CR; j += 2) {
        const double2 b = *reinterpret_cast<const double2 *>(pc + j);
#pragma unroll
        for (int q = 0; q < kR; q++) {
          v[q][j] = fma(-fac[q], b.x, v[q][j]);
          if (j + 1 < CR) v[q][j + 1] = fma(-fac[q], b.y, v[q][j + 1]);
        }
      }
#pragma unroll
      for (int c = 0; c < kS; c++) {
        const double b = pc[CR + c];
#pragma unroll
        for (int q = 0; q < kR; q++) xcol(c, q) = fma(-fac[q], b, xcol(c, q));
      }
#pragma unroll
      for (int q = 0; q < kR; q++) v[q][0] = own ? done[q] : v[q][0];
    } else {
      double head[kR];
#pragma unroll
      for (int j = 0; j < CR; j += 2) {
        const double2 b = *reinterpret_cast<const double2 *>(pc + j);
#pragma unroll
        for (int q = 0; q < kR; q++) {
          if (j) v[q][j - 1] = fma(-fac[q], b.x, v[q][j]);
          else head[q] = own ? done[q] : fma(-fac[q], b.x, v[q][0]);
          if (j + 1 < CR) v[q][j] = fma(-fac[q], b.y, v[q][j + 1]);
        }
      }
      if constexpr (kS > 0) {
        const double b = pc[CR];
#pragma unroll
        for (int q = 0; q < kR; q++) v[q][CR - 1] = fma(-fac[q], b, xcol(0, q));
#pragma unroll
        for (int c = 1; c < kS; c++) {
          const double bc = pc[CR + c];
#pragma unroll
          for (int q = 0; q < kR; q++) xcol(c, q) = fma(-fac[q], bc, xcol(c, q));
        }
#pragma unroll
        for (int q = 0; q < kR; q++) xcol(0, q) = head[q];
        hd = hd + 1 == kS ? 0 : hd + 1;
      } else {
#pragma unroll
        for (int q = 0; q < kR; q++) v[q][CR - 1] = head[q];
      }
    }
    if (k + 1 < n) {
      publish(k + 1, wk, ownn, x);
#pragma unroll
      for (int q = 0; q < kR; q++)
        f[q] = __shfl_sync(0xffffffffu, v[q][0], kRot ? 0 : u + 1, kL);
    }
  };
  int turns = 0;  // rotations done
#pragma unroll 1
  for (int k0 = 0; k0 < n; k0 += kL) {
    const int m = min(kL - 1, n - k0);
#pragma unroll 1
    for (int u = 0; u < m; u++) step(k0 + u, u, std::false_type());
    if (k0 + kL - 1 < n) {
      step(k0 + kL - 1, kL - 1, std::true_type());
      turns++;
    }
  }
  __syncthreads();  // perm, rowl, rinv, dk; the last step's candidates are read
  // rows normalised by their own pivot, transposed and in orbital order;
  // register j holds column kL ((turns + j) mod kC) + s
  auto store = [&](int j, int q, double x) {
    const int m = turns + j, c = kL * (m >= kC ? m - kC : m) + s, r = r0 + q;
    if (r < n && c < n)
      (kFused ? Wt + perm[c] * ld : Wg + perm[c] * ldw)[rowl[r]] = x * rinv[r];
  };
#pragma unroll
  for (int q = 0; q < kR; q++) {
#pragma unroll
    for (int j = 0; j < CR; j++) store(j, q, v[q][j]);
#pragma unroll
    for (int i = 0; i < kS; i++) store(CR + i, q, xcol(i, q));
  }
  if (kFused) {
    for (int e = t; e < 3 * ld; e += nthr) Wt[n * ld + e] = 0.0;
    for (int e = t; e < n * (ld - n); e += nthr) {
      const int k = e / (ld - n);
      Wt[k * ld + n + e - k * (ld - n)] = 0.0;
    }
  }
  // a NaN pivot counts as none, as in the complex kernels of these spins (looked
  // at here, off the chain of the pivot steps)
  if (t < n && dk[t] != dk[t]) singular = 1;
  double lg = t < n ? log(dk[t]) : 0.0;
#pragma unroll
  for (int q = 16; q > 0; q >>= 1) lg += __shfl_xor_sync(0xffffffffu, lg, q);
  if (lane == 0) red[wp] = lg;
  __syncthreads();
  if (t == 0) {
    double sum = 0.0;
    for (int q = 0; q < G; q++) sum += red[q];
    F[2 * n * n] = sum;
    F[2 * n * n + 1] = (double)singular;
  }
  if constexpr (kFused) {
    // D2_l = -sum_o Dinv(l, o) g_a g_b D(o, l), eight lanes per electron
    for (int lb = 0; lb < n; lb += nthr / 8) {
      const int l = lb + (t >> 3);
      double xx = 0.0, xy = 0.0, yy = 0.0;
      if (l < n)
        for (int o = t & 7; o < n - 1; o += 8) {
          const double x = Wt[o * ld + l] * Bs[o * ld + l];
          const double2 g = sg[o];
          xx -= x * (g.x * g.x);
          xy -= x * (g.x * g.y);
          yy -= x * (g.y * g.y);
        }
      xx = group8_sum(xx);
      xy = group8_sum(xy);
      yy = group8_sum(yy);
      if (l < n && (t & 7) == 0) {
        double *d2 = F + 2 * n * n + 2 + 3 * l;
        d2[0] = xx;
        d2[1] = xy;
        d2[2] = yy;
      }
    }
    // items of one row tile and up to four column tiles
    const int T = (n + 7) / 8, TC = (T + 3) / 4;
    for (int it = wp; it < T * TC; it += G) {
      const int l0 = 8 * (it / TC), j0 = 32 * (it % TC);
      double acc[1][4][2][2] = {};
      f_products<1, 4>(acc, n, l0, j0, sg,
                       [&](int o, int l) { return Wt[o * ld + min(l, ld - 1)]; },
                       [&](int o, int j) { return Bs[o * ld + min(j, ld - 1)]; });
      f_store<1, 4>(acc, F, n, l0, j0);
    }
  }
}

// F and D2 when the larger spin has more than kRealFused orbitals: a CTA takes every row and 32
// columns of F; the 32 orbital columns are resident, the transposed inverse
// streams through two buffers of kFK orbitals. A warp holds two row tiles
// and four column tiles of F_x and F_y.
constexpr int kFK = 16, kFLd = 36, kFThreads = 352;

inline size_t real_f_doubles(int n, int ldw) {
  return (size_t)(n + 15) / 16 * 16 * kFLd + (size_t)2 * kFK * odd4(ldw) + 2 * (n + 16);
}

__global__ void __launch_bounds__(kFThreads, 1) real_f_kernel(RealArgs a, int nw, int blocks) {
  extern __shared__ __align__(16) char smem[];
  pdl_wait();
  const int bj = blockIdx.x % blocks, item = blockIdx.x / blocks;
  const int w = a.nt > 1 ? item >> 1 : item, spn = a.nt > 1 ? item & 1 : 0;
  const int n = spn ? a.np[1] : a.np[0], j0 = 32 * bj;
  if (w >= nw || n <= 32 || j0 >= n || !real_on(a, w)) return;  // whole CTAs
  const int t = threadIdx.x, wp = t >> 5, lane = t & 31, lg = lane >> 2, lt = lane & 3;
  double *base = real_base(a, w);
  const int ldw = spn ? a.ldw[1] : a.ldw[0], ld = odd4(ldw), rows = (n + 15) / 16 * 16;
  const double *Wg = base + (spn ? a.w[1] : a.w[0]), *Bg = Wg + n * ldw;
  double *F = base + (spn ? a.f[1] : a.f[0]);
  double *Bs = reinterpret_cast<double *>(smem), *Wb = Bs + (size_t)rows * kFLd;
  double2 *sg = reinterpret_cast<double2 *>(Wb + (size_t)2 * kFK * ld);
  auto stage = [&](int c) {  // orbitals c kFK ..: rows of ldw doubles, 16-byte copies
    double *dst = Wb + (c & 1) * kFK * ld;
    const int q = ldw / 2;
    for (int e = t; e < kFK * q; e += kFThreads) {
      const int o = e / q, x = e - o * q;
      if (c * kFK + o < n)
        cp_async16(dst + o * ld + 2 * x, Wg + (size_t)(c * kFK + o) * ldw + 2 * x);
      else
        *reinterpret_cast<double2 *>(dst + o * ld + 2 * x) = make_double2(0.0, 0.0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage(0);
  for (int o = t; o < n + 16; o += kFThreads) sg[o] = orbital_g(a.gvec, o, n);
  for (int e = t; e < rows * 32; e += kFThreads) {
    const int o = e >> 5, j = e & 31;
    Bs[o * kFLd + j] = o < n && j0 + j < n ? Bg[o * ldw + j0 + j] : 0.0;
  }
  double acc[2][4][2][2] = {};
  double d2[3] = {0.0, 0.0, 0.0};
  const int l0 = 16 * wp, nc = rows / kFK;
  for (int c = 0; c < nc; c++) {
    if (c + 1 < nc) stage(c + 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const double *W = Wb + (c & 1) * kFK * ld;
    if (l0 < n)
#pragma unroll
      for (int k = 0; k < kFK; k += 4) {
        const int o = c * kFK + k + lt;
        const double2 g = sg[o];
        double ax[2], ay[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
          const double x = W[(k + lt) * ld + min(l0 + 8 * r + lg, ldw - 1)];
          ax[r] = x * g.x;
          ay[r] = x * g.y;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const double v = Bs[(o ^ 1) * kFLd + 8 * q + lg];
#pragma unroll
          for (int r = 0; r < 2; r++) {
            dmma_m8n8k4(acc[r][q][0], ax[r], v);
            dmma_m8n8k4(acc[r][q][1], ay[r], v);
          }
        }
      }
    if (t < 32 && j0 + t < n)  // D2 of these 32 electrons
      for (int k = 0; k < kFK; k++) {
        const double2 g = sg[c * kFK + k];
        const double x = W[k * ld + j0 + t] * Bs[(c * kFK + k) * kFLd + t];
        d2[0] -= x * (g.x * g.x);
        d2[1] -= x * (g.x * g.y);
        d2[2] -= x * (g.y * g.y);
      }
    __syncthreads();  // this buffer may be refilled
  }
  if (l0 < n) f_store<2, 4>(acc, F, n, l0, j0);
  if (t < 32 && j0 + t < n)
    for (int q = 0; q < 3; q++) F[2 * n * n + 2 + 3 * (j0 + t) + q] = d2[q];
}

// ------------------------------------------------- S, drift and Laplacian
// S_jk[a][c] = sum_i sum_b J_ji[a][b] J_ki[c][b] of one (walker, spin) on the
// FP64 tensor cores (mma.m8n8k4): in shared memory the Jacobian planes (xx,
// xy, yy) are matrices of rows j and columns i, so for 8 x 8 tiles of (j, k)
// and four electrons a warp loads three fragments per tile and issues eight
// products ((a, c) pairs times b; J is symmetric in (a, b)). The columns hold
// type 0's electrons, then type 1's, each padded with zeros to a multiple of
// four, and their stride is an odd multiple of four: the fragments' reads
// fall on distinct banks. At the end every lane multiplies its S entries by
// F_a(k,j) F_c(j,k) (and D2_j on the diagonal) and the CTA sums them. Bound by
// the FP64 pipe (one product of 256 FMAs per 16 cycles and sub-partition).
//
// kB: tiles per side of a warp's item. kB = 1 keeps its columns resident: those
// of both types, a tile pair's two types in one item, or (launch_s) those of
// one type per CTA, up to about 96 orbitals; kB = 2 streams chunks of columns
// through two buffers, one type after the other.
// Measured on one B200: 29 + 29, 4096 walkers 0.25 ms (0.60 with the
// move's end, as 3 x 3 register tiles of FMAs there); 161 polarised, 768 walkers 1.95 ms, 2.48
// before the staging visited only the triangle rows of its chunk and the last
// round's items were shared by several warps.
__host__ __device__ inline int s_chunk(int n) {  // columns per chunk: two buffers in 176 KB
  const int c = (int)(88 * 1024 / (sizeof(double) * 3 * n)) / 4;
  return (c & 1 ? c : c - 1) * 4;
}

// The three planes' entries at e of the triangle into shared address d
// (asynchronous 8-byte copies).
__device__ __forceinline__ void copy_entry(unsigned d, unsigned pl, const double *e, int jp) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(e) : "memory");
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + pl), "l"(e + jp) : "memory");
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + 2 * pl), "l"(e + 2 * jp) : "memory");
}

// The columns of one type (from column c0 of dst's first on, padded
// numbering) of spin spn's electrons j into dst[p][j][c], zeros in the padding.
// One pass over the triangle's rows r that hold them, lanes on consecutive
// entries (r, c): of the spin's own type each goes to (j, i) = (r, c) and
// (c, r); between the types to (r, c) or, for type 1's electrons, (c, r).
__device__ inline void stage_type(const RealArgs &a, double *dst, int ld, const double *jg, int spn,
                                  int type) {
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, nw = blockDim.x >> 5;
  const int n0 = a.np[0], N = a.N, n = spn ? a.np[1] : n0, f0 = spn ? n0 : 0;
  const int i0 = type ? n0 : 0, ni = type ? a.np[1] : n0;
  const bool own = spn == type;
  const int rb = own ? f0 : 0, re = own ? f0 + n : n0, ce = own ? re : N;
  const unsigned pl = 8 * n * ld, d = (unsigned)__cvta_generic_to_shared(dst);
  for (int r = rb + warp; r < re; r += nw) {
    const double *src = jg + jac_row(N, r);
    const unsigned row = d + 8 * ((r - f0) * ld - i0), col = d + 8 * (r - i0 - f0 * ld);
    for (int c = (own ? r : n0) + lane; c < ce; c += 32) {
      if (own || !spn) copy_entry(row + 8 * c, pl, src + c, a.jp);
      if (own ? c > r : spn) copy_entry(col + 8 * c * ld, pl, src + c, a.jp);
    }
  }
  const int np = -ni & 3;
  for (int e = t; e < n * np; e += blockDim.x) {
    double *z = dst + e / np * ld + ni + e % np;
    z[0] = z[n * ld] = z[2 * n * ld] = 0.0;
  }
}

// Columns c0 .. c1-1 of one type: from row j of the triangle for i >= j (lanes
// on consecutive i), from row i for i < j (lanes on consecutive j).
__device__ inline void stage_cols(const RealArgs &a, double *dst, int ld, const double *jg, int f0,
                                  int n, int c0, int c1) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int n0 = a.np[0], shift = a.pad0 - n0, t1 = c0 >= a.pad0;
  // electrons i0 .. i1-1; columns from i1 on are padding
  const int i0 = t1 ? c0 - shift : c0, i1 = min(t1 ? c1 - shift : c1, t1 ? a.N : n0);
  const unsigned pl = 8 * n * ld, d = (unsigned)__cvta_generic_to_shared(dst);
  for (int j = f0 + warp; j < min(f0 + n, i1); j += nw) {
    const double *src = jg + jac_row(a.N, j);
    for (int i = max(j, i0) + lane; i < i1; i += 32)
      copy_entry(d + 8 * ((j - f0) * ld + i - i0), pl, src + i, a.jp);
  }
  for (int i = i0 + warp; i < i1; i += nw) {
    const double *src = jg + jac_row(a.N, i);
    const unsigned col = d + 8 * (i - i0);
    for (int j = max(f0, i + 1) + lane; j < f0 + n; j += 32)
      copy_entry(col + 8 * ((j - f0) * ld), pl, src + j, a.jp);
  }
  const int np = c1 - c0 - (i1 - i0);
  for (int e = threadIdx.x; e < n * np; e += blockDim.x) {
    double *z = dst + e / np * ld + (i1 - i0) + e % np;
    z[0] = z[n * ld] = z[2 * n * ld] = 0.0;
  }
}

// Products of kB x kB tile pairs over the columns [k0, k1) of a buffer.
template <int kB>
__device__ __forceinline__ void s_products(double (&acc)[kB][kB][4][2], const double *buf, int ld,
                                           int n, int tj, int tk, int k0, int k1, int step = 4) {
  const int lane = threadIdx.x & 31, lg = lane >> 2, lt = lane & 3;
  const int pl = n * ld;
  const double *pj[kB], *pk[kB];
#pragma unroll
  for (int a = 0; a < kB; a++) {
    pj[a] = buf + min(8 * (kB * tj + a) + lg, n - 1) * ld + lt;
    pk[a] = buf + min(8 * (kB * tk + a) + lg, n - 1) * ld + lt;
  }
#pragma unroll 2
  for (int c = k0; c < k1; c += step) {
    double j[kB][3], k[kB][3];
#pragma unroll
    for (int a = 0; a < kB; a++)
#pragma unroll
      for (int p = 0; p < 3; p++) {
        j[a][p] = pj[a][p * pl + c];
        k[a][p] = pk[a][p * pl + c];
      }
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
      for (int a = 0; a < kB; a++)
#pragma unroll
        for (int d = 0; d < kB; d++)
#pragma unroll
          for (int q = 0; q < 4; q++)
            dmma_m8n8k4(acc[a][d][q], j[a][(q >> 1) + b], k[d][(q & 1) + b]);
  }
}

// The shares lt[0 .. kN) of the Laplacian of one item's kN sets of sums: S times
// F_a(k,j) F_c(j,k), unordered pairs of tiles twice, and D2 on the diagonal.
template <int kB, int kN>
__device__ __forceinline__ void s_contract(const double (&acc)[kN][kB][kB][4][2], const double *FX,
                                           const double *d2, int n, int tj, int tk, double *lt) {
  const int lane = threadIdx.x & 31, lg = lane >> 2, lq = lane & 3;
  const double *FY = FX + n * n;
#pragma unroll
  for (int a = 0; a < kB; a++)
#pragma unroll
    for (int d = 0; d < kB; d++) {
      const int jt = kB * tj + a, kt = kB * tk + d;
      if (kB > 1 && jt > kt) continue;  // inside a diagonal item: the other order counts
      const double wgt = jt == kt ? 1.0 : 2.0;
      const int j = 8 * jt + lg;
      // the loads of both entries in flight together. They are plain ones: the
      // read-only path is not for what a kernel before wrote that may still run
      // when this one starts.
      double f[2][4];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int jc = min(j, n - 1), kc = min(8 * kt + 2 * lq + e, n - 1);
        const int kj = kc + jc * n, jk = jc + kc * n;
        f[e][0] = FX[kj];
        f[e][1] = FX[jk];
        f[e][2] = FY[kj];
        f[e][3] = FY[jk];
      }
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int k = 8 * kt + 2 * lq + e;
        if (j < n && k < n) {
          const double xkj = wgt * f[e][0], xjk = f[e][1], ykj = wgt * f[e][2], yjk = f[e][3];
          double m0 = xkj * xjk, m1 = xkj * yjk, m2 = ykj * xjk, m3 = ykj * yjk;
          if (j == k) {
            m0 -= d2[3 * j];
            m1 -= d2[3 * j + 1];
            m2 -= d2[3 * j + 1];
            m3 -= d2[3 * j + 2];
          }
#pragma unroll
          for (int q = 0; q < kN; q++)
            lt[q] += m0 * acc[q][a][d][0][e] + m1 * acc[q][a][d][1][e] +
                     m2 * acc[q][a][d][2][e] + m3 * acc[q][a][d][3][e];
        }
      }
    }
}

// tile pair (tj <= tk) of index tp in the row-major lower triangle
__device__ __forceinline__ void tile_pair(int tp, int *tj, int *tk) {
  int k = (int)((sqrtf(8.0f * (float)tp + 1.0f) - 1.0f) * 0.5f);
  if (k * (k + 1) / 2 > tp) k--;
  if ((k + 1) * (k + 2) / 2 <= tp) k++;
  *tk = k;
  *tj = tp - k * (k + 1) / 2;
}

inline size_t s_smem_doubles(int n, int cols, bool resident) {
  // f, D2, warp sums, then the columns
  const size_t head = 2 * (size_t)n + ((3 * (size_t)n + 1) & ~size_t(1)) + 2 * 32;
  return head + (resident ? (size_t)3 * n * odd4(cols) : (size_t)2 * 3 * n * s_chunk(n));
}

constexpr int kSMaxThreads = 768;  // kB = 1: at most 80 registers, 24 warps on an SM

template <int kB>
__global__ void __launch_bounds__(kB == 1 ? kSMaxThreads : 512, 1)
    real_s_kernel(RealArgs a, const DevSys *ds, int nw, int split) {
  extern __shared__ __align__(16) char smem[];
  pdl_wait();
  // split (kB = 1, two types): one CTA per type of the columns
  const int item = blockIdx.x >> split, type = split ? blockIdx.x & 1 : 0;
  const int w = a.nt > 1 ? item >> 1 : item, spn = a.nt > 1 ? item & 1 : 0;
  if (w >= nw || !real_on(a, w)) return;  // whole CTAs
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, nthr = blockDim.x, NW = nthr >> 5;
  const int nt = a.nt, n = spn ? a.np[1] : a.np[0], f0 = spn ? a.f0[1] : a.f0[0];
  double *base = real_base(a, w);
  const double *FX = base + (spn ? a.f[1] : a.f[0]);
  double *out = base + (spn ? a.s[1] : a.s[0]);
  double *fd = reinterpret_cast<double *>(smem), *d2 = fd + 2 * n;
  double *red = d2 + ((3 * n + 1) & ~1), *jac = red + 2 * 32;
  const bool timed = ds->phase != nullptr;
  long long tph = timed ? clock64() : 0;
  auto mark = [&](int k) {
    if (timed) phase_mark(*ds, k, tph, t == 0);
  };
  const int n0 = a.np[0];
  // split: the type's columns in buffer numbering 0 .. cols-1
  const int pad0 = type ? 0 : a.pad0;
  const int cols = split ? (type ? a.cols - a.pad0 : a.pad0) : a.cols;
  const int ic = kB == 1 ? cols : s_chunk(n), ld = kB == 1 ? odd4(cols) : ic;
  const size_t bufd = (size_t)3 * n * ld;
  // kB = 2: chunks never span both types
  const int nch0 = kB == 1 ? 1 : (pad0 + ic - 1) / ic;
  const int nch = kB == 1 ? 1 : nch0 + (nt > 1 ? (cols - pad0 + ic - 1) / ic : 0);
  auto chunk = [&](int ch, int *c0, int *c1) {
    if (kB == 1) {
      *c0 = 0;
      *c1 = cols;
    } else if (ch < nch0) {
      *c0 = ch * ic;
      *c1 = min(pad0, *c0 + ic);
    } else {
      *c0 = pad0 + (ch - nch0) * ic;
      *c1 = min(cols, *c0 + ic);
    }
  };
  auto stage = [&](int ch, int buf) {
    int c0, c1;
    chunk(ch, &c0, &c1);
    if (kB == 1) {
      stage_type(a, jac, ld, base, spn, type);
      if (nt > 1 && !split) stage_type(a, jac + a.pad0, ld, base, spn, 1);
    } else stage_cols(a, jac + buf * bufd, ld, base, f0, n, c0, c1);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage(0, 0);
  for (int e = t; e < 2 * n; e += nthr)
    fd[e] = FX[(e & 1 ? n * n : 0) + (e >> 1) * (n + 1)];
  for (int e = t; e < 3 * n; e += nthr) d2[e] = FX[2 * n * n + 2 + e];
  double lt[2] = {0.0, 0.0};
  // drift of the columns of a buffer: four lanes per electron
  auto drift = [&](const double *buf, int c0, int c1) {
    const int l4 = t & 3, pl = n * ld;
    for (int cb = c0; cb < c1; cb += nthr / 4) {
      const int c = cb + (t >> 2), x = c < pad0 ? c : c - pad0;
      const bool on = c < c1 && x < (c < pad0 ? n0 : a.np[1]);
      double gx = 0.0, gy = 0.0;
      if (on)
        for (int j = l4; j < n; j += 4) {
          const double *r = buf + j * ld + (c - c0);
          const double xx = r[0], xy = r[pl], yy = r[2 * pl];
          const double2 f = *reinterpret_cast<const double2 *>(fd + 2 * j);
          gx += xx * f.x + xy * f.y;
          gy += xy * f.x + yy * f.y;
        }
      gx = group_sum<4>(gx);
      gy = group_sum<4>(gy);
      if (on && l4 < 2) out[2 * (c < pad0 ? c : n0 + x) + l4] = l4 ? -gy : -gx;
    }
  };
  const int T = ((n + 7) / 8 + kB - 1) / kB, pairs = T * (T + 1) / 2;
  if constexpr (kB == 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    mark(PH_DRIFT);
    drift(jac, 0, cols);
    // (tile pair, type) items in whole runs per warp: a tile pair whose types
    // fall to two warps is contracted by both
    const bool one = nt == 1 || split;
    const int items = one ? pairs : 2 * pairs;
    const int i0 = items * warp / NW, i1 = items * (warp + 1) / NW;
    for (int it = i0; it < i1;) {
      const int tp = one ? it : it >> 1;
      const bool first = one || !(it & 1), second = !one && 2 * tp + 1 < i1;
      int tj, tk;
      tile_pair(tp, &tj, &tk);
      double acc[2][1][1][4][2] = {};
      if (first) s_products<1>(acc[0], jac, ld, n, tj, tk, 0, one ? cols : pad0);
      if (second) s_products<1>(acc[1], jac, ld, n, tj, tk, pad0, cols);
      s_contract<1, 2>(acc, FX, d2, n, tj, tk, lt);
      it = (one ? tp : 2 * tp + 1) + 1;
    }
    if (type) {  // the sums are type 1's
      lt[1] = lt[0];
      lt[0] = 0.0;
    }
  } else {
    const int rounds = (pairs + NW - 1) / NW;
    for (int round = 0; round < rounds; round++) {
      // the last round's items are shared by ks warps each, which take every
      // ks-th product step of a chunk (the contraction is linear in the sums)
      const int left = min(pairs - round * NW, NW), ks = NW / left;
      const int it = round * NW + warp % left, kq = warp / left;
      const bool on = kq < ks;
      int tj = 0, tk = 0;
      if (on) tile_pair(it, &tj, &tk);
      double acc[1][kB][kB][4][2];
      for (int ch = 0; ch < nch; ch++) {
        if (ch == 0 || ch == nch0)
#pragma unroll
          for (int q = 0; q < kB * kB * 8; q++) (&acc[0][0][0][0][0])[q] = 0.0;
        // this chunk is in flight; the next one (of this round or the
        // first of the next) goes to the other buffer
        const int seq = round * nch + ch;
        if (ch + 1 < nch || round + 1 < rounds)
          stage(ch + 1 < nch ? ch + 1 : 0, (seq + 1) & 1);
        else
          asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        int c0, c1;
        chunk(ch, &c0, &c1);
        const double *buf = jac + (seq & 1) * bufd;
        if (round == 0) drift(buf, c0, c1);
        if (on) s_products<kB>(acc[0], buf, ld, n, tj, tk, 4 * kq, c1 - c0, 4 * ks);
        if (on && (ch + 1 == nch0 || ch + 1 == nch)) {
          double s = 0.0;
          s_contract<kB, 1>(acc, FX, d2, n, tj, tk, &s);
          lt[0] += ch < nch0 ? s : 0.0;
          lt[1] += ch < nch0 ? 0.0 : s;
        }
        __syncthreads();  // this chunk's buffer may be refilled
      }
    }
  }
  // - sum_j f_j . L_j
  const double *o = a.scr + w * a.stride;
  for (int e = t; e < 2 * n; e += nthr) {
    if (!type) lt[0] -= fd[e] * o[a.l_qbd + 2 * f0 + e];
    if (split ? type : nt > 1) lt[1] -= fd[e] * o[a.l_sb + 2 * f0 + e];
  }
#pragma unroll
  for (int q = 16; q > 0; q >>= 1) {
    lt[0] += __shfl_xor_sync(0xffffffffu, lt[0], q);
    lt[1] += __shfl_xor_sync(0xffffffffu, lt[1], q);
  }
  if (lane == 0) {
    red[2 * warp] = lt[0];
    red[2 * warp + 1] = lt[1];
  }
  __syncthreads();
  if (t < 2 && (!split || t == type)) {
    double s = 0.0;
    for (int q = 0; q < NW; q++) s += red[2 * q + t];
    out[2 * a.N + t] = s;
  }
  mark(PH_CROSS);
}

// Warps per CTA of the resident form, by the CTAs an SM's shared memory holds
// (us with the orbital kernel, one B200: 13 + 13, 4096 walkers: 3 warps 109, 4
// 117; 29 + 29: 4 443, 5 421, 6 413, 8 441; 37 + 37, 1001: 6 253, 8 244, 12 264;
// 45 + 45, 1024: 8 374, 10 364, 12 384; 61 + 61, a type per CTA: 8 749, 10 710, 12 698).
int s_warps(int n, size_t smem) {
  const int ctas = 227 * 1024 / (int)(smem + 1024);
  if (ctas >= 8) return 3;
  if (ctas >= 5) return 4;
  if (ctas == 4) return 6;
  if (ctas == 3 || n <= 40) return 8;
  if (ctas == 2) return n <= 45 ? 10 : 12;
  return 20;
}

cudaError_t launch_s(const DevSys &hs, const DevSys *ds, const RealArgs &a, int nw,
                     cudaStream_t st) {
  auto doubles = [&](int cols, bool resident) {
    size_t d = 0;
    for (int t = 0; t < hs.nt; t++) d = std::max(d, s_smem_doubles(hs.np[t], cols, resident));
    return sizeof(double) * d;
  };
  size_t sm = doubles(a.cols, true);
  // One CTA per type of the columns where an SM would hold one CTA with both
  // (or none): two or three then overlap staging and products (us with the
  // orbital kernel, 1024 walkers: 49 + 49: 549 -> 483, 61 + 61: 742 -> 698, 81 + 45:
  // 1757 -> 1387, 81 + 81: 2630 -> 2014, streamed before). Where two or more fit,
  // F read twice costs more: 29 + 29: 403 -> 420, 37 + 37: 240 -> 246, 45 + 45:
  // 359 -> 364.
  const int split = hs.nt > 1 && 2 * (sm + 1024) > 227 * 1024;
  if (split) sm = doubles(std::max(a.pad0, a.cols - a.pad0), true);
  const bool resident = sm <= 226 * 1024;
  if (!resident) sm = doubles(a.cols, false);
  const void *k = resident ? (const void *)real_s_kernel<1> : (const void *)real_s_kernel<2>;
  cudaError_t e = raise_smem_limit(k, sm);
  if (e != cudaSuccess) return e;
  return resident ? launch_pdl(real_s_kernel<1>, nw * hs.nt << split, 32 * s_warps(hs.nmax, sm),
                               sm, st, a, ds, nw, split)
                  : launch_pdl(real_s_kernel<2>, nw * hs.nt, 512, sm, st, a, ds, nw, 0);
}

template <int kL, int kR, int kC, int kS, int kMaxT, int kMB, bool kFused>
cudaError_t launch_inv_cta(const RealArgs &a, int n, int items, int nw, cudaStream_t st) {
  const size_t sm = sizeof(double) * inv_cta_doubles(n, kL, kR, kC, kS, kFused);
  auto k = real_inv_cta_kernel<kL, kR, kC, kS, kMaxT, kMB, kFused>;
  cudaError_t e = raise_smem_limit((const void *)k, sm);
  if (e != cudaSuccess) return e;
  return launch_pdl(k, items, 32 * gjc_warps(n, kL, kR), sm, st, a, nw);
}

template <int NM>
cudaError_t launch_det_warp(const RealArgs &a, int items, int nw, cudaStream_t st) {
  const size_t sm = sizeof(double) * kRealWarps * real_warp_doubles(NM);
  const void *k = (const void *)real_det_warp_kernel<NM>;
  cudaError_t e = raise_smem_limit(k, sm);
  if (e != cudaSuccess) return e;
  return launch_pdl(real_det_warp_kernel<NM>, (items + kRealWarps - 1) / kRealWarps,
                    32 * kRealWarps, sm, st, a, nw);
}

cudaError_t launch_orbitals_f(const DevSys &hs, const RealArgs &a, int nw, cudaStream_t st) {
  const int items = nw * hs.nt, nm = hs.nmax;
  // registers for the rows: the closed shells' sizes 13, 21, 25 and 29
  // exactly, others padded to 16 or 32 columns
  if (nm <= 13) return launch_det_warp<13>(a, items, nw, st);
  if (nm <= 16) return launch_det_warp<16>(a, items, nw, st);
  if (nm <= 21) return launch_det_warp<21>(a, items, nw, st);
  if (nm <= 25) return launch_det_warp<25>(a, items, nw, st);
  if (nm <= 29) return launch_det_warp<29>(a, items, nw, st);
  if (nm <= 32) return launch_det_warp<32>(a, items, nw, st);
  cudaError_t e;
  if (hs.nt > 1 && std::min(hs.np[0], hs.np[1]) <= 32) {
    // spins on both sides of 32: the warp kernel takes the smaller one
    if ((e = launch_det_warp<32>(a, items, nw, st)) != cudaSuccess) return e;
  }
  // lanes per group of rows, rows, columns per lane, of them in shared memory,
  // most threads, CTAs per SM that the registers are kept for
  e = nm <= 40           ? launch_inv_cta<8, 4, 5, 0, 96, 6, true>(a, nm, items, nw, st)
      : nm <= 48         ? launch_inv_cta<8, 4, 6, 0, 96, 6, true>(a, nm, items, nw, st)
      : nm <= 64         ? launch_inv_cta<8, 4, 8, 0, 128, 3, true>(a, nm, items, nw, st)
      : nm <= 88         ? launch_inv_cta<8, 4, 11, 0, 192, 2, true>(a, nm, items, nw, st)
      : nm <= 104        ? launch_inv_cta<8, 4, 13, 0, 224, 1, true>(a, nm, items, nw, st)
      : nm <= kRealFused ? launch_inv_cta<8, 4, 15, 0, 256, 1, true>(a, nm, items, nw, st)
      : nm <= 128        ? launch_inv_cta<8, 4, 16, 0, 256, 1, false>(a, nm, items, nw, st)
      : nm <= 144        ? launch_inv_cta<16, 8, 9, 1, 288, 1, false>(a, nm, items, nw, st)
      : nm <= 160        ? launch_inv_cta<16, 8, 10, 2, 320, 1, false>(a, nm, items, nw, st)
                         : launch_inv_cta<16, 8, 11, 3, 352, 1, false>(a, nm, items, nw, st);
  if (e != cudaSuccess || nm <= kRealFused) return e;
  const int blocks = (nm + 31) / 32;
  const size_t sm = sizeof(double) * real_f_doubles(nm, (nm + 3) & ~3);
  if ((e = raise_smem_limit((const void *)real_f_kernel, sm)) != cudaSuccess) return e;
  return launch_pdl(real_f_kernel, items * blocks, kFThreads, sm, st, a, nw, blocks);
}

}  // namespace

cudaError_t launch_real_det(const DevSys &hs, const DevSys *ds, int nw, double *scr,
                            cudaStream_t st, bool some) {
  if (nw <= 0) return cudaSuccess;
  RealArgs a = real_args(hs, scr);
  if (some) a.l_grows = move_scratch(hs).grows;
  const cudaError_t e = launch_orbitals_f(hs, a, nw, st);
  // a backflow of zeros needs no sums over Jacobian blocks (eval_det_real)
  if (e != cudaSuccess || hs.bf_zero) return e;
  return launch_s(hs, ds, a, nw, st);
}

}  // namespace q2d
