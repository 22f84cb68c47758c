// real_det.cuh - determinants over real orbitals (DevSys::real_orb): the
// walker's scratch layout, the real-orbital kernels' launchers, and the part
// of the evaluation that follows them.
//
// At the Gamma point the plane waves of an odd number of orbitals come as
// k = 0 and pairs +-k. The unitary combination of exp(ik.q) and exp(-ik.q),
// sqrt(2) cos(k.q) and sqrt(2) sin(k.q), leaves |det| and D^-1 grad D as they
// are and makes every matrix real: the inverse takes a quarter of the
// products, F_a = D^-1 d_a D is real, and the phase gradient is zero.
//
// With J_ji[a][b] = dq_ja/dx_ib the backflow Jacobian blocks and f_j the
// diagonal of F, the determinant's Laplacian over the electrons i of type t
// (slater_excitations, reptation.f:10201-10259) is
//   -sum_i lap_i ln|D| = -sum_j f_j.L_j - sum_j D2_j : S_jj
//                        + sum_jk sum_ac F_a(k,j) F_c(j,k) S_jk[a][c],
//   S_jk = sum_{i in t} J_ji J_ki,  L_j = sum_{i in t} lap_i q_j,
//   D2_j[a][c] = sum_k F_a(j,k) F_c(k,j) (the second derivatives of plane waves).
// S needs the Jacobian blocks alone, so its sums (eight FP64 instructions
// per pair and electron) run from registers and F is read once at the end,
// where the complex form multiplies a 2n x 2n matrix built from F by every
// Jacobian column.
#pragma once

#include "kernels.cuh"
#include "walker_eval.cuh"

namespace q2d {

// The sizes and offsets the real-orbital kernels need, formed once on the
// host: a kernel that reads them from its parameters spends no instructions
// on them.
struct RealArgs {
  int N, nt, np[2], f0[2], bf_zero, cols, pad0, jp;
  int l_q, l_qbd, l_sb, l_pair;
  int l_grows;  // MoveScratch::grows where it is to be looked at, else -1
  size_t stride, f[2], s[2], w[2];
  int ldw[2];
  const double *gvec;
  double *gbase;      // determinant blocks in device memory, or null
  size_t gstride;
  double *scr;
};
inline RealArgs real_args(const DevSys &hs, double *scr) {
  RealArgs a{};
  const MoveScratch l = move_scratch(hs);
  const RealLayout r = real_layout(hs);
  a.N = hs.N;
  a.nt = hs.nt;
  for (int t = 0; t < 2; t++) {
    a.np[t] = hs.np[t];
    a.f0[t] = hs.ipfrst[t];
    a.f[t] = r.f[t];
    a.s[t] = r.s[t];
    a.w[t] = r.w[t];
    a.ldw[t] = r.ldw[t];
  }
  a.bf_zero = hs.bf_zero;
  a.pad0 = (hs.np[0] + 3) & ~3;
  a.cols = a.pad0 + (hs.nt > 1 ? (hs.np[1] + 3) & ~3 : 0);
  a.jp = r.jp;
  a.l_q = l.q;
  a.l_qbd = l.qbd;
  a.l_sb = l.sb;
  a.l_pair = l.pair;
  a.l_grows = -1;
  a.stride = l.stride;
  a.gvec = hs.gvec;
  a.gbase = hs.gmat ? hs.gmat_base : nullptr;
  a.gstride = (size_t)hs.gmat_stride;
  a.scr = scr;
  return a;
}
// The walker's real-orbital region: in its determinant block when it has one
// in device memory (the complex matrices of the other route are larger),
// else in its move scratch behind the per-particle sums.
__host__ __device__ inline double *real_base(const RealArgs &a, size_t w) {
  return a.gbase ? a.gbase + w * a.gstride : a.scr + w * a.stride + a.l_pair;
}

// Whether walker w has anything to evaluate (a reptile whose move has fewer bead
// growths than this one has not).
__device__ __forceinline__ bool real_on(const RealArgs &a, size_t w) {
  return a.l_grows < 0 || a.scr[w * a.stride + a.l_grows] != 0.0;
}

// Shared memory of the evaluation's end: the per-particle arrays of EvalSmem
// that the assembly uses.
__host__ __device__ inline size_t real_carve(const DevSys &s, char *base, EvalSmem *m) {
  size_t off = 0;
  auto take = [&](size_t doubles) -> double * {
    char *p = base ? base + off : nullptr;
    off += align16(sizeof(double) * doubles);
    return (double *)p;
  };
  const size_t N = s.N;
  EvalSmem t{};
  t.x = take(2 * N);
  t.g = take(2 * N);
  t.lap = take(N);
  t.ltf = take(N);
  t.vp = take(N);
  t.ph2 = take(N);
  t.gd = take(2 * N);
  t.lapd = take(N);
  t.ph2d = take(N);
  t.rhok = take(4 * (size_t)(s.nk > 0 ? s.nk : 1));
  t.red = take(kThreads);
  if (m) *m = t;
  return off;
}

// Between the pair passes and the evaluation's end, for nw walkers: orbitals,
// inverse and F of every (walker, spin), then the S sums, drift and
// Laplacian shares, all in the walkers' real regions. some: of the walkers marked
// in their scratch (MoveScratch::grows) alone.
cudaError_t launch_real_det(const DevSys &hs, const DevSys *ds, int nw, double *scr,
                            cudaStream_t st, bool some = false);

// The pair passes' sums of walker w into shared memory, the determinant sums
// zeroed (asynchronous 8-byte copies; the caller waits).
template <int NT>
__device__ __forceinline__ void load_real_sums(const DevSys &S, const EvalSmem &m,
                                               const double *o, const MoveScratch &L) {
  const int N = S.N, tid = threadIdx.x;
  for (int j = tid; j < 2 * N; j += NT) {
    cp_async8(m.x + j, o + L.x + j);
    cp_async8(m.g + j, o + L.g + j);
  }
  for (int j = tid; j < N; j += NT) {
    cp_async8(m.lap + j, o + L.lap + j);
    cp_async8(m.ltf + j, o + L.ltf + j);
    cp_async8(m.vp + j, o + L.vp + j);
    m.lapd[j] = 0.0;
    m.ph2[j] = 0.0;
    m.ph2d[j] = 0.0;
  }
}

// The end of an evaluation after launch_real_det, as eval_det: m holds x, g,
// lap, ltf, vp of the pair passes (their asynchronous copies may be in
// flight) and zeroed lapd, ph2, ph2d; o is the walker's scratch block, base its
// real region.
template <int NT>
__device__ inline int eval_det_real(const DevSys &S, const EvalSmem &m, double *hl, double *props,
                                    double *sign, long long &tph, const double *o,
                                    const MoveScratch &L, const RealArgs &R,
                                    const double *base) {
  const int tid = threadIdx.x, N = S.N, nt = S.nt;
  for (int e = tid; e < 4 * S.nk; e += NT) cp_async8(m.rhok + e, o + L.rhok + e);
  int status = ST_OK;
  double logdet_sum = 0.0, l0 = 0.0, l1 = 0.0;
  if (S.bf_zero) {
    // J = 1: the drift of an electron is its own f, and of the sums over F
    // and D2 the products F_a(j,k) F_a(k,j), j != k, are left
    double s[2] = {0.0, 0.0};
#pragma unroll
    for (int t = 0; t < 2; t++) {
      if (t >= nt) continue;
      const int n = S.np[t];
      const double *FX = base + R.f[t], *FY = FX + n * n;
      for (int j = tid; j < 2 * n; j += NT)
        m.gd[2 * S.ipfrst[t] + j] = -(j & 1 ? FY : FX)[(j >> 1) * (n + 1)];
      for (int e = tid; e < n * n; e += NT) {
        const int j = e / n, k = e - j * n;
        if (k > j)
          s[t] -= 2.0 * (FX[k + j * n] * FX[j + k * n] + FY[k + j * n] * FY[j + k * n]);
      }
    }
    block_sum_n<2, NT>(s, m.red);
    l0 = s[0];
    l1 = s[1];
  } else {
    // the determinants' drift: every spin's share
    for (int j = tid; j < 2 * N; j += NT) {
      double g = base[R.s[0] + j];
      if (nt > 1) g += base[R.s[1] + j];
      m.gd[j] = g;
    }
  }
#pragma unroll
  for (int t = 0; t < 2; t++) {
    if (t >= nt) continue;
    const double *f = base + R.f[t] + 2 * S.np[t] * S.np[t], *s = base + R.s[t] + 2 * N;
    logdet_sum += f[0];
    if (f[1] != 0.0) status |= ST_SINGULAR;
    if (!S.bf_zero) {
      l0 += s[0];
      l1 += s[1];
    }
  }
  cp_async_wait_all();
  __syncthreads();
  // the assembly sums lapd per type
  if (tid == 0) m.lapd[0] = l0;
  if (tid == 1 && nt > 1) m.lapd[S.ipfrst[1]] = l1;
  double ltf_j[1] = {0.0};
  for (int j = tid; j < N; j += NT) ltf_j[0] += m.ltf[j];
  block_sum_n<1, NT>(ltf_j, m.red);  // its barriers cover lapd too
  phase_mark(S, PH_ORBITALS, tph);
  return eval_assemble<NT>(S, m, ltf_j[0], logdet_sum, status, hl, props, sign, tph);
}

}  // namespace q2d
