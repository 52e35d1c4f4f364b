// Kernel (c), stage 2: eigenvalues and oscillator strengths of the real symmetric
// tridiagonal T = Q^H H Q produced by tridiag.cu.
//
// Reference: ZHEEV('V','U') + dielbsev/dielbsep (subprograms/bse_solver-tool-diel.f90:485-602,
// subroutines/bse_subs.f90:278-378).  The oscillator strength of exciton n is
//   f_n = |sum_j A_jn h_j|^2 = |z_n^T g|^2,  g = Q^T h,  A = Q Z,
// so after the reduction only the tridiagonal eigenvectors z_n are needed, and only inside
// the dot products with the five g vectors.
//   * eigenvalues: one coarse round of Sturm counts at 32769 points of the Gershgorin interval
//     gives every eigenvalue index its starting cell; then Sturm-count multisection, L lanes
//     per eigenvalue index (L = 1: bisection), to full precision;
//   * eigenvectors: the recurrence of T - lambda from the top and from the bottom, joined at the
//     row where the product of the two is largest (k_twist), the dot products with g taken in the
//     last pass over the vector; one row's residual shows whether the vector is good;
//   * eigenvalues closer than 1e-7 * ||T|| form a cluster: its vectors are orthonormalised in
//     order (k_cluster), so degenerate excitons get orthogonal vectors;
//   * what neither makes well (a residual that is too large, a cluster of nearly parallel
//     vectors) is made by inverse iteration with a partial-pivoting tridiagonal LU, three steps
//     from a deterministic pseudo-random start vector (k_inviter).
// Selected exciton eigenvectors (BSE_WF) are back-transformed A_n = Q z_n panel by panel
// with the compact-WY form I - V T V^H of each panel's reflectors.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

#include "common.cuh"

namespace {

constexpr int NG = 10;   // largest number of reduced h vectors (5, or 10 with temperature)

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N_>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N_) : "memory"); }

// Records of T scaled by sc = 2^-j so that ||sc T|| <= 1, padded to a multiple of TD_TILE rows by rows that
// change no count: cnt[k] = (d_k, -e_{k-1}^2) for the counts, vec[2k], vec[2k+1] = (d_k, e_k), (-1/e_k, -1/e_{k-1}) for
// the vectors.  |e| is held above TD_EMIN, far below the rounding of T itself, so that the recurrences never
// run into zero: eight steps shrink them by less than 2^-1000.
constexpr int TD_TILE = 128;
constexpr double TD_EMIN = 0x1p-80;
__global__ void k_td_records(const double* __restrict__ d, const double* __restrict__ e, int n, int npad, double sc,
                             double2* __restrict__ cnt, double2* __restrict__ vec) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= npad) return;
  auto off = [&](int i) {
    const double x = e[i] * sc;
    return fabs(x) < TD_EMIN ? copysign(TD_EMIN, x) : x;
  };
  const double ep = (k >= 1 && k < n) ? off(k - 1) : 0.0, ek = (k < n - 1) ? off(k) : 1.0;
  const double dk = (k < n) ? d[k] * sc : 4.0;
  cnt[k] = make_double2(dk, -ep * ep);
  vec[2 * k] = make_double2(dk, ek);
  vec[2 * k + 1] = make_double2(-1.0 / ek, (k >= 1 && k < n) ? -1.0 / ep : 0.0);
}

// Number of eigenvalues of the scaled T below x, one point per thread: the sign changes of the leading
// minors p_{k+1} = (d_k - x) p_k - e_{k-1}^2 p_{k-1} (the counts of the pivots p_{k+1} / p_k, and as backward
// stable: each step is exact for d_k - x and e_{k-1}^2 changed by a few roundings).  Without a division the chain
// is one FMA a step (N = 576 0.41 -> 0.07 ms, 3600 3.6 -> 0.71 ms); scaled every eight steps.  The records stream
// through a four-stage ring shared by the block of TD_TILE threads, all of which must call this.
constexpr int TD_ST = 4;
__device__ __forceinline__ int block_sturm(const double2* __restrict__ rec, int n, double x,
                                           double2 (*ring)[TD_TILE]) {
  const int tid = threadIdx.x, ntile = (n + TD_TILE - 1) / TD_TILE;
  for (int t = 0; t < TD_ST - 1; ++t) {
    if (t < ntile) cp_async16(&ring[t][tid], rec + (size_t)t * TD_TILE + tid);
    cp_async_commit();
  }
  double p = 1.0, pp = 0.0;
  int cnt = 0;
  for (int t = 0; t < ntile; ++t) {
    cp_async_wait<TD_ST - 2>();
    __syncthreads();
    const int tn = t + TD_ST - 1;
    if (tn < ntile) cp_async16(&ring[tn % TD_ST][tid], rec + (size_t)tn * TD_TILE + tid);
    cp_async_commit();
    const double2* c = ring[t % TD_ST];
    double2 a[8], b[8];   // eight records at work, the next eight on their way
    auto load = [&](double2* v, int g) {
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = c[g + q];
    };
    auto steps = [&](const double2* v) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const double pn = fma(v[q].x - x, p, v[q].y * pp);
        cnt += (unsigned)(__double2hiint(pn) ^ __double2hiint(p)) >> 31;
        pp = p;
        p = pn;
      }
      pow2_rescale(p, pp);
    };
    load(a, 0);
    if (n - t * TD_TILE >= TD_TILE) {
#pragma unroll 1
      for (int g = 0; g < TD_TILE; g += 16) {
        load(b, g + 8);
        steps(a);
        load(a, (g + 16) & (TD_TILE - 1));
        steps(b);
      }
    } else {   // the last tile: the padding counts nothing (one loop of variable length: solve of N = 3600 1.44 -> 1.62 ms)
#pragma unroll 1
      for (int g = 0; g < n - t * TD_TILE; g += 8) {
        load(b, (g + 8) & (TD_TILE - 1));
        steps(a);
#pragma unroll
        for (int q = 0; q < 8; ++q) a[q] = b[q];
      }
    }
  }
  __syncthreads();
  return cnt;
}

// Coarse round: Sturm counts at the P + 1 points x_j = lo + (hi - lo) j / P of the Gershgorin
// interval (count 0 at lo and n at hi by construction), one thread per point.
constexpr int BIS_P = 32768;
__global__ void __launch_bounds__(TD_TILE) k_bisect_grid(const double2* __restrict__ rec, int n, double lo, double hi,
                                                         double sc, double* __restrict__ xg,
                                                         int* __restrict__ cg) {
  __shared__ __align__(16) double2 ring[TD_ST][TD_TILE];
  const int j = min(blockIdx.x * TD_TILE + (int)threadIdx.x, BIS_P);
  const double x = (j == BIS_P) ? hi : lo + (hi - lo) * ((double)j / (double)BIS_P);
  const int c = block_sturm(rec, n, x * sc, ring);
  xg[j] = x;
  cg[j] = (j == 0) ? 0 : (j == BIS_P ? n : c);
}

// Multisection: L consecutive lanes (L a power of two, L <= 32) share eigenvalue m and, per
// round, take Sturm counts at L interior points of its interval [a, b]; the new interval runs
// from the highest point with count <= m to the next point (or b), so count(a) <= m < count(b)
// holds whatever the counts at the other points.  A round divides the interval by L + 1 (by 2,
// at the midpoint, for L = 1: plain bisection), so the chain of dependent Sturm passes per
// eigenvalue is log2(L + 1) times shorter, for L times more total passes; the host picks L.
// Stopping rule as in bisection: width <= 2 eps max(|a|, |b|) + pivmin, or no double between.
__global__ void __launch_bounds__(TD_TILE) k_bisect(const double2* __restrict__ rec, long long n,
                                                    const double* __restrict__ xg, const int* __restrict__ cg,
                                                    double pivmin, double sc, int L, double* lam) {
  __shared__ __align__(16) double2 ring[TD_ST][TD_TILE];
  const long long gt = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long m = gt / L;
  const int lane = threadIdx.x & 31, sl = lane & (L - 1), base = lane - sl;
  const bool active = m < n;
  // start from the coarse cell [x_j, x_{j+1}] with count(x_j) <= m < count(x_{j+1}) (binary
  // search keeping that invariant; cg[0] = 0 <= m < n = cg[P])
  double a = xg[0], b = xg[BIS_P];
  if (active) {
    int jl = 0, jh = BIS_P;
    while (jh - jl > 1) {
      const int jm = (jl + jh) >> 1;
      if (cg[jm] <= m) jl = jm;
      else jh = jm;
    }
    a = xg[jl];
    b = xg[jh];
  }
  for (int it = 0; it < 256; ++it) {
    const double mid = 0.5 * (a + b);
    const bool done = !active || !(mid > a && mid < b) || (b - a <= 2.0 * DBL_EPSILON * fmax(fabs(a), fabs(b)) + pivmin);
    if (__syncthreads_and(done)) break;
    const double x = (L == 1) ? mid : a + (b - a) * ((double)(sl + 1) / (double)(L + 1));
    const bool le = block_sturm(rec, (int)n, x * sc, ring) <= m && !done;
    const unsigned gb = (__ballot_sync(0xffffffffu, le) >> base) & (L == 32 ? 0xffffffffu : ((1u << L) - 1u));
    const int jhi = gb ? 31 - __clz(gb) : -1;   // highest point with count <= m
    const double xa = __shfl_sync(0xffffffffu, x, base + max(jhi, 0));
    const double xb = __shfl_sync(0xffffffffu, x, base + min(jhi + 1, L - 1));
    if (!done) {
      if (jhi >= 0) a = xa;
      if (jhi + 1 < L) b = xb;
    }
  }
  if (active && sl == 0) lam[m] = 0.5 * (a + b);
}

// Lanes per eigenvalue for k_bisect: after the coarse round (15 bits) rounds ~ 38 / log2(L+1), each of n
// steps of about 21 cycles with one block on an SM and of 15 per block with more
// (N = 576 with L = 32, 3600 with L = 4, 14400 with L = 1 and the coarse round).
int bisect_lanes(long long n, int nsm) {
  int best = 1;
  double bt = 1e300;
  for (int L = 1; L <= 32; L *= 2) {
    const double rounds = std::ceil(38.0 / std::log2((double)L + 1.0));
    const double blocks = std::ceil(std::ceil((double)n * L / TD_TILE) / std::max(nsm, 1));
    const double t = rounds * std::max(21.0, 15.0 * blocks);
    if (t < bt) {
      bt = t;
      best = L;
    }
  }
  return best;
}

__device__ __forceinline__ double start_value(long long m, long long k) {
  unsigned long long z = (unsigned long long)m * 0x9E3779B97F4A7C15ull + (unsigned long long)k * 0xD1B54A32D192ED03ull + 0x632BE59BD9B4E019ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return ((double)(z >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0;
}

struct InvArgs {
  const double* d;
  const double* e;
  long long n;
  const double* lam;
  const int* csize;     // cluster size at a leader index that is to be done, 0 for the others
  long long m0;         // first eigenvalue index of the chunk
  long long m1;         // one past the last eigenvalue index of the chunk
  int M;                // slots in the chunk
  double* ws;           // 4 * n * M
  double pert;          // eps * ||T||: pivot floor
  const double2* g;     // [ng][n]: h (x, y, z, sp, sm) [, h * f with temperature]
  int ng;
  double* act;          // [8][n]
  int dtfull, cpol;
  double* zsel;         // selected vectors (column-major n x nsel) or null
  long long zs0, zs1;
};

// act(a, b) = Re[(z^T g_a) conj(z^T g'_b)], g' = g (dielbsev/dielbsep) or the f-weighted
// vectors with temperature (dielbseptemp)
__device__ __forceinline__ void write_act(const double2* sg, int ng, int dtfull, int cpol, double* act, long long n,
                                          long long mm) {
  auto re = [&](int p, int q) {
    const double2 u = sg[p], v = (ng == 10) ? sg[5 + q] : sg[q];
    return u.x * v.x + u.y * v.y;
  };
  act[0 * n + mm] = re(0, 0);
  act[1 * n + mm] = re(1, 1);
  act[2 * n + mm] = re(2, 2);
  act[3 * n + mm] = dtfull ? re(0, 1) : 0.0;
  act[4 * n + mm] = dtfull ? re(0, 2) : 0.0;
  act[5 * n + mm] = dtfull ? re(1, 2) : 0.0;
  act[6 * n + mm] = cpol ? re(3, 3) : 0.0;
  act[7 * n + mm] = cpol ? re(4, 4) : 0.0;
}

struct TwistArgs {
  const double2* rec;   // vector records of k_td_records
  int n, npad;
  double sc;
  const double* lam;
  const int* csize;     // cluster size at a leader index, 0 for non-leaders
  int* todo;            // csize of the leaders that k_inviter has to do
  int m0, m1, M;        // eigenvalue indices of the chunk; slots (a multiple of 32)
  double* t;            // [npad][M]: the recurrence from the top; for members of clusters then the vector
  int* te;              // [npad / 8][M]: its exponents
  const double2* g;     // [NG][n]
  double* act;
  int dtfull, cpol;
  double rtol;          // largest residual of the joined row, ||sc T|| <= 1
  bool keep;            // vectors are wanted, not only the sums: k_cluster normalises all of them in t
};

// Eigenvector m of T without a factorisation, one lane each.  From the top z_{k+1} = -((d_k - lam) z_k + e_{k-1}
// z_{k-1}) / e_k, and from the bottom the same upwards, satisfy every row of T - lam to rounding; joined at the
// row r where |top_r bottom_r| is largest (there the diagonal of (T - lam)^-1 is largest, and so the residual of
// the one row left smallest) they are the eigenvector, and that row's residual over the norm tells how good.
// Three passes: top (stored, 8 bytes a step), bottom (finds r), bottom again with the sums over the joined vector.
// Every eight steps the pair is scaled by a power of two.  A chain of an FMA and a multiplication a step, no
// division, and one pass written and one and a half read, against three factorisations with their divisions and
// 33 passes in inverse iteration.  Bound by that chain where the vectors are few: N = 576 0.82 -> 0.07 ms, 3600
// 6.4 -> 0.42 ms, 14400 (one launch; a cluster of two in it made 51 ms) 1.8 ms.
constexpr int TW = 32;   // rows of a tile of the ring
constexpr int TW_ST = 3;
template <int NGT>
struct __align__(16) TwTile {
  double2 rec[2 * TW];
  double t[TW][32];
  int te[TW / 8][32];
  double2 g[NGT][TW];
};
__device__ __forceinline__ double tw_step(double a, double z, double e, double zp, double nie) {
  return __dmul_rn(__fma_rn(a, z, __dmul_rn(e, zp)), nie);
}

template <int NGT>
__global__ void __launch_bounds__(32) k_twist(TwistArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  TwTile<NGT>* ring = reinterpret_cast<TwTile<NGT>*>(smem);
  const int lane = threadIdx.x, j0 = blockIdx.x * 32, jj = j0 + lane, M = a.M, n = a.n;
  const int m = min(a.m0 + jj, a.m1 - 1);
  const bool live = a.m0 + jj < a.m1;
  const double lam = a.lam[m] * a.sc;
  const int nt = (n + TW - 1) / TW;
  double* __restrict__ T = a.t + jj;
  int* __restrict__ TE = a.te + jj;
  // what: 1 = records, 2 = + top recurrence, 4 = + g
  auto issue = [&](int tile, int st, int what) {
    if (tile >= 0 && tile < nt) {
      TwTile<NGT>& s = ring[st];
      const int k0 = tile * TW;
      cp_async16(&s.rec[lane], a.rec + 2 * (size_t)k0 + lane);
      cp_async16(&s.rec[lane + 32], a.rec + 2 * (size_t)k0 + lane + 32);
      if (what & 2) {
        const int r0 = lane >> 4, c0 = (lane & 15) * 2;
        for (int q = 0; q < TW; q += 2) cp_async16(&s.t[q + r0][c0], a.t + (size_t)(k0 + q + r0) * M + j0 + c0);
        cp_async16(&s.te[lane >> 3][(lane & 7) * 4], a.te + (size_t)(k0 / 8 + (lane >> 3)) * M + j0 + (lane & 7) * 4);
      }
      if (what & 4)
        for (int al = 0; al < NGT; ++al) cp_async16(&s.g[al][lane], a.g + (size_t)al * n + min(k0 + lane, n - 1));
    }
    cp_async_commit();
  };
  // ---- from the top
  {
    double z = 1.0, zp = 0.0, ep = 0.0;
    int E = 0;
    for (int t = 0; t < TW_ST - 1; ++t) issue(t, t, 1);
    for (int t = 0; t < nt; ++t) {
      cp_async_wait<TW_ST - 2>();
      __syncwarp();
      issue(t + TW_ST - 1, (t + TW_ST - 1) % TW_ST, 1);
      const TwTile<NGT>& s = ring[t % TW_ST];
      for (int b = 0; b < TW; b += 8) {
        E += pow2_rescale(z, zp);
        TE[(size_t)((t * TW + b) >> 3) * M] = E;
        double2 de[8];
        double nie[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          de[q] = s.rec[2 * (b + q)];
          nie[q] = s.rec[2 * (b + q) + 1].x;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          T[(size_t)(t * TW + b + q) * M] = z;
          const double zn = tw_step(__dsub_rn(de[q].x, lam), z, ep, zp, nie[q]);
          zp = z;
          z = zn;
          ep = de[q].y;
        }
      }
    }
  }
  __threadfence_block();
  cp_async_wait<0>();
  __syncwarp();
  // ---- from the bottom: r, and the two values there
  const double z0 = (n % 8) ? 0.0 : 1.0;   // blocks of eight rows: the last may begin behind row n - 1
  int r = n - 1, bE = 0, bTE = 0, bBE = 0;
  double bM = 0.0, bT = 1.0, bB = 1.0;
  bool have = false;
  {
    double z = z0, zp = 0.0;
    int E = 0;
    for (int t = 0; t < TW_ST - 1; ++t) issue(nt - 1 - t, t, 3);
    for (int t = 0; t < nt; ++t) {
      cp_async_wait<TW_ST - 2>();
      __syncwarp();
      issue(nt - 1 - (t + TW_ST - 1), (t + TW_ST - 1) % TW_ST, 3);
      const TwTile<NGT>& s = ring[t % TW_ST];
      const int k0 = (nt - 1 - t) * TW;
      for (int b = TW - 8; b >= 0; b -= 8) {
        if (k0 + b >= n) continue;
        E += pow2_rescale(z, zp);
        double vb = 0.0, tb = 1.0, bb = 1.0, tv[8], nie[8];
        double2 de[8];
        int kb = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          de[q] = s.rec[2 * (b + q)];
          nie[q] = s.rec[2 * (b + q) + 1].y;
          tv[q] = s.t[b + q][lane];
        }
#pragma unroll
        for (int q = 7; q >= 0; --q) {
          const double v = fabs(tv[q] * z);
          if (v > vb) {
            vb = v;
            kb = q;
            tb = tv[q];
            bb = z;
          }
          const double zn = tw_step(__dsub_rn(de[q].x, lam), z, de[q].y, zp, nie[q]);
          zp = z;
          z = zn;
          if (k0 + b + q == n) z = 1.0;   // rows behind the last: zeros up to it
        }
        const int tE = s.te[b >> 3][lane], h = __double2hiint(vb), ve = tE + E + (h >> 20) - 1023;
        const double vm = __hiloint2double((h & 0x000fffff) | 0x3ff00000, __double2loint(vb));
        if (vb > 0.0 && (!have || ve > bE || (ve == bE && vm > bM))) {
          have = true;
          bE = ve;
          bM = vm;
          r = k0 + b + kb;
          bT = tb;
          bTE = tE;
          bB = bb;
          bBE = E;
        }
      }
    }
  }
  cp_async_wait<0>();
  __syncwarp();
  // ---- from the bottom again, joined with the top at r and scaled to z_r = 1
  const bool member = a.keep || a.csize[m] != 1, members = __any_sync(0xffffffffu, member);
  const double st = 1.0 / bT, sb = 1.0 / bB;
  const int rmax = __reduce_max_sync(0xffffffffu, r);
  double2 sg[NGT];
#pragma unroll
  for (int al = 0; al < NGT; ++al) sg[al] = make_double2(0, 0);
  double nrm = 0.0, zup = 0.0, zdn = 0.0;   // z_{r-1}, z_{r+1}
  {
    double z = z0, zp = 0.0;
    int E = 0;
    auto what = [&](int tile) { return 5 | (tile * TW <= rmax ? 2 : 0); };
    for (int t = 0; t < TW_ST - 1; ++t) issue(nt - 1 - t, t, what(nt - 1 - t));
    for (int t = 0; t < nt; ++t) {
      cp_async_wait<TW_ST - 2>();
      __syncwarp();
      const int tn = nt - 1 - (t + TW_ST - 1);
      issue(tn, (t + TW_ST - 1) % TW_ST, what(tn));
      const TwTile<NGT>& s = ring[t % TW_ST];
      const int k0 = (nt - 1 - t) * TW;
      for (int b = TW - 8; b >= 0; b -= 8) {
        if (k0 + b >= n) continue;
        E += pow2_rescale(z, zp);
        const double fb = sb * pow2_clamped(E - bBE);
        const double ft = st * pow2_clamped(s.te[b >> 3][lane] - bTE);
        double x[8], nie[8];
        double2 de[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          de[q] = s.rec[2 * (b + q)];
          nie[q] = s.rec[2 * (b + q) + 1].y;
          x[q] = s.t[b + q][lane] * ft;   // taken up to row r only: a tile without the top is above it
        }
#pragma unroll
        for (int q = 7; q >= 0; --q) {
          const int k = k0 + b + q;
          if (k > r) x[q] = z * fb;
          if (k == r + 1) zdn = x[q];
          if (k == r - 1) zup = x[q];
          const double zn = tw_step(__dsub_rn(de[q].x, lam), z, de[q].y, zp, nie[q]);
          zp = z;
          z = zn;
          if (k == n) z = 1.0;
        }
#pragma unroll
        for (int q = 7; q >= 0; --q) {
          nrm = fma(x[q], x[q], nrm);
#pragma unroll
          for (int al = 0; al < NGT; ++al) {
            const double2 gk = s.g[al][b + q];
            sg[al].x = fma(x[q], gk.x, sg[al].x);
            sg[al].y = fma(x[q], gk.y, sg[al].y);
          }
        }
        if (members && member && live) {
#pragma unroll
          for (int q = 0; q < 8; ++q) T[(size_t)(k0 + b + q) * M] = x[q];
        }
      }
    }
  }
  if (!live) return;
  const double2 de = a.rec[2 * (size_t)r];
  const double res = fma(r > 0 ? a.rec[2 * (size_t)r - 2].y : 0.0, zup, fma(de.x - lam, 1.0, (r < n - 1 ? de.y : 0.0) * zdn));
  if (!have || !(fabs(res) <= a.rtol * sqrt(nrm)) || !(nrm < 1e300)) {
    int l = m;   // inverse iteration makes this vector, or the cluster that it is in
    while (l > 0 && a.csize[l] == 0) --l;
    a.todo[l] = a.csize[l];
    return;
  }
  const double c = 1.0 / sqrt(nrm);
#pragma unroll
  for (int al = 0; al < NGT; ++al) sg[al] = cscale(sg[al], c);
  write_act(sg, NGT, a.dtfull, a.cpol, a.act, n, m);
}

// The vectors of a cluster, one block each: modified Gram-Schmidt in order against the earlier members, then
// the sums again.  Where less than a third of a vector is left the members were nearly parallel (eigenvalues
// equal to rounding), and inverse iteration makes the cluster.  With keep also a vector by itself: normalised.
constexpr int CL_T = 256;
__device__ __forceinline__ double block_sum(double x, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int q = 0; q < CL_T / 32; ++q) s += red[q];
  return s;
}
template <int NGT>
__global__ void __launch_bounds__(CL_T) k_cluster(TwistArgs a) {
  __shared__ double red[CL_T / 32];
  const int m = a.m0 + blockIdx.x, cs = a.csize[m], n = a.n, tid = threadIdx.x;
  if (cs < (a.keep ? 1 : 2) || a.todo[m] != 0) return;
  double* __restrict__ X = a.t + blockIdx.x;
  const size_t M = (size_t)a.M;
  for (int s = 0; s < cs; ++s) {
    double before = 0.0, left = 0.0;
    for (int k = tid; k < n; k += CL_T) before = fma(X[k * M + s], X[k * M + s], before);
    before = block_sum(before, red);
    for (int t = 0; t < s; ++t) {
      double dot = 0.0;
      for (int k = tid; k < n; k += CL_T) dot = fma(X[k * M + s], X[k * M + t], dot);
      dot = block_sum(dot, red);
      for (int k = tid; k < n; k += CL_T) X[k * M + s] = fma(-dot, X[k * M + t], X[k * M + s]);
    }
    for (int k = tid; k < n; k += CL_T) left = fma(X[k * M + s], X[k * M + s], left);
    left = block_sum(left, red);
    if (!(left >= 0.1 * before)) {
      if (tid == 0) a.todo[m] = cs;
      return;
    }
    const double c = 1.0 / sqrt(left);
    double2 sg[NGT];
#pragma unroll
    for (int al = 0; al < NGT; ++al) sg[al] = make_double2(0, 0);
    for (int k = tid; k < n; k += CL_T) {
      const double x = X[k * M + s] * c;
      X[k * M + s] = x;
#pragma unroll
      for (int al = 0; al < NGT; ++al) {
        const double2 gk = a.g[(size_t)al * n + k];
        sg[al].x = fma(x, gk.x, sg[al].x);
        sg[al].y = fma(x, gk.y, sg[al].y);
      }
    }
#pragma unroll
    for (int al = 0; al < NGT; ++al) {
      sg[al].x = block_sum(sg[al].x, red);
      sg[al].y = block_sum(sg[al].y, red);
    }
    if (tid == 0) write_act(sg, NGT, a.dtfull, a.cpol, a.act, n, m + s);
  }
}

// vectors zs0 .. zs1 of the chunk as columns of zsel, except those that k_inviter has made
__global__ void k_take_vectors(TwistArgs a, int zs0, double* zsel) {
  const int c = blockIdx.y, m = zs0 + c, k = blockIdx.x * blockDim.x + threadIdx.x;
  int l = m;
  while (l > 0 && a.csize[l] == 0) --l;
  if (k < a.n && a.todo[l] == 0) zsel[(size_t)c * a.n + k] = a.t[(size_t)k * a.M + (m - a.m0)];
}

template <int NGT>
static int launch_twist(wtbg_ctx* ctx, const TwistArgs& a, bool clusters) {
  const int cnt = a.m1 - a.m0, smem = TW_ST * (int)sizeof(TwTile<NGT>);
  CK(cudaFuncSetAttribute(k_twist<NGT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  k_twist<NGT><<<(cnt + 31) / 32, 32, smem, ctx->stream>>>(a); WTBG_COUNT(ctx, 1);
  CKL("k_twist");
  if (clusters || a.keep) {
    k_cluster<NGT><<<cnt, CL_T, 0, ctx->stream>>>(a); WTBG_COUNT(ctx, 1);
    CKL("k_cluster");
  }
  return 0;
}

// Below this the vectors are all made by inverse iteration: its chain is then no longer than the launches around
// k_twist (vectors of N = 2 0.057 ms against 0.073, 8 0.117 / 0.126, 12 0.172 / 0.176, 16 0.245 both).
constexpr long long TWIST_FROM = 16;

constexpr int SB = 8;   // inverse-iteration steps whose loads are issued together

__global__ void __launch_bounds__(64) k_inviter(InvArgs a) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= a.M) return;
  const long long m = a.m0 + j;
  if (m >= a.m1 || m >= a.n) return;
  const int cs = a.csize[m];
  if (cs == 0) return;
  const long long n = a.n;
  const int M = a.M;
  // Four disjoint slices of the workspace, laid out [k][slot]: each step of the elimination and
  // of the substitution is one link of a chain through a division, while its workspace loads
  // (one DRAM round trip each) do not depend on the chain; so the loads of SB steps are issued
  // together before the SB dependent steps run (same arithmetic, one round trip per SB steps).
  double* __restrict__ X = a.ws;
  double* __restrict__ U1 = a.ws + n * M;
  double* __restrict__ U2 = a.ws + 2 * n * M;
  double* __restrict__ U3 = a.ws + 3 * n * M;
  const double* __restrict__ dd_ = a.d;
  const double* __restrict__ ee_ = a.e;
  const double pert = a.pert;
  for (int s = 0; s < cs; ++s) {
    const long long mm = m + s;
    const int jj = j + s;
    const double lam = a.lam[mm];
    double sc = 1.0;
    for (long long k = 0; k < n; ++k) X[k * M + jj] = start_value(mm, k);
    for (int it = 0; it < 3; ++it) {
      // factor T - lam I with partial pivoting, eliminating the right-hand side on the fly
      double diag = dd_[0] - lam;
      double sup = (n > 1) ? ee_[0] : 0.0;
      double cur = X[jj] * sc;
      for (long long k0 = 0; k0 < n - 1; k0 += SB) {
        // the block's operands first (independent of the chain), then its SB dependent steps
        double xs[SB], es[SB + 1], ds[SB];
#pragma unroll
        for (int q = 0; q < SB; ++q) {
          const long long k = k0 + q;
          if (k < n - 1) {
            xs[q] = X[(k + 1) * M + jj];
            es[q] = ee_[k];
            ds[q] = dd_[k + 1];
          }
        }
        es[SB] = (k0 + SB < n - 1) ? ee_[k0 + SB] : 0.0;
#pragma unroll
        for (int q = 0; q < SB; ++q) {
          const long long k = k0 + q;
          if (k >= n - 1) break;
          const double sub = es[q];
          const double nd = ds[q] - lam;
          const double nsup = (k + 1 < n - 1) ? es[q + 1] : 0.0;
          const double nxt = xs[q] * sc;
          if (fabs(diag) >= fabs(sub)) {
            if (fabs(diag) < pert) diag = copysign(pert, diag);
            const double mult = sub / diag;
            U1[k * M + jj] = diag;
            U2[k * M + jj] = sup;
            U3[k * M + jj] = 0.0;
            X[k * M + jj] = cur;
            cur = nxt - mult * cur;
            diag = nd - mult * sup;
            sup = nsup;
          } else {
            const double mult = diag / sub;
            U1[k * M + jj] = sub;
            U2[k * M + jj] = nd;
            U3[k * M + jj] = nsup;
            X[k * M + jj] = nxt;
            cur = cur - mult * nxt;
            diag = sup - mult * nd;
            sup = -mult * nsup;
          }
        }
      }
      if (fabs(diag) < pert) diag = copysign(pert, diag);
      // back substitution (U1 of the last row kept in a register)
      double x2 = 0.0, x1 = cur / diag;
      X[(n - 1) * M + jj] = x1;
      double nrm = x1 * x1;
      for (long long kb = n - 2; kb >= 0; kb -= SB) {
        double xs[SB], u1[SB], u2[SB], u3[SB];
#pragma unroll
        for (int q = 0; q < SB; ++q) {
          const long long k = kb - q;
          if (k >= 0) {
            xs[q] = X[k * M + jj];
            u1[q] = U1[k * M + jj];
            u2[q] = U2[k * M + jj];
            u3[q] = U3[k * M + jj];
          }
        }
#pragma unroll
        for (int q = 0; q < SB; ++q) {
          const long long k = kb - q;
          if (k < 0) break;
          const double xk = (xs[q] - u2[q] * x1 - u3[q] * x2) / u1[q];
          X[k * M + jj] = xk;
          nrm += xk * xk;
          x2 = x1;
          x1 = xk;
        }
      }
      sc = 1.0 / sqrt(nrm);
      // orthogonalise against the earlier members of the cluster (normalised, in slots j..jj-1)
      if (s > 0) {
        for (int t = 0; t < s; ++t) {
          double dot = 0.0;
          for (long long k = 0; k < n; ++k) dot += X[k * M + jj] * X[k * M + j + t];
          for (long long k = 0; k < n; ++k) X[k * M + jj] -= dot * X[k * M + j + t];
        }
        double n2 = 0.0;
        for (long long k = 0; k < n; ++k) n2 += X[k * M + jj] * X[k * M + jj];
        sc = 1.0 / sqrt(n2);
      }
    }
    // final pass: normalise and accumulate the oscillator dot products
    double2 sg[NG];
#pragma unroll
    for (int al = 0; al < NG; ++al) sg[al] = make_double2(0, 0);
    const bool keep = (a.zsel != nullptr && mm >= a.zs0 && mm <= a.zs1);
    const int ng = a.ng;
    for (long long k0 = 0; k0 < n; k0 += SB) {
      double xs[SB];
#pragma unroll
      for (int q = 0; q < SB; ++q)
        if (k0 + q < n) xs[q] = X[(k0 + q) * M + jj];
#pragma unroll
      for (int q = 0; q < SB; ++q) {
        const long long k = k0 + q;
        if (k >= n) break;
        const double x = xs[q] * sc;
        X[k * M + jj] = x;
#pragma unroll
        for (int al = 0; al < NG; ++al) {
          if (al < ng) {
            const double2 gk = a.g[al * n + k];
            sg[al].x += x * gk.x;
            sg[al].y += x * gk.y;
          }
        }
        if (keep) a.zsel[(mm - a.zs0) * n + k] = x;
      }
    }
    write_act(sg, ng, a.dtfull, a.cpol, a.act, n, mm);
  }
}

// ---- back-transform of selected vectors: X <- Q X, Q = H_0 H_1 ... H_{n-2}
constexpr int PB = WTBG_PANEL;
constexpr int BT_RB = 256;

// partials of G = V^H V (PB x PB) and P = V^H X (PB x nv) over row blocks
__global__ void __launch_bounds__(BT_RB) k_bt_gram(const double2* A, long long n, int j0, int jb, const double2* X, int nvec,
                                                  double2* part) {
  extern __shared__ double2 sh[];
  const int tid = threadIdx.x;
  const int ncols = jb + nvec;
  const long long r = (long long)j0 + 1 + (long long)blockIdx.x * BT_RB + tid;
  // load this row of V (jb) and X (nvec)
  double2 vrow[PB];
#pragma unroll
  for (int q = 0; q < PB; ++q) {
    double2 v = make_double2(0, 0);
    if (q < jb && r < n && r >= (long long)j0 + q + 1) v = A[r + (long long)(j0 + q) * n];
    vrow[q] = v;
  }
  // each thread accumulates its row's outer products into shared memory via a block reduction
  double2* acc = sh;  // [jb][ncols]
  for (int it = tid; it < jb * ncols; it += BT_RB) acc[it] = make_double2(0, 0);
  __syncthreads();
  for (int qi = 0; qi < jb; ++qi) {
    for (int cj = 0; cj < ncols; ++cj) {
      double2 rhs = make_double2(0, 0);
      if (r < n) {
        if (cj < jb) rhs = vrow[cj];
        else rhs = X[(long long)(cj - jb) * n + r];
      }
      double2 t = cmulc(vrow[qi], rhs);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
        t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
      }
      if ((tid & 31) == 0) {
        atomicAdd(&acc[qi * ncols + cj].x, t.x);
        atomicAdd(&acc[qi * ncols + cj].y, t.y);
      }
    }
  }
  __syncthreads();
  for (int it = tid; it < jb * ncols; it += BT_RB) part[(long long)blockIdx.x * PB * (PB + 64) + it] = acc[it];
}

// reduce partials, build T (zlarft forward/columnwise), Y = T P
__global__ void k_bt_tmat(const double2* part, int nparts, int jb, int nvec, const double2* tau, int j0, double2* Y) {
  __shared__ double2 G[PB][PB], Tm[PB][PB], P[PB][32];
  const int tid = threadIdx.x;
  const int ncols = jb + nvec;
  for (int it = tid; it < jb * ncols; it += blockDim.x) {
    double2 s = make_double2(0, 0);
    for (int k = 0; k < nparts; ++k) s = cadd(s, part[(long long)k * PB * (PB + 64) + it]);
    const int qi = it / ncols, cj = it % ncols;
    if (cj < jb) G[qi][cj] = s;
    else P[qi][cj - jb] = s;
  }
  __syncthreads();
  if (tid == 0) {
    for (int i = 0; i < jb; ++i) {
      const double2 ti = tau[j0 + i];
      Tm[i][i] = ti;
      // T(0:i, i) = -tau_i * T(0:i,0:i) * G(0:i, i)
      double2 tmp[PB];
      for (int r = 0; r < i; ++r) tmp[r] = cscale(cmul(ti, G[r][i]), -1.0);
      for (int r = 0; r < i; ++r) {
        double2 s = make_double2(0, 0);
        for (int c = r; c < i; ++c) s = cadd(s, cmul(Tm[r][c], tmp[c]));
        Tm[r][i] = s;
      }
      for (int r = i + 1; r < jb; ++r) Tm[r][i] = make_double2(0, 0);
    }
  }
  __syncthreads();
  for (int it = tid; it < jb * nvec; it += blockDim.x) {
    const int r = it / nvec, c = it % nvec;
    double2 s = make_double2(0, 0);
    for (int k = r; k < jb; ++k) s = cadd(s, cmul(Tm[r][k], P[k][c]));
    Y[r * 64 + c] = s;
  }
}

__global__ void k_bt_apply(const double2* A, long long n, int j0, int jb, double2* X, int nvec, const double2* Y) {
  const long long r = (long long)j0 + 1 + blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (r >= n) return;
  for (int c = 0; c < nvec; ++c) {
    double2 s = make_double2(0, 0);
    for (int q = 0; q < jb; ++q) {
      if (r < (long long)j0 + q + 1) continue;
      s = cadd(s, cmul(A[r + (long long)(j0 + q) * n], Y[q * 64 + c]));
    }
    X[(long long)c * n + r] = csub(X[(long long)c * n + r], s);
  }
}

__global__ void k_real_to_complex(const double* z, double2* X, long long cnt) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < cnt) X[i] = make_double2(z[i], 0.0);
}

// rotate each vector so that its last component is real and >= 0 (ZHEEV 'U' convention)
// each vector times conj(last)/|last|: the last component becomes real >= 0 (exactly real, as
// ZHEEV('V','U') returns it).  The last component is read before any thread writes.
__global__ void k_gauge_last(double2* X, long long n, int nvec) {
  const int c = blockIdx.x;
  if (c >= nvec) return;
  __shared__ double2 s_last;
  if (threadIdx.x == 0) s_last = X[(long long)c * n + n - 1];
  __syncthreads();
  const double2 last = s_last;
  const double r = hypot(last.x, last.y);
  double2 ph = make_double2(1, 0);
  if (r > 0) ph = make_double2(last.x / r, -last.y / r);
  for (long long k = threadIdx.x; k < n; k += blockDim.x) {
    double2 v = cmul(X[(long long)c * n + k], ph);
    if (k == n - 1) v = make_double2(r, 0.0);
    X[(long long)c * n + k] = v;
  }
}

}  // namespace

static int tridiagonal_solve_body(wtbg_ctx* ctx, int dtfull, int cpol, bool vectors);

// the recurrences run on T scaled by a power of two to ||T|| <= 1
static double td_scale(double tnorm) {
  int ex = 0;
  if (tnorm > 0.0 && std::isfinite(tnorm)) (void)std::frexp(tnorm, &ex);
  return std::ldexp(1.0, -std::min(std::max(ex, -1000), 1000));
}

// Eigenvalues (bisection) and, with vectors, the fused oscillator sums of the tridiagonal
// form; timed as a whole when profiling.
int run_tridiagonal_solve(wtbg_ctx* ctx, int dtfull, int cpol, bool vectors) {
  if (!ctx->profiling) return tridiagonal_solve_body(ctx, dtfull, cpol, vectors);
  if (int r = ensure_events(ctx, 2)) return r;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  cudaEventRecord(e0, ctx->stream);
  const int r = tridiagonal_solve_body(ctx, dtfull, cpol, vectors);
  cudaEventRecord(e1, ctx->stream);
  cudaEventSynchronize(e1);
  float t = 0.f;
  if (!r && cudaEventElapsedTime(&t, e0, e1) == cudaSuccess) ctx->stats.tdsolve_ms += t;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return r;
}

static int tridiagonal_solve_body(wtbg_ctx* ctx, int dtfull, int cpol, bool vectors) {
  const long long n = ctx->N;
  cudaStream_t s = ctx->stream;
  std::vector<double> hd(n), he(n > 1 ? n - 1 : 1, 0.0);
  CK(cudaMemcpyAsync(hd.data(), ctx->d.as<double>(), n * 8, cudaMemcpyDeviceToHost, s));
  if (n > 1) CK(cudaMemcpyAsync(he.data(), ctx->e.as<double>(), (n - 1) * 8, cudaMemcpyDeviceToHost, s));
  int tri_err = 0;
  if (ctx->triErr.p) CK(cudaMemcpyAsync(&tri_err, ctx->triErr.p, 4, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (tri_err) return set_err(ctx, WTBG_ERR_CUDA, "tridiagonalise: a mat-vec pipeline wait timed out");
  double lo = hd[0], hi = hd[0], emax2 = 0.0;
  for (long long i = 0; i < n; ++i) {
    const double r = (i > 0 ? fabs(he[i - 1]) : 0.0) + (i < n - 1 ? fabs(he[i]) : 0.0);
    lo = std::min(lo, hd[i] - r);
    hi = std::max(hi, hd[i] + r);
    if (i < n - 1) emax2 = std::max(emax2, he[i] * he[i]);
  }
  const double tnorm = std::max(fabs(lo), fabs(hi));
  const double pivmin = DBL_MIN * std::max(1.0, emax2);
  // widen the Gershgorin interval slightly so that the extreme eigenvalues are interior
  const double pad = 2.0 * DBL_EPSILON * tnorm + 4.0 * pivmin + 1e-300;
  lo -= pad;
  hi += pad;
  ENSURE(ctx->lam, (size_t)n * 8);
  const double sc = td_scale(tnorm);
  const int npad = (int)((n + TD_TILE - 1) / TD_TILE * TD_TILE);
  ENSURE(ctx->tmp2, (size_t)npad * 48);
  double2* rcnt = ctx->tmp2.as<double2>();
  double2* rvec = rcnt + npad;
  k_td_records<<<(npad + 255) / 256, 256, 0, s>>>(ctx->d.as<double>(), ctx->e.as<double>(), (int)n, npad, sc, rcnt, rvec);
  CKL("k_td_records");
  if (ctx->nsm <= 0) cudaDeviceGetAttribute(&ctx->nsm, cudaDevAttrMultiProcessorCount, ctx->device);
  const int lanes = bisect_lanes(n, ctx->nsm);
  ENSURE(ctx->bgrid, (size_t)(BIS_P + 1) * (8 + 4) + 64);
  double* xg = ctx->bgrid.as<double>();
  int* cg = reinterpret_cast<int*>(xg + BIS_P + 1);
  k_bisect_grid<<<(BIS_P + TD_TILE) / TD_TILE, TD_TILE, 0, s>>>(rcnt, (int)n, lo, hi, sc, xg, cg);
  CKL("k_bisect_grid");
  k_bisect<<<(int)((n * lanes + TD_TILE - 1) / TD_TILE), TD_TILE, 0, s>>>(rcnt, n, xg, cg, pivmin, sc, lanes,
                                                                        ctx->lam.as<double>()); WTBG_COUNT(ctx, 3);
  CKL("k_bisect");
  ctx->lam_host.resize(n);
  CK(cudaMemcpyAsync(ctx->lam_host.data(), ctx->lam.as<double>(), n * 8, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (!vectors) return 0;

  // clusters (host): leaders carry the cluster size
  const std::vector<double>& L = ctx->lam_host;
  const double ctol = 1e-7 * std::max(1.0, tnorm);
  std::vector<int> csize(n, 0);
  long long maxc = 1;
  for (long long i = 0; i < n;) {
    long long jx = i + 1;
    while (jx < n && L[jx] - L[jx - 1] <= ctol) ++jx;
    csize[i] = (int)(jx - i);
    maxc = std::max(maxc, jx - i);
    i = jx;
  }
  // chunk size: the vectors of one launch run their chains side by side, so one launch for all
  // of them where the workspace fits (43.5 GB at N = 36864), else chunks
  size_t freeb = 0, totb = 0;
  CK(cudaMemGetInfo(&freeb, &totb));
  const double budget = std::min((double)freeb * 0.6 + (double)ctx->ws.bytes, 96e9);
  long long M = (long long)(budget / (4.0 * 8.0 * (double)n));
  if (M < n && lane_bytes(ctx) > 0) {   // the Q lanes of an earlier call do not split this one
    M = (long long)(std::min(budget + 0.6 * (double)lane_bytes(ctx), 96e9) / (4.0 * 8.0 * (double)n));
    release_lanes(ctx);
  }
  M = std::max<long long>(M, maxc);
  M = std::min<long long>(M, n);
  M = std::max<long long>(M, 1);
  const long long tM = (M + 31) / 32 * 32;   // slots of k_twist (its [npad][tM] is smaller but at the smallest n)
  ENSURE(ctx->ws, std::max<size_t>((size_t)4 * 8 * n * M, (size_t)npad * tM * 8 + (size_t)npad / 8 * tM * 4));
  ENSURE(ctx->act, (size_t)8 * 8 * n);
  ENSURE(ctx->csz, (size_t)n * 8 + 64);
  int* todo = ctx->csz.as<int>() + n;
  const bool twist = n >= TWIST_FROM;
  if (twist) {
    CK(cudaMemsetAsync(todo, 0, (size_t)n * 4, s));
    CK(cudaMemcpyAsync(ctx->csz.as<int>(), csize.data(), n * 4, cudaMemcpyHostToDevice, s));
  } else {
    CK(cudaMemcpyAsync(todo, csize.data(), n * 4, cudaMemcpyHostToDevice, s));
  }
  ctx->csize_host = csize;
  ctx->tnorm = tnorm;
  InvArgs a;
  a.d = ctx->d.as<double>();
  a.e = ctx->e.as<double>();
  a.n = n;
  a.lam = ctx->lam.as<double>();
  a.csize = todo;
  a.ws = ctx->ws.as<double>();
  a.pert = DBL_EPSILON * std::max(tnorm, DBL_MIN);
  a.g = ctx->g.as<double2>();
  a.ng = ctx->ng;
  a.act = ctx->act.as<double>();
  a.dtfull = dtfull;
  a.cpol = cpol;
  a.zsel = nullptr;
  a.zs0 = -1;
  a.zs1 = -1;
  TwistArgs tw;
  tw.rec = rvec;
  tw.n = (int)n;
  tw.npad = npad;
  tw.sc = sc;
  tw.lam = a.lam;
  tw.csize = ctx->csz.as<int>();
  tw.todo = todo;
  tw.M = (int)tM;
  tw.t = ctx->ws.as<double>();
  tw.te = reinterpret_cast<int*>(tw.t + (size_t)npad * tM);
  tw.g = a.g;
  tw.act = a.act;
  tw.dtfull = dtfull;
  tw.cpol = cpol;
  // the residual of the joined row is |lambda's error| / |z_r|, and |z_r| >= ||z|| / sqrt(n)
  tw.rtol = 8.0 * DBL_EPSILON * std::sqrt((double)n);
  tw.keep = false;
  for (long long m0 = 0; m0 < n;) {
    // end the chunk at a cluster start
    long long m1 = std::min(n, m0 + M);
    if (m1 < n) {
      while (m1 > m0 && csize[m1] == 0) --m1;
      if (m1 == m0) m1 = std::min(n, m0 + M);
    }
    a.m0 = m0;
    a.m1 = m1;
    a.M = (int)M;
    const int cnt = (int)(m1 - m0);
    tw.m0 = (int)m0;
    tw.m1 = (int)m1;
    if (twist)
      if (int r = a.ng == 10 ? launch_twist<10>(ctx, tw, maxc > 1) : launch_twist<5>(ctx, tw, maxc > 1)) return r;
    k_inviter<<<(cnt + 63) / 64, 64, 0, s>>>(a); WTBG_COUNT(ctx, 1);
    CKL("k_inviter");
    m0 = m1;
  }
  return 0;
}

int run_eigvecs(wtbg_ctx* ctx, int n0, int n1, double2* d_out) {
  const long long n = ctx->N;
  const int nvec = n1 - n0 + 1;
  if (nvec > 32) return set_err(ctx, WTBG_ERR_UNSUPPORTED, "eigvecs: at most 32 vectors per launch");
  cudaStream_t s = ctx->stream;
  // tridiagonal eigenvectors of the requested range, recomputed over the whole clusters that contain
  // n0-1 .. n1-1 (0-based)
  {
    const std::vector<int>& cs = ctx->csize_host;
    long long lead = n0 - 1;
    while (lead > 0 && cs[lead] == 0) --lead;
    long long end = n1 - 1;
    {
      long long l2 = end;
      while (l2 > 0 && cs[l2] == 0) --l2;
      end = l2 + cs[l2];
    }
    const long long M = end - lead, tM = (M + 31) / 32 * 32;
    const int npad = (int)((n + TD_TILE - 1) / TD_TILE * TD_TILE);
    ENSURE(ctx->ws, (size_t)4 * 8 * n * M + (size_t)npad * tM * 8 + (size_t)npad / 8 * tM * 4);
    ENSURE(ctx->zsel, (size_t)8 * n * nvec);
    ENSURE(ctx->tmp2, (size_t)npad * 48 + (size_t)8 * 8 * n);
    double2* rec = ctx->tmp2.as<double2>();
    int* todo = ctx->csz.as<int>() + n;
    TwistArgs tw;
    tw.rec = rec + npad;
    tw.n = (int)n;
    tw.npad = npad;
    tw.sc = td_scale(ctx->tnorm);
    tw.lam = ctx->lam.as<double>();
    tw.csize = ctx->csz.as<int>();
    tw.todo = todo;
    tw.m0 = (int)lead;
    tw.m1 = (int)end;
    tw.M = (int)tM;
    tw.t = ctx->ws.as<double>() + (size_t)4 * n * M;
    tw.te = reinterpret_cast<int*>(tw.t + (size_t)npad * tM);
    tw.g = ctx->g.as<double2>();
    tw.act = reinterpret_cast<double*>(rec + 3 * (size_t)npad);   // not kept
    tw.dtfull = 0;
    tw.cpol = 0;
    tw.rtol = 8.0 * DBL_EPSILON * std::sqrt((double)n);
    tw.keep = true;
    const bool twist = n >= TWIST_FROM;   // else todo still holds the clusters of the solve
    if (twist) {
      k_td_records<<<(npad + 255) / 256, 256, 0, s>>>(ctx->d.as<double>(), ctx->e.as<double>(), (int)n, npad, tw.sc, rec,
                                                      rec + npad);
      WTBG_COUNT(ctx, 1);
      CKL("k_td_records");
      CK(cudaMemsetAsync(todo, 0, (size_t)n * 4, s));
      if (int r = ctx->ng == 10 ? launch_twist<10>(ctx, tw, true) : launch_twist<5>(ctx, tw, true)) return r;
    }
    InvArgs a;
    a.d = ctx->d.as<double>();
    a.e = ctx->e.as<double>();
    a.n = n;
    a.lam = ctx->lam.as<double>();
    a.csize = todo;
    a.m0 = lead;
    a.m1 = end;
    a.M = (int)M;
    a.ws = ctx->ws.as<double>();
    a.pert = DBL_EPSILON * std::max(ctx->tnorm, DBL_MIN);
    a.g = ctx->g.as<double2>();
    a.ng = ctx->ng;
    a.act = tw.act;
    a.dtfull = 0;
    a.cpol = 0;
    a.zsel = ctx->zsel.as<double>();
    a.zs0 = n0 - 1;
    a.zs1 = n1 - 1;
    k_inviter<<<(int)((M + 63) / 64), 64, 0, s>>>(a); WTBG_COUNT(ctx, 1);
    CKL("k_inviter(eigvecs)");
    if (twist) {
      k_take_vectors<<<dim3((unsigned)((n + 255) / 256), nvec), 256, 0, s>>>(tw, n0 - 1, ctx->zsel.as<double>());
      WTBG_COUNT(ctx, 1);
      CKL("k_take_vectors");
    }
  }
  const long long cnt = (long long)nvec * n;
  k_real_to_complex<<<(int)((cnt + 255) / 256), 256, 0, s>>>(ctx->zsel.as<double>(), d_out, cnt); WTBG_COUNT(ctx, 1);
  CKL("k_real_to_complex");
  if (ctx->tri_two) {
    if (int r = run_backtransform2(ctx, d_out, nvec)) return r;
    k_gauge_last<<<nvec, 256, 0, s>>>(d_out, n, nvec); WTBG_COUNT(ctx, 1);
    CKL("k_gauge_last");
    return 0;
  }
  const int nparts_max = (int)((n + BT_RB - 1) / BT_RB) + 1;
  ENSURE(ctx->tmp, (size_t)nparts_max * PB * (PB + 64) * 16 + PB * 64 * 16 + 1024);
  double2* part = ctx->tmp.as<double2>();
  double2* Y = part + (size_t)nparts_max * PB * (PB + 64);
  const size_t shb = (size_t)PB * (PB + 64) * 16;
  CK(cudaFuncSetAttribute(k_bt_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shb));
  // panels in reverse order: Q X = P_0 (P_1 (... (P_last X)))
  const long long npan = (n - 1 + PB - 1) / PB;
  for (long long pnl = npan - 1; pnl >= 0; --pnl) {
    const int j0 = (int)(pnl * PB);
    const int jb = (int)std::min<long long>(PB, n - 1 - j0);
    const int nrows = (int)(n - j0 - 1);
    const int nparts = (nrows + BT_RB - 1) / BT_RB;
    k_bt_gram<<<nparts, BT_RB, shb, s>>>(ctx->H.as<double2>(), n, j0, jb, d_out, nvec, part); WTBG_COUNT(ctx, 1);
    k_bt_tmat<<<1, 256, 0, s>>>(part, nparts, jb, nvec, ctx->tau.as<double2>(), j0, Y); WTBG_COUNT(ctx, 1);
    k_bt_apply<<<(nrows + 255) / 256, 256, 0, s>>>(ctx->H.as<double2>(), n, j0, jb, d_out, nvec, Y); WTBG_COUNT(ctx, 1);
  }
  CKL("back-transform");
  k_gauge_last<<<nvec, 256, 0, s>>>(d_out, n, nvec); WTBG_COUNT(ctx, 1);
  CKL("k_gauge_last");
  return 0;
}
