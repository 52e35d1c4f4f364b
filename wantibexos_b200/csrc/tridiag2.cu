// Kernel (c), two-stage form: reduction of the Hermitian BSE matrix to real symmetric
// tridiagonal form in two steps, dense -> band (bandwidth b = 32) -> tridiagonal.
//
// Reference: the dense ZHEEV('V','U') of bsesolver (subprograms/bse_solver-tool-diel.f90:
// 485-492) and ZHEEV('N','U') of bsebnds (bse_kpath-tool.f90:384-387).  The one-stage
// reduction (tridiag.cu) streams the whole trailing matrix once per column in a Hermitian
// matrix-vector product, so half of its flops run at HBM speed.  Here:
//
// Stage 1 (dense -> band), per panel of b columns j0..j0+b-1 with k0 = j0 + b:
//   (1) k_panel_qr_cl, k_panel_qr: Householder QR of the panel A[k0:N, j0:j0+b] (ZLARFG reflectors,
//       one cluster whose CTAs keep their rows in registers, or for long panels one cooperative
//       launch with the row slices in shared memory); the T factor of the block reflector Q = I - V T V^H; the velocity
//       vectors g <- Q^T g = g - conj(V) T^T (V^T g).
//   (2) k_hemm2: X = A22 V on the FP64 tensor cores (mma.sync m16n8k16), A22 = A[k0:N, k0:N]
//       read once from its stored lower triangle (tiles above the diagonal are read transposed
//       and conjugated, the diagonal tiles mirrored on the way), split over K into
//       deterministic partial sums.
//   (3) k_wfuse: W = (X - 1/2 V T^H V^H X) T, with the corrections of the look-ahead group.
//   (4) k_her2k (tridiag.cu): A22 -= V W^H + W V^H, so that A22 <- Q^H A22 Q.
//   Both large products are GEMM-shaped, so the stage runs at tensor-core speed where the
//   one-stage mat-vec runs at HBM speed.
// Stage 2 (band -> tridiagonal, bulge chasing) is in the second half of this file.
// The oscillator strengths need only A^T h = Z^T (Q^T h), so no O(N^3) back-transform is formed.
#include <cfloat>

#include "common.cuh"
#include "tc_sm100.cuh"

#include <algorithm>
#include <mutex>
#include <string>

// implemented in tridiag.cu
int launch_her2k_v(wtbg_ctx* ctx, double2* A, long long N, const double2* Wp, const double2* V, long long vld, int vc0,
                   int jb, long long k0, bool beside);

namespace {

constexpr int BW = 32;            // band width b of the two-stage reduction (= WTBG_PANEL)
constexpr int PQ_THREADS = 256;   // threads of the panel QR kernel
constexpr int PQ_MAXG = 160;      // largest panel-QR grid (one CTA per SM; the host checks)
constexpr int NGMAX = 10;         // velocity vectors carried through (x, y, z, sp, sm [, times f])

__device__ __forceinline__ double2 warp_sum2(double2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned int* p, unsigned int v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
constexpr unsigned long long kWaitNs = 2000000000ull;   // 2 s bound on every spin wait

// Bounded acquire-wait until *p >= need.  The error flag and the clock are read every 64 polls,
// so that a detection costs one L2 round trip; after 2 s, or when another CTA or warp has
// failed, the flag is set and the wait reports failure.
__device__ __forceinline__ bool wait_at_least(const unsigned int* p, unsigned int need, int* err) {
  unsigned int spins = 0;
  unsigned long long t0 = 0;
  while (ld_acquire(p) < need) {
    if ((++spins & 63u) == 0u) {
      if (t0 == 0) t0 = globaltimer();
      if (ld_acquire(reinterpret_cast<unsigned int*>(err)) != 0u || globaltimer() - t0 > kWaitNs) {
        atomicExch(err, 1);
        return false;
      }
    }
  }
  return true;
}

// Grid barrier among the co-resident CTAs of a cooperative launch.  Each launch has its own
// arrival counter, zeroed before the launch; barrier k of the launch is passed when the counter
// reaches k * gridDim.x.  Thread 0 arrives with a release reduction (no returned value, no reset
// step) and polls with acquire loads; the CTA barrier around it orders the other threads' memory
// operations (as in a cooperative-groups grid sync).  The wait is bounded (2 s of %globaltimer);
// on time-out (or when another CTA has already failed) the CTA sets *err and the barrier reports
// failure, after which every CTA leaves the kernel.
__device__ bool grid_sync(unsigned int* cnt, unsigned int target, int* err) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(cnt) : "memory");
    s_ok = wait_at_least(cnt, target, err) ? 1 : 0;
  }
  __syncthreads();
  return s_ok != 0;
}

// ----------------------------------------------------------------------------- stage 1
// Panel QR.  CTA c owns rows [k0 + c*R, k0 + min((c+1)*R, m)) of the panel, kept in shared
// memory as P[col][row] (row fastest).  Per column p: ZLARFG from the grid-reduced norm (every
// CTA sums the same partials in the same order, so all hold identical scalars), then the
// reflector is applied to the panel's remaining columns with grid-reduced dot products.
// The column step is one latency chain (grid barrier, reduction of the CTAs' partials, scalars,
// update, next partials), so every part of it uses all threads: 8 threads per column reduce the
// partials and form the next ones (fixed order, width-8 shuffle tree), every thread evaluates
// the reflector scalars itself, and the update runs over (row, 8-column chunk) items.
struct PanelArgs {
  double2* A;
  long long N;
  int j0, k0, jb;      // panel columns j0 .. j0+jb-1, first panel row k0
  int nref;            // reflectors: min(jb, N - k0)
  int R;               // rows per CTA
  int RS;              // column stride of the panel slice in shared memory (R rounded up to odd)
  double2* Vp;         // [32][N] dense V (rows k0.. written, explicit unit and zeros)
  double2* Tout;       // [32][32] column-major T factor
  double2* g;          // [ng][N]
  int ng;
  double2* partW;      // [2][grid][32] partial norms (column p) and unscaled dots, by parity of p
  double2* partG;      // [grid][32*32]
  double2* partVg;     // [grid][32*NGMAX]
  double2* alpha;      // [2][32] posted row k0 + p (alpha = its column-p entry), by parity of p
  unsigned int* cnt;   // this launch's grid-barrier arrival counter (zero at launch)
  int* err;
};

__device__ __forceinline__ double2 ldcg2(const double2* p) { return __ldcg(p); }
// a following kernel launched to run beside this one may start (any other still waits for the end)
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__global__ void __launch_bounds__(PQ_THREADS, 1) k_panel_qr(PanelArgs a) {
  pdl_release();
  extern __shared__ __align__(16) double2 P[];   // [jb][R]
  __shared__ double2 s_tau[BW];
  __shared__ double2 s_w[BW];
  __shared__ double2 s_S[BW];    // grid-reduced S_q of the current column (q >= p)
  __shared__ double2 s_al[BW];   // posted row k0 + p
  __shared__ double2 s_T[BW * BW];
  __shared__ double2 s_y[BW * NGMAX];
  const int tid = threadIdx.x;
  const int R = a.R, RS = a.RS, jb = a.jb;   // rows per CTA; shared-memory column stride (odd)
  const long long N = a.N;
  const int G = (int)gridDim.x;
  const long long rbeg = (long long)a.k0 + (long long)blockIdx.x * R;
  const long long rend = min((long long)a.k0 + (long long)(blockIdx.x + 1) * R, N);
  const int nr = (int)max(0LL, rend - rbeg);
  unsigned int nbar = 0;
  auto sync_grid = [&]() -> bool {
    ++nbar;
    return grid_sync(a.cnt, nbar * (unsigned int)G, a.err);
  };
  for (int q = 0; q < jb; ++q)
    for (int i = tid; i < R; i += PQ_THREADS)
      P[(size_t)q * RS + i] = (i < nr) ? a.A[(rbeg + i) + (long long)(a.j0 + q) * N] : make_double2(0, 0);
  __syncthreads();

  // width-8 sum over the aligned lane groups of 8 (every lane of a group ends with the same sum)
  auto sum8 = [](double2 v) {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
  };
  const int qq = tid >> 3, sl = tid & 7;   // column offset and slice of the 8-thread groups

  // Partials of column p over the own rows below row k0 + p, one reduction for both the norm
  // and the unscaled dot products: S_q = sum_{r > k0+p} conj(P[r,p]) P[r,q] for q = p .. jb-1
  // (S_p = |x|^2); thread slice sl takes the rows i = sl (mod 8).  The owner of row k0 + p
  // posts that row (alpha = P[k0+p, p] and P[k0+p, q]).  Buffers alternate with the parity of
  // p: a CTA writes the partials of column p+1 while others may still read those of p, but
  // never those of p+2 before everyone passed the barrier of p+1.
  auto partials = [&](int p) {
    const long long rp = (long long)a.k0 + p;
    const int buf = p & 1;
    double2 sacc = make_double2(0, 0);
    if (qq < jb - p) {
      const double2* Pp = P + (size_t)p * RS;
      const double2* Pq = P + (size_t)(p + qq) * RS;
      const int i0 = (int)max(0LL, rp + 1 - rbeg);
      for (int i = i0 + ((sl - i0) & 7); i < nr; i += 8) sacc = cadd(sacc, cmulc(Pp[i], Pq[i]));
    }
    sacc = sum8(sacc);
    if (qq < jb - p && sl == 0) a.partW[((size_t)buf * G + blockIdx.x) * BW + p + qq] = sacc;
    if (rp >= rbeg && rp < rend)
      for (int q = p + tid; q < jb; q += PQ_THREADS) a.alpha[buf * BW + q] = P[(size_t)q * RS + (rp - rbeg)];
  };

  partials(0);
  for (int p = 0; p < a.nref; ++p) {
    if (!sync_grid()) return;
    const long long rp = (long long)a.k0 + p;
    const int buf = p & 1;
    // grid reduction of S_q (q = p + qq): slice sl sums the CTAs c = sl (mod 8) in order, its
    // (at most PQ_MAXG / 8) loads issued together
    {
      double2 sacc = make_double2(0, 0);
      if (qq < jb - p) {
        double2 pv[PQ_MAXG / 8];
#pragma unroll
        for (int u = 0; u < PQ_MAXG / 8; ++u) {
          const int c = sl + 8 * u;
          pv[u] = (c < G) ? ldcg2(a.partW + ((size_t)buf * G + c) * BW + p + qq) : make_double2(0, 0);
        }
#pragma unroll
        for (int u = 0; u < PQ_MAXG / 8; ++u)
          if (sl + 8 * u < G) sacc = cadd(sacc, pv[u]);
      }
      sacc = sum8(sacc);
      if (qq < jb - p) {
        if (sl == 0) s_S[p + qq] = sacc;
        else if (sl == 1) s_al[p + qq] = ldcg2(a.alpha + buf * BW + p + qq);
      }
    }
    __syncthreads();
    // ZLARFG scalars, evaluated by every thread from the same shared values
    double2 tau, scal;
    double beta;
    {
      const double xn2 = s_S[p].x;
      const double2 al = s_al[p];
      if (xn2 == 0.0 && al.y == 0.0) {
        tau = make_double2(0, 0);
        scal = make_double2(0, 0);
        beta = al.x;
      } else {
        beta = -copysign(sqrt(al.x * al.x + al.y * al.y + xn2), al.x);
        tau = make_double2((beta - al.x) / beta, -al.y / beta);
        const double2 den = make_double2(al.x - beta, al.y);
        const double dd = den.x * den.x + den.y * den.y;
        scal = make_double2(den.x / dd, -den.y / dd);
      }
    }
    if (tid == 0) s_tau[p] = tau;
    // P[r,q] -= conj(tau) v_r w_q (r >= k0+p, q > p), with v_r = P[r,p] scal (v = 1 at row
    // k0+p) and w_q = sum_{r >= k0+p} conj(v_r) P[r,q] = P[k0+p, q] + conj(scal) S_q
    {
      const double2 ct = cconj(tau);
      const int nch = (jb - p - 1 + 7) >> 3;
      for (int it = tid; it < nr * nch; it += PQ_THREADS) {
        const int i = it % nr, ch = it / nr;
        const long long r = rbeg + i;
        if (r < rp) continue;
        const double2 v = (r == rp) ? make_double2(1.0, 0.0) : cmul(P[(size_t)p * RS + i], scal);
        const double2 cv = cmul(ct, v);
        const int q0 = p + 1 + ch * 8, q1 = min(q0 + 8, jb);
        for (int q = q0; q < q1; ++q) {
          const double2 wq = cadd(s_al[q], cmul(cconj(scal), s_S[q]));
          P[(size_t)q * RS + i] = csub(P[(size_t)q * RS + i], cmul(cv, wq));
        }
      }
    }
    __syncthreads();
    // column p becomes v (beta on row k0+p), then the partials of column p+1
    for (int i = tid; i < nr; i += PQ_THREADS) {
      const long long r = rbeg + i;
      if (r == rp) P[(size_t)p * RS + i] = make_double2(beta, 0.0);
      else if (r > rp) P[(size_t)p * RS + i] = cmul(P[(size_t)p * RS + i], scal);
    }
    if (p + 1 < a.nref) partials(p + 1);
  }
  __syncthreads();
  // write back: A keeps R (rows <= k0+q) and v below; Vp gets V with its unit and zeros
  auto vval = [&](int q, int i) -> double2 {
    const long long r = rbeg + i, rq = (long long)a.k0 + q;
    if (q >= a.nref || r < rq) return make_double2(0, 0);
    if (r == rq) return make_double2(1.0, 0.0);
    return P[(size_t)q * RS + i];
  };
  for (int q = 0; q < jb; ++q)
    for (int i = tid; i < nr; i += PQ_THREADS) {
      a.A[(rbeg + i) + (long long)(a.j0 + q) * N] = P[(size_t)q * RS + i];
      a.Vp[(rbeg + i) + (long long)q * N] = vval(q, i);
    }
  // P becomes the explicit V (unit on row k0+q, zeros above it and in columns >= nref), so that
  // the Gram and velocity sums below run without branches
  __syncthreads();
  const int nref = a.nref;
  for (int q = 0; q < jb; ++q)
    for (int i = tid; i < nr; i += PQ_THREADS) {
      const long long r = rbeg + i, rq = (long long)a.k0 + q;
      if (q >= nref || r < rq) P[(size_t)q * RS + i] = make_double2(0, 0);
      else if (r == rq) P[(size_t)q * RS + i] = make_double2(1.0, 0.0);
    }
  __syncthreads();
  // Gram partial V^H V over the own rows: thread t sums the four entries (t mod 32, t/32 + 8k) in
  // one pass (one column per lane, the odd stride keeps the 32 lanes on distinct banks; the
  // other column is a broadcast), rows in order
  {
    const int qi = tid & (BW - 1), qj0 = tid >> 5;
    double2 s4[4] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
    const double2* Pi = P + (size_t)qi * RS;
    for (int i = 0; i < nr; ++i) {
      const double2 vi = Pi[i];
#pragma unroll
      for (int k = 0; k < 4; ++k) s4[k] = cadd(s4[k], cmulc(vi, P[(size_t)(qj0 + 8 * k) * RS + i]));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) a.partG[(size_t)blockIdx.x * BW * BW + tid + PQ_THREADS * k] = s4[k];
  }
  // V^T g over the own rows, rows in order; the loads of 16 rows are issued together
  for (int e = tid; e < BW * a.ng; e += PQ_THREADS) {
    const int q = e % BW, al = e / BW;
    const double2* gp = a.g + (long long)al * N + rbeg;
    double2 s = make_double2(0, 0);
    for (int i0 = 0; i0 < nr; i0 += 16) {
      double2 gv[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) gv[u] = (i0 + u < nr) ? __ldcg(gp + i0 + u) : make_double2(0, 0);
#pragma unroll
      for (int u = 0; u < 16; ++u)
        if (i0 + u < nr) s = cadd(s, cmul(P[(size_t)q * RS + i0 + u], gv[u]));
    }
    a.partVg[(size_t)blockIdx.x * BW * NGMAX + e] = s;
  }
  if (!sync_grid()) return;
  // Sum of the CTAs' partials in CTA order, the loads of 8 partials issued together
  auto sum_parts = [&](const double2* base, size_t stride, int e) {
    double2 s = make_double2(0, 0);
    for (int c0 = 0; c0 < G; c0 += 8) {
      double2 pv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) pv[u] = (c0 + u < G) ? ldcg2(base + (size_t)(c0 + u) * stride + e) : make_double2(0, 0);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (c0 + u < G) s = cadd(s, pv[u]);
    }
    return s;
  };
  // every CTA: y = V^T g (needed after the T factor; reduced while CTA 0 forms T)
  for (int e = tid; e < BW * a.ng; e += PQ_THREADS) s_y[e] = sum_parts(a.partVg, (size_t)BW * NGMAX, e);   // [q + al*BW]
  // T factor (ZLARFT forward columnwise): T[i][i] = tau_i, T[0:i, i] = -tau_i T[0:i, 0:i] G[0:i, i]
  if (blockIdx.x == 0) {
    for (int e = tid; e < BW * BW; e += PQ_THREADS) s_T[e] = sum_parts(a.partG, (size_t)BW * BW, e);   // G for now (qi + qj * BW)
    __syncthreads();
    // column by column on one warp; column i of T is built in s_w from G(:, i) before T(:, i) is
    // stored
    if (tid < BW) {
      for (int i = 0; i < BW; ++i) {
        s_w[tid] = (tid < i && i < nref) ? s_T[tid + i * BW] : make_double2(0, 0);
        __syncwarp();
        double2 t = make_double2(0, 0);
        if (i < nref && tid < i) {
          for (int l = tid; l < i; ++l) t = cadd(t, cmul(s_T[tid + l * BW], s_w[l]));   // T[tid][l] for l < i
          t = cscale(cmul(s_tau[i], t), -1.0);
        } else if (i < nref && tid == i) {
          t = s_tau[i];
        }
        // column i of the G storage is no longer needed below the diagonal: the T entries of
        // rows < i overwrite G(0:i, i); rows >= i become T's diagonal and zeros
        s_T[tid + i * BW] = t;
        __syncwarp();
      }
    }
    __syncthreads();
    // s_T now holds T upper triangular; G entries below the diagonal were overwritten with 0
    for (int e = tid; e < BW * BW; e += PQ_THREADS) a.Tout[e] = s_T[e];
  }
  if (!sync_grid()) return;
  // g <- g - conj(V) T^T (V^T g)
  for (int e = tid; e < BW * BW; e += PQ_THREADS) s_T[e] = ldcg2(a.Tout + e);
  __syncthreads();
  // z = T^T y into s_w-sized scratch: z[j][al] = sum_{i <= j} T[i][j] y[i][al]
  __shared__ double2 s_z[BW * NGMAX];
  for (int e = tid; e < BW * a.ng; e += PQ_THREADS) {
    const int j = e % BW, al = e / BW;
    double2 s = make_double2(0, 0);
    for (int i = 0; i <= j; ++i) s = cadd(s, cmul(s_T[i + j * BW], s_y[i + al * BW]));
    s_z[e] = s;
  }
  __syncthreads();
  for (int e = tid; e < nr * a.ng; e += PQ_THREADS) {
    const int i = e % nr, al = e / nr;
    double2 s = make_double2(0, 0);
    for (int q = 0; q < nref; ++q) s = cadd(s, cmul(cconj(vval(q, i)), s_z[q + al * BW]));
    double2* gp = a.g + (long long)al * N + rbeg + i;
    *gp = csub(*gp, s);
  }
}


__device__ __forceinline__ double2 shfl2(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
__device__ __forceinline__ double2 shfl2_xor(double2 v, int o) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
// c + a b, c - a b, c + conj(a) b, c - conj(a) b: four FMAs each
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {
  return make_double2(fma(-a.y, b.y, fma(a.x, b.x, c.x)), fma(a.y, b.x, fma(a.x, b.y, c.y)));
}
__device__ __forceinline__ double2 cfms(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.y, b.y, fma(-a.x, b.x, c.x)), fma(-a.y, b.x, fma(-a.x, b.y, c.y)));
}
__device__ __forceinline__ double2 cfmac(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.y, b.y, fma(a.x, b.x, c.x)), fma(-a.y, b.x, fma(a.x, b.y, c.y)));
}
__device__ __forceinline__ double2 cfmsc(double2 a, double2 b, double2 c) {
  return make_double2(fma(-a.y, b.y, fma(-a.x, b.x, c.x)), fma(a.y, b.x, fma(-a.x, b.y, c.y)));
}
__device__ __forceinline__ double2 caxpy(double a, double2 b, double2 c) {
  return make_double2(fma(a, b.x, c.x), fma(a, b.y, c.y));
}
// Reflector scalars of x (first entry al, xn2 = the squared norm of the others): beta =
// -sign(Re al) |x|, kappa = -u_0 / (beta |u_0|^2), 1/beta, 1/|u_0|^2; no reflector (kappa = 0, al kept)
// where x is already (real, 0, ..., 0), or so small that |x|^2 is not a normal number.  kappa is of order |x|^-2 and
// formed from factors that stay between |x|^-2 and 2, so it is finite for every |x| that is taken; of its products
// only those with two vectors of order |x| are formed, never its square (which is infinite from |x| = 1e-77 down).
__device__ __forceinline__ void reflector_scalars(double2 al, double xn2, double2& kap, double& beta, double& ib, double& rd) {
  const double ay2 = al.y * al.y;
  const double q = fma(al.x, al.x, ay2 + xn2);
  kap = make_double2(0, 0);
  beta = al.x;
  ib = rd = 0.0;
  if (q >= DBL_MIN && !(xn2 == 0.0 && al.y == 0.0)) {
    ib = -copysign(rsqrt(q), al.x);
    beta = -copysign(sqrt(q), al.x);
    const double ux = al.x - beta;
    rd = 1.0 / fma(ux, ux, ay2);
    kap = make_double2(-(ib * ux) * rd, -(ib * al.y) * rd);
  }
}

// Panel QR on one cluster of C <= 16 CTAs, for panels of up to 16 x 8 x PC_NR rows.  CTA c owns rows
// [k0 + cR, k0 + (c+1)R), R = 8 NR, and keeps them in registers: eight threads per column hold its rows
// i = 8u + sl, and the conjugated velocity vectors are further columns.  Column step p: every column's
// dot product S_q = sum_{r > k0+p} conj(x_r) P_rq with the pivot column x (in shared memory, zero up to
// row p), the CTAs' sums exchanged through distributed shared memory, counted by mbarriers; then with the
// unscaled vector u = x - beta e_p the reflector is H = I - kappa u u^H and w_q = u^H P_q = S_q +
// conj(u_p) P_pq (row p is posted by CTA 0) serves three ends: columns q > p are updated by P_q -=
// conj(kappa) w_q u, finished columns q < p give the Gram entry v_q^H v_p = conj(w_q) / u_p that the T factor
// needs, and the velocity columns give V^T g the same way.  The last warp, which holds no column, forms T
// one column behind.
// Bound by the latency of the column chain.  The grid-wide form (k_panel_qr, still used for longer
// panels) pays a barrier and two round trips through L2 per column, keeps the slice in shared memory
// (whose bandwidth bounds update and dot products) and forms Gram matrix and V^T g in passes of their
// own.  Per panel, grid-wide against cluster: N = 576 170 / 68 us, 2304 189 / 91 us (with cluster barriers and T by
// doubling; 59 us at 144 rows and 105 at 2272 against 70 and 115 since the exchange is counted and T formed along).
constexpr int PC_THREADS = 384;   // 48 columns x 8 threads: 32 of the panel, up to 10 velocity vectors
constexpr int PC_COLS = BW + NGMAX;
constexpr int PC_MAXC = 16;
constexpr int PC_MAX_NR = 24;
constexpr size_t pc_smem(int nr) {
  return sizeof(double2) * (size_t)(2 * PC_MAXC * PC_COLS + 2 * BW * BW + 2 * BW * NGMAX + BW * (8 * nr + 1));
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address in CTA `cta` of the cluster of what lies at p here
__device__ __forceinline__ uint32_t cluster_map(const void* p, uint32_t cta) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(cta));
  return r;
}
// 16 bytes into another CTA's shared memory, counted by its mbarrier
__device__ __forceinline__ void st_async16(uint32_t addr, uint32_t mbar, double2 v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "d"(v.x), "d"(v.y), "r"(mbar)
               : "memory");
}
// arrive for a phase of the own mbarrier that `bytes` will come to
__device__ __forceinline__ void mbar_expect(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t mbar, uint32_t parity) {
  unsigned long long t0 = 0;
  for (unsigned int spins = 1;; ++spins) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((spins & 63u) == 0u) {
      if (t0 == 0) t0 = globaltimer();
      if (globaltimer() - t0 > kWaitNs) return false;
    }
  }
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int NR>
__global__ void __launch_bounds__(PC_THREADS, 1) k_panel_qr_cl(PanelArgs a, int C) {
  pdl_release();
  constexpr int R = 8 * NR, VS = R + 1;
  extern __shared__ __align__(16) double2 psm[];
  double2(*s_part)[PC_MAXC][PC_COLS] = reinterpret_cast<double2(*)[PC_MAXC][PC_COLS]>(psm);   // dot products, by parity of p
  double2* s_G = psm + 2 * PC_MAXC * PC_COLS;
  double2* s_T = s_G + BW * BW;
  double2* s_y = s_T + BW * BW;
  double2* s_z = s_y + BW * NGMAX;
  double2* Vs = s_z + BW * NGMAX;                      // [32][VS]: V of the own rows, at the end
  __shared__ double2 s_x[2][R];                        // pivot column by parity of p
  __shared__ double2 s_al[2][PC_COLS];                 // row p
  __shared__ double2 s_tau[BW];
  __shared__ double2 s_sc[2][3];                       // kappa; (beta, 0); 1/u_p
  __shared__ __align__(8) unsigned long long s_bar[2]; // arrivals for column p, by parity of p
  const int tid = threadIdx.x, lane = tid & 31, sl = tid & 7, q = tid >> 3;
  const int c = (int)cluster_rank();
  const long long N = a.N;
  const long long rbeg = (long long)a.k0 + (long long)c * R;
  const int nr = (int)max(0LL, min((long long)R, N - rbeg));
  const int nref = a.nref, ng = a.ng;
  const bool panel = q < BW, vel = q >= BW && q < BW + ng;
  double2 P[NR];
#pragma unroll
  for (int u = 0; u < NR; ++u) {
    const int i = 8 * u + sl;
    P[u] = make_double2(0, 0);
    if (i < nr) {
      if (panel) P[u] = a.A[(rbeg + i) + (long long)(a.j0 + q) * N];
      else if (vel) P[u] = cconj(__ldcg(a.g + (long long)(q - BW) * N + rbeg + i));
    }
  }
  // the pivot column p into s_x (zero up to row p, which only CTA 0 holds), by its eight threads
  auto post = [&](int p) {
#pragma unroll
    for (int u = 0; u < NR; ++u) s_x[p & 1][8 * u + sl] = (c == 0 && 8 * u + sl <= p) ? make_double2(0, 0) : P[u];
  };
  auto sum8 = [](double2 v) {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v = cadd(v, shfl2_xor(v, o));
    return v;
  };
  // T(0:p, p) = -tau_p T(0:p, 0:p) G(0:p, p), lane = row
  auto t_column = [&](int p) {
    const double2 tau = s_tau[p];
    double2 t0 = make_double2(0, 0), t1 = t0;
    int l = 0;
    for (; l + 1 < p; l += 2) {   // T is zero below its diagonal
      t0 = cfma(s_T[lane + l * BW], s_G[l + p * BW], t0);
      t1 = cfma(s_T[lane + (l + 1) * BW], s_G[l + 1 + p * BW], t1);
    }
    if (l < p) t0 = cfma(s_T[lane + l * BW], s_G[l + p * BW], t0);
    const double2 t = cmul(tau, cadd(t0, t1));
    if (lane <= p) s_T[lane + p * BW] = lane == p ? tau : make_double2(-t.x, -t.y);
    __syncwarp();
  };
  for (int e = tid; e < BW * BW; e += PC_THREADS) s_G[e] = s_T[e] = make_double2(0, 0);
  for (int e = tid; e < BW * NGMAX; e += PC_THREADS) s_y[e] = make_double2(0, 0);
  if (tid < BW) s_tau[tid] = make_double2(0, 0);
  if (q == 0) post(0);
  const uint32_t bar = (uint32_t)__cvta_generic_to_shared(s_bar);
  const int nq = BW + ng;                                   // columns that are exchanged
  const uint32_t bytes = (uint32_t)((C + 1) * nq * 16);     // their sums from every CTA, and row p from CTA 0
  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8 * b) : "memory");
      mbar_expect(bar + 8 * b, bytes);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  cluster_sync();   // every CTA of the cluster runs and has its mbarriers (both are written below)
  uint32_t rpart[2], ral[2], rbar[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t cta = (uint32_t)min(sl + 8 * k, C - 1);
    rpart[k] = cluster_map(&s_part[0][c][min(q, PC_COLS - 1)], cta);
    ral[k] = cluster_map(&s_al[0][min(q, PC_COLS - 1)], cta);
    rbar[k] = cluster_map(s_bar, cta);
  }
  bool late = false;
  for (int p = 0; p < nref; ++p) {
    const int buf = p & 1;
    double2* xs = s_x[buf];
    {
      double2 s0 = make_double2(0, 0), s1 = s0;
#pragma unroll
      for (int u = 0; u < NR; u += 2) {
        s0 = cfmac(xs[8 * u + sl], P[u], s0);
        if (u + 1 < NR) s1 = cfmac(xs[8 * u + 8 + sl], P[u + 1], s1);
      }
      const double2 S = sum8(cadd(s0, s1));
      const uint32_t po = buf * (uint32_t)sizeof(s_part[0]), ao = buf * (uint32_t)sizeof(s_al[0]);
      if (q < nq) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
          if (sl + 8 * k < C) st_async16(rpart[k] + po, rbar[k] + 8 * buf, S);
      }
      if (c == 0) {   // row p of every column, held by the thread sl = p mod 8 at u = p / 8 (rows < 32: u < 4)
        const double2 v = (p >> 3) == 0 ? P[0] : ((p >> 3) == 1 ? P[1] : ((p >> 3) == 2 ? P[2] : P[3]));
        const double2 r = shfl2(v, (lane & 24) | (p & 7));
        if (q < nq) {
#pragma unroll
          for (int k = 0; k < 2; ++k)
            if (sl + 8 * k < C) st_async16(ral[k] + ao, rbar[k] + 8 * buf, r);
        }
      }
    }
    if ((tid >> 5) == PC_THREADS / 32 - 1) {   // the last warp holds no column: it forms T column by column
      if (p > 0) t_column(p - 1);
    } else if (!late) {
      late = !mbar_wait_cluster(bar + 8 * buf, (p >> 1) & 1);
    }
    if (tid == 0) mbar_expect(bar + 8 * buf, bytes);   // for column p + 2
    double2 S = make_double2(0, 0);
    if (q < nq) {
      if (sl < C) S = s_part[buf][sl][q];
      if (sl + 8 < C) S = cadd(S, s_part[buf][sl + 8][q]);
    }
    S = sum8(S);
    if ((tid >> 5) == (p >> 2)) {   // the warp that holds column p forms the scalars
      const double xn2 = __shfl_sync(0xffffffffu, S.x, 8 * (p & 3));
      const double2 al = s_al[buf][p];
      double2 kap;
      double beta, ib, rd;
      reflector_scalars(al, xn2, kap, beta, ib, rd);
      if (lane == 0) {
        const double2 u0 = make_double2(al.x - beta, al.y);
        s_sc[buf][0] = kap;
        s_sc[buf][1] = make_double2(beta, 0.0);
        s_sc[buf][2] = cscale(cconj(u0), rd);
        s_tau[p] = cscale(u0, -ib);
        if (c == 0) xs[p] = u0;
      }
    }
    __syncthreads();
    const double2 kap = s_sc[buf][0], scal = s_sc[buf][2];
    const double beta = s_sc[buf][1].x;
    // w_q = S_q + conj(u_p) P_pq
    const double2 al = s_al[buf][p];
    const double2 w = q < nq ? cfmac(make_double2(al.x - beta, al.y), s_al[buf][q], S) : S;
    if (panel && q > p) {
      const double2 cw = cmulc(kap, w);
#pragma unroll
      for (int u = 0; u < NR; ++u) P[u] = cfms(xs[8 * u + sl], cw, P[u]);
      if (q == p + 1 && q < nref) post(q);
    } else if (q == p) {
#pragma unroll
      for (int u = 0; u < NR; ++u) {
        const int i = 8 * u + sl;
        if (c > 0 || i > p) P[u] = cmul(P[u], scal);
        else if (i == p) P[u] = make_double2(beta, 0.0);
      }
    } else if (sl == 0) {
      const double2 e = cmul(scal, cconj(w));
      if (panel) s_G[q + p * BW] = e;                 // v_q^H v_p, q < p
      else if (vel) s_y[p + (q - BW) * BW] = e;       // (V^T g)_p
    }
    __syncthreads();
  }
  if (late) atomicExch(a.err, 1);
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // waited for at the end
  if ((tid >> 5) == PC_THREADS / 32 - 1) t_column(nref - 1);
  // write back: A keeps R (rows <= k0+q) and v below; Vp and Vs get V with its unit and zeros
  if (panel) {
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      const int i = 8 * u + sl;
      double2 v = P[u];
      if (q >= nref || (c == 0 && i < q)) v = make_double2(0, 0);
      else if (c == 0 && i == q) v = make_double2(1.0, 0.0);
      Vs[q * VS + i] = v;
      if (i < nr) {
        a.A[(rbeg + i) + (long long)(a.j0 + q) * N] = P[u];
        a.Vp[(rbeg + i) + (long long)q * N] = v;
      }
    }
  }
  __syncthreads();
  if (c == 0)
    for (int e = tid; e < BW * BW; e += PC_THREADS) a.Tout[e] = s_T[e];
  // g <- g - conj(V) T^T (V^T g)
  for (int e = tid; e < BW * ng; e += PC_THREADS) {
    const int j = e % BW, al = e / BW;
    double2 t = make_double2(0, 0);
    for (int i = 0; i <= j; ++i) t = cfma(s_T[i + j * BW], s_y[i + al * BW], t);
    s_z[e] = t;
  }
  __syncthreads();
  for (int e = tid; e < nr * ng; e += PC_THREADS) {
    const int i = e % nr, al = e / nr;
    double2 t0 = make_double2(0, 0), t1 = t0;
#pragma unroll 4
    for (int k = 0; k < BW; k += 2) {
      t0 = cfmac(Vs[k * VS + i], s_z[k + al * BW], t0);
      t1 = cfmac(Vs[(k + 1) * VS + i], s_z[k + 1 + al * BW], t1);
    }
    double2* gp = a.g + (long long)al * N + rbeg + i;
    *gp = csub(*gp, cadd(t0, t1));
  }
  // no CTA leaves while another may still write to it (after a wait that ran out)
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}


// D += A B with A 16x16 (a_i: row gq + 8*(i%2), k = tq + 4*(i/2)) and B 16x8 (b_j: k = tq + 4*j,
// column gq): FP64 tensor-core MMA.
__device__ __forceinline__ void dmma16(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]), "d"(b[1]),
        "d"(b[2]), "d"(b[3]));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  const unsigned sh = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sh), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N_>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N_) : "memory"); }

// X = A22 V, A22 Hermitian (lower triangle of A from row/column k0), V = Vp (32 columns).
// CTA (I, s): the 64 rows I of X, column blocks J of A22 in split s, K staged in chunks of 32
// through a two-stage cp.async ring.  The A operand of chunk (J, kc) is A[I, J] (J < I, staged
// k-major), conj(A[J, I])^T (J > I, staged row-major, conjugated when the fragment is built) or
// the diagonal tile (J = I, each element from the stored triangle, the mirrored ones conjugated and the
// diagonal made real when the fragment is built).  Complex products as real MMAs with the real and
// imaginary parts concatenated along k: X_re = [Ar | Ai] [Vr; -Vi], X_im = [Ar | Ai] [Vi; Vr].
// Warp (wr, wc): rows 16 wr .. +16, columns 16 wc .. +16 (two 8-wide n blocks).
constexpr int HM_LDA = 66;   // sA[k][row], 64 rows + 2 (conflict-free fragment loads)
constexpr int HM_LDT = 36;   // sAT[row][k], 32 k + 4
constexpr int HM_LDV = 36;   // sV[col][k], 32 k + 4 (the staging writes along k and the fragment
                             // reads of 8 columns x 4 k both fall on distinct banks)
constexpr int HM_ABUF = 64 * HM_LDT;   // >= 32 * HM_LDA; union of the two A layouts
constexpr int HM_STAGE = HM_ABUF + 32 * HM_LDV;
constexpr size_t HM_SMEM = 2 * (size_t)HM_STAGE * sizeof(double2);

__global__ void __launch_bounds__(256, 2) k_hemm2(const double2* __restrict__ A, long long N, long long k0,
                                                  const double2* __restrict__ V, int nI, int chunkJ,
                                                  double2* __restrict__ Xpart) {
  extern __shared__ __align__(16) double2 hs[];
  const int I = blockIdx.x, sp = blockIdx.y;
  const int J0 = sp * chunkJ, J1 = min(J0 + chunkJ, nI);
  const long long m = N - k0;
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int wr = wp & 3, wc = wp >> 2, gq = lane >> 2, tq = lane & 3;
  const long long rI = k0 + (long long)I * 64;

  double accr[2][4], acci[2][4];
#pragma unroll
  for (int nb = 0; nb < 2; ++nb)
#pragma unroll
    for (int k = 0; k < 4; ++k) accr[nb][k] = acci[nb][k] = 0.0;
  const int nch = 2 * max(0, J1 - J0);

  auto stage = [&](int c, int buf) {
    const int J = J0 + (c >> 1), kc = (c & 1) * 32;
    double2* sA = hs + (size_t)buf * HM_STAGE;
    double2* sV = sA + HM_ABUF;
    const long long cJ = k0 + (long long)J * 64 + kc;   // first global index of the k range
    if (J < I) {
      for (int e = tid; e < 64 * 32; e += 256) {
        const int r = e & 63, k = e >> 6;
        const long long gr = rI + r, gc = cJ + k;
        const bool ok = gr < N && gc < N;
        cp_async16(sA + k * HM_LDA + r, ok ? A + gr + gc * N : A, ok);
      }
    } else if (J > I) {
      for (int e = tid; e < 64 * 32; e += 256) {
        const int k = e & 31, r = e >> 5;
        const long long gr = cJ + k, gc = rI + r;   // stored element A[gr, gc], gr > gc
        const bool ok = gr < N && gc < N;
        cp_async16(sA + r * HM_LDT + k, ok ? A + gr + gc * N : A, ok);
      }
    } else {
      for (int e = tid; e < 64 * 32; e += 256) {
        const int r = e & 63, k = e >> 6;
        const long long lo = max(rI + r, cJ + k), hi = min(rI + r, cJ + k);
        const bool ok = lo < N;
        cp_async16(sA + k * HM_LDA + r, ok ? A + lo + hi * N : A, ok);
      }
    }
    for (int e = tid; e < 32 * 32; e += 256) {
      const int k = e & 31, col = e >> 5;
      const long long gr = cJ + k;
      const bool ok = gr < N;
      cp_async16(sV + col * HM_LDV + k, ok ? V + gr + (long long)col * N : V, ok);
    }
    cp_async_commit();
  };

  if (nch > 0) stage(0, 0);
  if (nch > 1) stage(1, 1);
  for (int c = 0; c < nch; ++c) {
    if (c + 1 < nch) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncthreads();
    const double2* sA = hs + (size_t)(c & 1) * HM_STAGE;
    const double2* sV = sA + HM_ABUF;
    const bool tr = (J0 + (c >> 1)) > I, dg = (J0 + (c >> 1)) == I;
    const int r0 = wr * 16 + gq, r1 = r0 + 8, kc = (c & 1) * 32;
#pragma unroll
    for (int kk = 0; kk < 32; kk += 8) {
      const int ka = kk + tq, kb = ka + 4;
      double2 x00, x10, x01, x11;
      if (tr) {
        x00 = cconj(sA[r0 * HM_LDT + ka]);
        x10 = cconj(sA[r1 * HM_LDT + ka]);
        x01 = cconj(sA[r0 * HM_LDT + kb]);
        x11 = cconj(sA[r1 * HM_LDT + kb]);
      } else {
        x00 = sA[ka * HM_LDA + r0];
        x10 = sA[ka * HM_LDA + r1];
        x01 = sA[kb * HM_LDA + r0];
        x11 = sA[kb * HM_LDA + r1];
        if (dg) {
          auto herm = [](double2& x, int d) { x.y = d > 0 ? x.y : (d < 0 ? -x.y : 0.0); };   // d = row - column
          herm(x00, r0 - kc - ka);
          herm(x10, r1 - kc - ka);
          herm(x01, r0 - kc - kb);
          herm(x11, r1 - kc - kb);
        }
      }
      const double a[8] = {x00.x, x10.x, x01.x, x11.x, x00.y, x10.y, x01.y, x11.y};
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        const int col = wc * 16 + nb * 8 + gq;
        const double2 v0 = sV[col * HM_LDV + ka], v1 = sV[col * HM_LDV + kb];
        const double bre[4] = {v0.x, v1.x, -v0.y, -v1.y};
        const double bim[4] = {v0.y, v1.y, v0.x, v1.x};
        dmma16(accr[nb], a, bre);
        dmma16(acci[nb], a, bim);
      }
    }
    __syncthreads();
    if (c + 2 < nch) stage(c + 2, c & 1);
  }
#pragma unroll
  for (int nb = 0; nb < 2; ++nb)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long row = rI + wr * 16 + gq + ((k >> 1) ? 8 : 0);
      const int col = wc * 16 + nb * 8 + 2 * tq + (k & 1);
      if (row < N) Xpart[((size_t)sp * 32 + col) * (size_t)m + (size_t)(row - k0)] = make_double2(accr[nb][k], acci[nb][k]);
    }
}

// W of a panel from X = A22 V (split partials): one cooperative launch for what needs the whole column range
// three times over.  With C1 = Wacc^H V, C2 = Vacc^H V for the pending updates of the look-ahead group (K = 32 KB
// columns), B = V^H X - C2^H C1 - C1^H C2 and Z = T^H B:
//   W = (X - Vacc C1 - Wacc C2 - 1/2 V Z) T.
// A share is the 16-row tiles b, b + shares, ... and CTA c takes the shares c, c + G, ... (one, but where several
// Q points run side by side).  (1) sums the split partials and takes the share of V^H X, C1 and C2;
// (2) after a grid barrier the shares are summed, 32 entries a CTA, in a fixed order; (3, K > 0) after another the
// 1024 entries of B, a warp each; (4) after the last W.  All products on the FP64 MMA; 16 rows so that up to
// nsm * 16 rows run side by side.  The work itself is 1 to 7 us of FP64 an SM; as seven launches with their tails,
// on 64-row blocks and with one CTA summing all shares, it took 76 us a panel at N = 2304,
// as one 31 (whole stage 1: N = 576 3.04 -> 2.40 ms, 2304 16.6 -> 13.4, 3600 34.9 -> 29.8, 8100 179 -> 167).
constexpr int WF_TR = 16;
constexpr int WF_LT = 20;    // row tiles [col][row], 16 rows + 4
constexpr int WF_LS = 36;    // 32 x 32 matrices [col][row]
constexpr size_t wf_smem(int KB) {
  return (size_t)((64 * KB + 64) * WF_LT + 32 * (64 * KB + 36) + 32 * WF_LS + 32 * WF_TR) * sizeof(double2);
}
struct WfArgs {
  double2* X;            // [S][32][m] split partials; slot 0 takes their sum
  int S;
  long long N, k0;
  const double2 *V, *T, *Vacc, *Wacc;
  double2* W;
  int shares;            // partial sums: one per CTA of a full device, so the sums do not depend on the grid
  double2* part;         // [shares][1 + 2 KB][32 x 32]
  double2* red;          // [1 + 2 KB][32 x 32], then B
  unsigned int* cnt;     // this launch's grid-barrier counter (zero at launch)
  int* err;
};
// c += a b for a 16 x 8 (complex) fragment a = (x00 x01; x10 x11) and b = (v0; v1): see dmma16
__device__ __forceinline__ void cmma(double (&cr)[4], double (&ci)[4], double2 x00, double2 x10, double2 x01, double2 x11,
                                     double2 v0, double2 v1) {
  const double a[8] = {x00.x, x10.x, x01.x, x11.x, x00.y, x10.y, x01.y, x11.y};
  const double bre[4] = {v0.x, v1.x, -v0.y, -v1.y};
  const double bim[4] = {v0.y, v1.y, v0.x, v1.x};
  dmma16(cr, a, bre);
  dmma16(ci, a, bim);
}

template <int KB>
__global__ void __launch_bounds__(256, 1) k_wfuse(WfArgs a) {
  constexpr int K = 32 * KB, NB = 1 + 2 * KB, LDC = 2 * K + 36;
  extern __shared__ __align__(16) double2 wsm[];
  double2* sL = wsm;                        // [Vacc | Wacc | V][WF_LT]
  double2* sV = sL + (size_t)2 * K * WF_LT;
  double2* sX = sV + 32 * WF_LT;
  double2* sC = sX + 32 * WF_LT;            // [col][C1; C2; Z / 2]
  double2* sT = sC + 32 * LDC;
  double2* sP = sT + 32 * WF_LS;            // [col][row] half sums
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int G = gridDim.x, bid = blockIdx.x;
  const long long m = a.N - a.k0;
  const int ntile = (int)((m + WF_TR - 1) / WF_TR);
  auto load_tile = [&](long long r0) {
    for (int e = tid; e < (2 * K + 32) * WF_TR; e += 256) {
      const int r = e % WF_TR, q = e / WF_TR;
      const double2* src = q < K ? a.Vacc + (long long)q * a.N : (q < 2 * K ? a.Wacc + (long long)(q - K) * a.N
                                                                            : a.V + (long long)(q - 2 * K) * a.N);
      sL[q * WF_LT + r] = r0 + r < m ? src[a.k0 + r0 + r] : make_double2(0, 0);
    }
  };
  // (1)
  for (int sh = bid; sh < a.shares; sh += G) {
    const int ih = (wp & 1) * 16, col = (wp >> 1) * 8 + gq;
    double cr[NB][4], ci[NB][4];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int k = 0; k < 4; ++k) cr[b][k] = ci[b][k] = 0.0;
    for (int t = sh; t < ntile; t += a.shares) {
      const long long r0 = (long long)t * WF_TR;
      __syncthreads();
      for (int e = tid; e < 32 * WF_TR; e += 256) {
        const int r = e % WF_TR, c = e / WF_TR;
        double2 x = make_double2(0, 0);
        if (r0 + r < m) {
          double2 xp[8];
#pragma unroll
          for (int s = 0; s < 8; ++s)
            xp[s] = (s < a.S) ? a.X[((size_t)s * 32 + c) * (size_t)m + r0 + r] : make_double2(0, 0);
#pragma unroll
          for (int s = 0; s < 8; ++s)
            if (s < a.S) x = cadd(x, xp[s]);
          a.X[(size_t)c * m + r0 + r] = x;
        }
        sX[c * WF_LT + r] = x;
      }
      load_tile(r0);
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < WF_TR; kk += 8) {
        const int ka = kk + tq, kb = ka + 4;
        const double2 v0 = sV[col * WF_LT + ka], v1 = sV[col * WF_LT + kb];
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          // left operand, conjugate transposed: V, then Wacc (C1), then Vacc (C2)
          const double2* L = b == 0 ? sV : (b <= KB ? sL + (K + 32 * (b - 1)) * WF_LT : sL + 32 * (b - 1 - KB) * WF_LT);
          const double2 x00 = cconj(L[(ih + gq) * WF_LT + ka]), x10 = cconj(L[(ih + gq + 8) * WF_LT + ka]);
          const double2 x01 = cconj(L[(ih + gq) * WF_LT + kb]), x11 = cconj(L[(ih + gq + 8) * WF_LT + kb]);
          if (b == 0) cmma(cr[b], ci[b], x00, x10, x01, x11, sX[col * WF_LT + ka], sX[col * WF_LT + kb]);
          else cmma(cr[b], ci[b], x00, x10, x01, x11, v0, v1);
        }
      }
    }
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        a.part[((size_t)sh * NB + b) * 1024 + ih + gq + 8 * (k >> 1) + 32 * ((wp >> 1) * 8 + 2 * tq + (k & 1))] =
            make_double2(cr[b][k], ci[b][k]);
  }
  if (!grid_sync(a.cnt, G, a.err)) return;
  // (2)
  for (int g = bid; g < 32 * NB; g += G) {
    const double2* p = a.part + (size_t)g * 32 + lane;
    double2 t = make_double2(0, 0);
    for (int b0 = wp; b0 < a.shares; b0 += 64) {
      double2 pv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) pv[u] = (b0 + 8 * u < a.shares) ? ldcg2(p + (size_t)(b0 + 8 * u) * NB * 1024) : make_double2(0, 0);
#pragma unroll
      for (int u = 0; u < 8; ++u) t = cadd(t, pv[u]);
    }
    sP[wp * 32 + lane] = t;
    __syncthreads();
    if (wp == 0) {
#pragma unroll
      for (int u = 1; u < 8; ++u) t = cadd(t, sP[u * 32 + lane]);
      a.red[g * 32 + lane] = t;
    }
    __syncthreads();
  }
  if (!grid_sync(a.cnt, 2 * G, a.err)) return;
  // (3)
  const double2* B = a.red;
  if constexpr (KB > 0) {
    for (int o = bid * 8 + wp; o < 1024; o += G * 8) {
      const int i = o & 31, j = o >> 5;
      double2 t = make_double2(0, 0);
#pragma unroll
      for (int b = 0; b < KB; ++b) {
        const double2* c1 = a.red + (1 + b) * 1024 + lane;
        const double2* c2 = a.red + (1 + KB + b) * 1024 + lane;
        t = cadd(t, cmulc(ldcg2(c2 + 32 * i), ldcg2(c1 + 32 * j)));
        t = cadd(t, cmulc(ldcg2(c1 + 32 * i), ldcg2(c2 + 32 * j)));
      }
      t = warp_sum2(t);
      if (lane == 0) a.red[NB * 1024 + o] = csub(ldcg2(a.red + o), t);
    }
    if (!grid_sync(a.cnt, 3 * G, a.err)) return;
    B = a.red + NB * 1024;
  }
  // (4) T, B (over the row tiles, which come later), C1, C2; Z / 2 = T^H B / 2
  for (int e = tid; e < 1024; e += 256) {
    const int i = e & 31, j = e >> 5;
    sT[j * WF_LS + i] = i <= j ? a.T[e] : make_double2(0, 0);
    sL[j * WF_LS + i] = ldcg2(B + e);
  }
  for (int e = tid; e < 2 * K * 32; e += 256) {
    const int b = e >> 10, i = e & 31, j = (e >> 5) & 31;
    sC[j * LDC + 32 * b + i] = ldcg2(a.red + 1024 + e);
  }
  __syncthreads();
  {
    const int ih = (wp & 1) * 16, cb = (wp >> 1) * 8;
    double zr[4] = {0, 0, 0, 0}, zi[4] = {0, 0, 0, 0};
#pragma unroll
    for (int kk = 0; kk < 32; kk += 8) {
      const int ka = kk + tq, kb = ka + 4;
      cmma(zr, zi, cconj(sT[(ih + gq) * WF_LS + ka]), cconj(sT[(ih + gq + 8) * WF_LS + ka]),
           cconj(sT[(ih + gq) * WF_LS + kb]), cconj(sT[(ih + gq + 8) * WF_LS + kb]), sL[(cb + gq) * WF_LS + ka],
           sL[(cb + gq) * WF_LS + kb]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      sC[(cb + 2 * tq + (k & 1)) * LDC + 2 * K + ih + gq + 8 * (k >> 1)] = make_double2(0.5 * zr[k], 0.5 * zi[k]);
  }
  const int cb = (wp & 3) * 8, kh = wp >> 2;
  for (int sh = bid; sh < a.shares; sh += G)
  for (int t = sh; t < ntile; t += a.shares) {
    const long long r0 = (long long)t * WF_TR;
    __syncthreads();
    load_tile(r0);
    for (int e = tid; e < 32 * WF_TR; e += 256) {
      const int r = e % WF_TR, c = e / WF_TR;
      sX[c * WF_LT + r] = r0 + r < m ? a.X[(size_t)c * m + r0 + r] : make_double2(0, 0);
    }
    __syncthreads();
    double cr[4] = {0, 0, 0, 0}, ci[4] = {0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < (2 * K + 32) / 16; ++q) {
      const int ka = 8 * (2 * q + kh) + tq, kb = ka + 4;
      cmma(cr, ci, sL[ka * WF_LT + gq], sL[ka * WF_LT + gq + 8], sL[kb * WF_LT + gq], sL[kb * WF_LT + gq + 8],
           sC[(cb + gq) * LDC + ka], sC[(cb + gq) * LDC + kb]);
    }
    auto at = [&](int k) { return (cb + 2 * tq + (k & 1)) * WF_TR + gq + 8 * (k >> 1); };
    if (kh == 1) {
#pragma unroll
      for (int k = 0; k < 4; ++k) sP[at(k)] = make_double2(cr[k], ci[k]);
    }
    __syncthreads();
    if (kh == 0) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = (cb + 2 * tq + (k & 1)) * WF_LT + gq + 8 * (k >> 1);
        sX[i] = csub(sX[i], cadd(make_double2(cr[k], ci[k]), sP[at(k)]));
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) cr[k] = ci[k] = 0.0;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int ka = 8 * (2 * q + kh) + tq, kb = ka + 4;
      cmma(cr, ci, sX[ka * WF_LT + gq], sX[ka * WF_LT + gq + 8], sX[kb * WF_LT + gq], sX[kb * WF_LT + gq + 8],
           sT[(cb + gq) * WF_LS + ka], sT[(cb + gq) * WF_LS + kb]);
    }
    if (kh == 1) {
#pragma unroll
      for (int k = 0; k < 4; ++k) sP[at(k)] = make_double2(cr[k], ci[k]);
    }
    __syncthreads();
    if (kh == 0) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const long long r = r0 + gq + 8 * (k >> 1);
        if (r < m) a.W[a.k0 + r + (long long)(cb + 2 * tq + (k & 1)) * a.N] = cadd(make_double2(cr[k], ci[k]), sP[at(k)]);
      }
    }
  }
}

// Look-ahead group of panels.  Vacc, Wacc hold the group's V and W side by side (32 columns per
// panel, leading dimension N); K = 32 * (panels already factored in the group).

// Strip of the next panel: columns c in [c0, c0+32), rows r >= c, get the pending updates of the
// group's earlier panels, A[r,c] -= sum_{q<K} V[r,q] conj(W[c,q]) + W[r,q] conj(V[c,q]).
// One warp per row (lane = column); the column rows of V and W in shared memory.
__global__ void __launch_bounds__(256) k_strip_update(double2* __restrict__ A, long long N, long long c0, int K,
                                                      const double2* __restrict__ V, const double2* __restrict__ W) {
  // sVc, sWc [K][32]: the strip's column rows; sVr, sWr [K][33]: this CTA's 32 rows (coalesced
  // loads); thread (lane = row, warp w) takes the columns w + 8v; sums in the order as before
  extern __shared__ __align__(16) double2 ssm[];
  double2* sVc = ssm;
  double2* sWc = ssm + (size_t)K * 32;
  double2* sVr = sWc + (size_t)K * 32;
  double2* sWr = sVr + (size_t)K * 33;
  const long long rb = c0 + (long long)blockIdx.x * 32;
  for (int e = threadIdx.x; e < K * 32; e += 256) {
    const int q = e >> 5, c = e & 31;
    const long long rc = c0 + c, rr = rb + c;
    sVc[e] = rc < N ? V[rc + (long long)q * N] : make_double2(0, 0);
    sWc[e] = rc < N ? W[rc + (long long)q * N] : make_double2(0, 0);
    sVr[q * 33 + c] = rr < N ? V[rr + (long long)q * N] : make_double2(0, 0);
    sWr[q * 33 + c] = rr < N ? W[rr + (long long)q * N] : make_double2(0, 0);
  }
  __syncthreads();
  const int u = threadIdx.x & 31, cg = threadIdx.x >> 5;
  const long long r = rb + u;
  if (r >= N) return;
  double2 t0[4], t1[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) t0[v] = t1[v] = make_double2(0, 0);
  for (int q = 0; q < K; q += 2) {
    const double2 v0 = sVr[q * 33 + u], w0 = sWr[q * 33 + u], v1 = sVr[(q + 1) * 33 + u], w1 = sWr[(q + 1) * 33 + u];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int c = cg + 8 * v;
      t0[v] = cadd(t0[v], cadd(cmulc(sWc[q * 32 + c], v0), cmulc(sVc[q * 32 + c], w0)));
      t1[v] = cadd(t1[v], cadd(cmulc(sWc[(q + 1) * 32 + c], v1), cmulc(sVc[(q + 1) * 32 + c], w1)));
    }
  }
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const int c = cg + 8 * v;
    if (c0 + c >= N || r < c0 + c) continue;
    const long long idx = r + (c0 + c) * N;
    double2 a = csub(A[idx], cadd(t0[v], t1[v]));
    if (r == c0 + c) a.y = 0.0;
    A[idx] = a;
  }
}

// ----------------------------------------------------------------------------- stage 2
// Band storage: column j holds A[j + o, j] for o = 0 .. LDB-1 (the band, o <= b, and the bulges,
// o <= 2b - 1).  Entries past row N are zero and stay zero, and AB_PAD zero columns follow column
// N-1, so that the chase reads whole blocks at the end of the matrix without masks.
constexpr int LDB = 2 * BW;
constexpr int AB_PAD = 2 * BW;
constexpr int BG_WARPS = 4;                 // sweep workers per CTA
constexpr int BG_LD = BW + 1;               // padded row length of the per-warp work tiles
constexpr int BG_WARP_TILE = 3 * BW * BG_LD + 2 * BW;   // Bs, Ds, B1s, v, w (double2) per warp

__device__ __forceinline__ long long nsteps_of(long long N, long long s) { return (N - 1 - s + BW - 1) / BW; }
// sum_{u=1}^{U} ceil(u / b)
__device__ __host__ __forceinline__ long long ceil_sum(long long U) {
  if (U <= 0) return 0;
  const long long q = U / BW, r = U % BW;
  return BW * q * (q + 1) / 2 + r * (q + 1);
}
// index of the first reflector of sweep s in the flat tau2 array
__device__ __host__ __forceinline__ long long tau2_offset(long long N, long long s) {
  return ceil_sum(N - 1) - ceil_sum(N - 1 - s);
}

__global__ void __launch_bounds__(256) k_band_extract(const double2* __restrict__ A, long long N, double2* __restrict__ AB) {
  const long long j = blockIdx.x;
  for (int o = threadIdx.x; o < LDB; o += blockDim.x) {
    double2 v = make_double2(0, 0);
    if (o <= BW && j + o < N) v = A[(j + o) + j * N];   // zero in the padding columns j >= N
    if (o == 0) v.y = 0.0;
    AB[j * LDB + o] = v;
  }
}

struct BulgeArgs {
  double2* AB;
  long long N;
  double2* A;            // upper triangle: reflector vectors (sweep s in column N-1-s, rows 0..)
  double2* tau2;         // [tau2_offset(N, s) + t]
  double2* g;            // [ng][N]
  int ng;
  unsigned int* prog;    // [N] steps published per sweep
  int* err;
  int store;             // keep the reflectors for the eigenvector back-transform
  int nprob;             // independent bands chased in one launch (eigenvalues only when > 1)
  long long ab_stride;   // elements between consecutive bands in AB
  long long prog_stride; // entries between consecutive progress arrays
};

// One step of sweep s (warp-wide; lane i <-> row r0 + i of the step's blocks).  All the
// blocks the step reads (bulge block B_t, diagonal block D_t, block below B_{t+1}) are fetched
// at once with cp.async into the warp's shared tiles, so the step pays one L2 round trip; the
// dot products run with four independent partial sums per lane.
__device__ __forceinline__ void cpa16(double2* dst, const double2* src, bool valid) {
  const unsigned sh = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sh), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

__device__ void bulge_step(const BulgeArgs& a, long long s, long long t, double2* Bs, double2* Ds, double2* B1s,
                           double2* vs, double2* ws) {
  const int lane = threadIdx.x & 31;
  const long long N = a.N;
  double2* AB = a.AB;
  const long long r0 = s + 1 + t * BW;
  const int L = (int)min((long long)BW, N - r0);
  const long long c0 = r0 - BW;   // first column of the bulge block (t >= 1)
  const long long r1 = r0 + L;
  const int L1 = (r1 < N) ? (int)min((long long)BW, N - r1) : 0;
  // ---- fetch
  if (t > 0) {
#pragma unroll 8
    for (int q = 0; q < BW; ++q) cpa16(Bs + lane * BG_LD + q, AB + (c0 + q) * LDB + (BW + lane - q), lane < L);
  }
  for (int q = 0; q < L; ++q) {
    const bool ok = lane >= q && lane < L;
    cpa16(Ds + lane * BG_LD + q, ok ? AB + (r0 + q) * LDB + (lane - q) : AB, ok);
  }
  for (int q = 0; q < L; ++q) cpa16(B1s + lane * BG_LD + q, AB + (r0 + q) * LDB + (L + lane - q), lane < L1);
  asm volatile("cp.async.commit_group;" ::: "memory");
  double2 gv[NGMAX];
#pragma unroll
  for (int al2 = 0; al2 < NGMAX; ++al2)
    gv[al2] = (al2 < a.ng && lane < L) ? __ldcg(a.g + (long long)al2 * N + r0 + lane) : make_double2(0, 0);
  double2 x = make_double2(0, 0);
  if (t == 0 && lane < L) x = __ldcg(AB + s * LDB + 1 + lane);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  if (t > 0) x = Bs[lane * BG_LD];
  // ---- reflector (ZLARFG)
  double xn2 = (lane >= 1 && lane < L) ? x.x * x.x + x.y * x.y : 0.0;
  xn2 = warp_sum(xn2);
  const double2 al = make_double2(__shfl_sync(0xffffffffu, x.x, 0), __shfl_sync(0xffffffffu, x.y, 0));
  double2 tau, scal;
  double beta;
  if (xn2 == 0.0 && al.y == 0.0) {
    tau = make_double2(0, 0);
    scal = make_double2(0, 0);
    beta = al.x;
  } else {
    beta = -copysign(sqrt(al.x * al.x + al.y * al.y + xn2), al.x);
    tau = make_double2((beta - al.x) / beta, -al.y / beta);
    const double2 den = make_double2(al.x - beta, al.y);
    const double dd = den.x * den.x + den.y * den.y;
    scal = make_double2(den.x / dd, -den.y / dd);
  }
  const double2 v = (lane == 0) ? make_double2(1.0, 0.0) : (lane < L ? cmul(x, scal) : make_double2(0, 0));
  vs[lane] = v;
  // Hermitian fill of D (upper = conj of lower, real diagonal)
  if (lane < L)
    for (int q = 0; q <= lane; ++q) {
      double2 d = Ds[lane * BG_LD + q];
      if (q == lane) {
        d.y = 0.0;
        Ds[lane * BG_LD + q] = d;
      } else {
        Ds[q * BG_LD + lane] = cconj(d);
      }
    }
  __syncwarp();
  // ---- annihilated column and the left application to the rest of the bulge block
  if (lane < L) {
    const double2 nv = (lane == 0) ? make_double2(beta, 0.0) : make_double2(0, 0);
    if (t == 0) AB[s * LDB + 1 + lane] = nv;
    else AB[c0 * LDB + BW + lane] = nv;
  }
  if (t > 0) {
    if (lane >= 1) {   // w_q = sum_i conj(v_i) B(i, q), lane q
      double2 w0 = make_double2(0, 0), w1 = w0, w2 = w0, w3 = w0;
      for (int i = 0; i < L; i += 4) {
        w0 = cadd(w0, cmulc(vs[i], Bs[i * BG_LD + lane]));
        if (i + 1 < L) w1 = cadd(w1, cmulc(vs[i + 1], Bs[(i + 1) * BG_LD + lane]));
        if (i + 2 < L) w2 = cadd(w2, cmulc(vs[i + 2], Bs[(i + 2) * BG_LD + lane]));
        if (i + 3 < L) w3 = cadd(w3, cmulc(vs[i + 3], Bs[(i + 3) * BG_LD + lane]));
      }
      ws[lane] = cadd(cadd(w0, w1), cadd(w2, w3));
    }
    __syncwarp();
    if (lane < L) {
      const double2 cv = cmul(cconj(tau), v);
#pragma unroll 4
      for (int q = 1; q < BW; ++q)
        AB[(c0 + q) * LDB + (BW + lane - q)] = csub(Bs[lane * BG_LD + q], cmul(cv, ws[q]));
    }
    __syncwarp();
  }
  // ---- two-sided update of D: D <- H^H D H
  double2 y = make_double2(0, 0);
  if (lane < L) {
    double2 y1 = y, y2 = y, y3 = y;
    for (int q = 0; q < L; q += 4) {
      y = cadd(y, cmul(Ds[lane * BG_LD + q], vs[q]));
      if (q + 1 < L) y1 = cadd(y1, cmul(Ds[lane * BG_LD + q + 1], vs[q + 1]));
      if (q + 2 < L) y2 = cadd(y2, cmul(Ds[lane * BG_LD + q + 2], vs[q + 2]));
      if (q + 3 < L) y3 = cadd(y3, cmul(Ds[lane * BG_LD + q + 3], vs[q + 3]));
    }
    y = cadd(cadd(y, y1), cadd(y2, y3));
  }
  // v^H y (real for Hermitian D) and, interleaved, v^T g of the velocity vectors
  double pvx = cmulc(v, y).x;
  double2 sg[NGMAX];
#pragma unroll
  for (int al2 = 0; al2 < NGMAX; ++al2) sg[al2] = cmul(v, gv[al2]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    pvx += __shfl_xor_sync(0xffffffffu, pvx, o);
#pragma unroll
    for (int al2 = 0; al2 < NGMAX; ++al2) {
      if (al2 < a.ng) {
        sg[al2].x += __shfl_xor_sync(0xffffffffu, sg[al2].x, o);
        sg[al2].y += __shfl_xor_sync(0xffffffffu, sg[al2].y, o);
      }
    }
  }
  const double t2 = tau.x * tau.x + tau.y * tau.y;
  const double2 w = csub(cmul(tau, y), cscale(v, 0.5 * t2 * pvx));
  ws[lane] = w;
  __syncwarp();
  if (lane < L)
#pragma unroll 4
    for (int q = 0; q <= lane; ++q) {
      double2 d = csub(Ds[lane * BG_LD + q], cadd(cmulc(ws[q], v), cmulc(vs[q], w)));   // v_i conj(w_q) + w_i conj(v_q)
      if (q == lane) d.y = 0.0;
      AB[(r0 + q) * LDB + (lane - q)] = d;
    }
  // ---- right application to the block below: B1 <- B1 H
  if (L1 > 0) {
    double2 z = make_double2(0, 0);
    if (lane < L1) {
      double2 z1 = z, z2 = z, z3 = z;
      for (int q = 0; q < L; q += 4) {
        z = cadd(z, cmul(B1s[lane * BG_LD + q], vs[q]));
        if (q + 1 < L) z1 = cadd(z1, cmul(B1s[lane * BG_LD + q + 1], vs[q + 1]));
        if (q + 2 < L) z2 = cadd(z2, cmul(B1s[lane * BG_LD + q + 2], vs[q + 2]));
        if (q + 3 < L) z3 = cadd(z3, cmul(B1s[lane * BG_LD + q + 3], vs[q + 3]));
      }
      z = cadd(cadd(z, z1), cadd(z2, z3));
      const double2 tz = cmul(tau, z);
#pragma unroll 4
      for (int q = 0; q < L; ++q)
        AB[(r0 + q) * LDB + (L + lane - q)] = csub(B1s[lane * BG_LD + q], cmul(tz, cconj(vs[q])));
    }
  }
  // ---- velocity vectors: g <- g - tau conj(v) (v^T g)
  if (lane < L) {
    const double2 tcv = cmul(tau, cconj(v));
#pragma unroll
    for (int al2 = 0; al2 < NGMAX; ++al2)
      if (al2 < a.ng) a.g[(long long)al2 * N + r0 + lane] = csub(gv[al2], cmul(tcv, sg[al2]));
  }
  if (a.store) {
    if (lane < L) a.A[(r0 + lane - s - 1) + (N - 1 - s) * N] = v;
    if (lane == 0) a.tau2[tau2_offset(N, s) + t] = tau;
  }
  __syncwarp();
}

// Persistent bulge chasing: warp w of the grid runs sweeps w, w + W, w + 2W, ...; sweep s
// starts step t after sweep s-1 has published step t+2 (or finished): the elements of step t
// of sweep s have rows and columns <= s + 1 + (t+2) b, those of step t+3 of sweep s-1 rows
// >= s + (t+3) b + 1, so the two never touch the same element (nor the same rows of g).
__global__ void __launch_bounds__(32 * BG_WARPS, 1) k_bulge(BulgeArgs a) {
  extern __shared__ __align__(16) double2 bsm[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2* Bs = bsm + (size_t)wid * BG_WARP_TILE;
  double2* Ds = Bs + BW * BG_LD;
  double2* B1s = Ds + BW * BG_LD;
  double2* vs = B1s + BW * BG_LD;
  double2* ws = vs + BW;
  const long long W = (long long)gridDim.x * BG_WARPS;
  const long long N = a.N;
  const long long np = a.nprob;
  // sweep u of the launch = sweep s = u / np of band q = u % np: sweeps are taken in increasing
  // u, and a sweep waits only on sweep s-1 of its own band (index u - np), so every wait is on a
  // sweep that some resident warp has already started or finished
  for (long long u = (long long)blockIdx.x * BG_WARPS + wid; u < np * (N - 1); u += W) {
    const long long q = u % np, s = u / np;
    BulgeArgs b = a;
    b.AB = a.AB + q * a.ab_stride;
    unsigned int* prog = a.prog + q * a.prog_stride;
    const long long ns = nsteps_of(N, s);
    const long long nprev = (s > 0) ? nsteps_of(N, s - 1) : 0;
    for (long long t = 0; t < ns; ++t) {
      if (s > 0) {
        const unsigned int need = (unsigned int)min(t + 3, nprev);
        int bad = 0;
        if (lane == 0) bad = wait_at_least(prog + s - 1, need, a.err) ? 0 : 1;
        bad = __shfl_sync(0xffffffffu, bad, 0);
        if (bad) return;
      }
      bulge_step(b, s, t, Bs, Ds, B1s, vs, ws);
      // publish: the warp barrier orders the lanes' writes before lane 0's release store
      __syncwarp();
      if (lane == 0) st_release(prog + s, (unsigned int)(t + 1));
    }
  }
}

// Stage 2 with one CTA per sweep and specialised warps.  The launch is one dependency chain: sweep
// s may start step t once sweep s-1 has published step t+2, so it takes about N times (three
// steps + one hand-over between CTAs), and everything in a step that is not on the way from one
// reflector to the next is moved off that way:
//   * the reflector's vector is used unscaled: with u = x - beta e_0 the reflector is
//     H = I - kappa u u^H, kappa = -u_0 / (beta |u_0|^2), and every product D u, B1 u, u^H B is the
//     product with x minus beta times the first column (row), so the products of a step run beside
//     the scalars (a root, its reciprocal and one more reciprocal) instead of after them;
//   * the block below (B1) is the next step's bulge block (B): the four warps that update it keep it
//     in registers, so it is written once, after its second update.  Four groups of four warps take
//     turns: group n mod 4 does B1 of step n, then B of step n+1, then the diagonal block of step n+2,
//     so that the chain from x to x passes from group to group and waits for none of the rest;
//   * only the first column of B1 (the next x) is on the chain; it is updated first and announced,
//     and the rest of B1, the B update with its stores, the diagonal block and the velocity vectors
//     have their own warps and follow through mbarriers;
//   * one warp waits for the predecessor and copies the next blocks into a ring in shared memory,
//     one publishes finished steps, so no poll, no L2 round trip and no fence stalls the others.
// A step is bound by the latency of its instruction chain (2700 cycles from x to x; the FP64 pipe is
// busy 24 % of them), so index arithmetic is kept out of it: a warp holds 8 rows x 32 columns of a
// 32 x 32 block, lane -> rows i = 8 wg + ig + 4r (r < 2), columns c = qb + 8m (m < 4) with ig = lane & 3,
// qb = 4 (bit 2) + (lane >> 3), and an element's place in the band, 63 c + i from its block's corner, is
// one lane offset plus the constant 504 m + 4 r; the sums over the columns (B1, D) stay within one
// warp, and the shared-memory accesses are free of bank conflicts.
// Measured (whole stage, five velocity vectors): N = 576 4.3 ms, 2304 19.2 ms, 8100 85 ms, 14400 178 ms;
// with one CTA of four warps per sweep and CTA barriers between the parts of a step it was 10.9, 46.7,
// 169 and 309 ms.  Tried: bulk copies instead of cp.async (longer latency, 19.5 ms at 2304), blocks
// loaded from L2 into a second set of registers (spills, 24 ms), two groups that swap B1 and B (21 ms).
constexpr int CH_NS = 4;    // ring slots: steps the groups may be apart
constexpr int CH_NX = 8;    // steps of x and scalars kept (more than CH_NS + 2)
constexpr int CH_WARPS = 19;   // 4 x 4 block warps, velocity, producer, publisher (104 registers a thread)
constexpr int CH_THREADS = 32 * CH_WARPS;
constexpr int CH_BLK = BW * LDB;                      // one block of 32 band columns
constexpr int CH_SLOT = CH_BLK + LDB + NGMAX * BW;    // + column s (first step), velocity rows
constexpr size_t CH_SMEM = (size_t)CH_NS * CH_SLOT * sizeof(double2);

// named barriers of whole warps: bar is an aligned instruction, so the warp's lanes are brought
// together first (they may have left a wait or a lane branch one by one)
__device__ __forceinline__ void bar_sync(int id, int cnt) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(cnt) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int cnt) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(cnt) : "memory");
}
// bounded wait for a phase of an mbarrier; the clock is read every 64 polls (a read takes longer than
// most waits)
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t a, uint32_t parity) {
  unsigned int spins = 0;
  unsigned long long t0 = 0;
  while (!tc::mbar_try(a, parity)) {
    if ((++spins & 63u) == 0u) {
      if (t0 == 0) t0 = globaltimer();
      if (globaltimer() - t0 > kWaitNs) return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool mbar_test(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
               : "=r"(ok)
               : "r"(a), "r"(parity)
               : "memory");
  return ok != 0;
}

__global__ void __launch_bounds__(CH_THREADS, 1) k_chase(BulgeArgs a) {
  extern __shared__ __align__(128) double2 ring[];
  // full: a step's blocks are in its ring slot; empty: every reader has taken them (each arrives after
  // its wait for full, so the phases stay in step); xr: x of a step is in s_x (4 arrivals); sr: its
  // scalars are in s_sc; done: every store of a step has been issued
  __shared__ __align__(8) uint64_t s_full[CH_NS], s_empty[CH_NS], s_done[CH_NX], s_xr[CH_NX], s_sr[CH_NX];
  __shared__ __align__(16) double2 s_x[CH_NX][BW];
  __shared__ __align__(16) double s_np[CH_NX][4];    // partial |x_i|^2, i >= 1
  __shared__ __align__(16) double2 s_sc[CH_NX][2];   // kappa, (beta, 1/beta)
  __shared__ double s_rd[CH_NX];                     // 1/|u_0|^2
  __shared__ double2 s_pw[4][4][BW], s_b0[4][BW];    // per group: partial x^H B, first row of B
  __shared__ double2 s_wv[16][BW];                   // per warp: w of the B and D updates
  __shared__ double2 s_y[4][BW], s_d0[4][BW];        // by step mod 4: D x, first column of D
  // the warp's index as a value that is uniform by construction, and (below) waits that end by a vote:
  // where the compiler can see that a warp is together, a shuffle is one instruction, else a guarded one
  const int lane = threadIdx.x & 31, wid = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int N = (int)a.N;
  const long long np = a.nprob;
  if (threadIdx.x == 0) {
    for (int k = 0; k < CH_NS; ++k) {
      tc::mbar_init(tc::smem_u32(&s_full[k]), 32);    // the producer's lanes
      tc::mbar_init(tc::smem_u32(&s_empty[k]), 10);   // B1 4, D 4, velocity, publisher
    }
    for (int k = 0; k < CH_NX; ++k) {
      tc::mbar_init(tc::smem_u32(&s_done[k]), 9);     // B 4, D 4, velocity
      tc::mbar_init(tc::smem_u32(&s_xr[k]), 4);
      tc::mbar_init(tc::smem_u32(&s_sr[k]), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  static_assert((CH_NS & (CH_NS - 1)) == 0 && (CH_NX & (CH_NX - 1)) == 0, "ring sizes are powers of two");
  // Every wait is bounded.  A wait on another sweep that runs out sets *err, after which this CTA
  // goes on without waiting for its predecessors (indices stay in range, the results are void); the
  // copies it issues always complete, so the waits inside the CTA end as well.
  auto wait_bar = [&](uint64_t* b, int cnt, int n) {
    if (!mbar_wait_bounded(tc::smem_u32(b + (n & (cnt - 1))), (unsigned)(n / cnt) & 1u)) atomicExch(a.err, 1);
  };
  // the same by all lanes of a warp, which leave together
  auto wait_warp = [&](uint64_t* b, int cnt, int n) {
    const uint32_t bar = tc::smem_u32(b + (n & (cnt - 1))), par = (unsigned)(n / cnt) & 1u;
    unsigned int spins = 0;
    unsigned long long t0 = 0;
    while (!__all_sync(0xffffffffu, tc::mbar_try(bar, par))) {
      if ((++spins & 63u) == 0u) {
        const unsigned long long now = globaltimer();
        if (t0 == 0) t0 = now;
        if (__any_sync(0xffffffffu, now - t0 > kWaitNs)) {
          if (lane == 0) atomicExch(a.err, 1);
          break;
        }
      }
    }
  };
  auto arrive = [&](uint64_t* b, int cnt, int n) {
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(tc::smem_u32(b + (n & (cnt - 1))));
  };
  const int grp = wid >> 2, wg = wid & 3;
  int ig = lane & 3, qb = 4 * ((lane >> 2) & 1) + (lane >> 3);
  int i0 = 8 * wg + ig;
  asm("" : "+r"(qb), "+r"(i0));   // opaque: the compiler folded the tests i >= c below wrongly from the bit ranges
  const int lb = (LDB - 1) * qb + i0;   // lane offset of a block's elements; element (r, m) at lb + EM m + 4 r
  constexpr int EM = 8 * (LDB - 1);
  int n = 0;   // steps of this CTA so far
  // sweep u of the launch = sweep s = u / np of band u % np: a sweep waits only on sweep s-1 of its
  // own band, which has a smaller u and is running or finished.  Each role loops by itself (one loop
  // around the roles would keep the block warps' registers alive in all of them).
  auto sweeps = [&](auto&& body) {
    for (long long u = blockIdx.x; u < np * (N - 1); u += gridDim.x) {
      const int q = (int)(u % np), s = (int)(u / np);
      body(a.AB + q * a.ab_stride, a.prog + q * a.prog_stride, s, (int)nsteps_of(N, s));
    }
  };
  if (wid == 17) {   // producer
    bool alone = false;   // a wait on a predecessor has failed
    sweeps([&](double2* AB, unsigned int* prog, int s, int ns) {
      const int nprev = (s > 0) ? (int)nsteps_of(N, s - 1) : 0;
      int seen = 0;
      const double2* src = AB + (long long)(s + 1) * LDB + lane;
      for (int t = 0; t < ns; ++t, ++n, src += CH_BLK) {
        if (n >= CH_NS) wait_bar(s_empty, CH_NS, n - CH_NS);
        const int need = min(t + 3, nprev);
        if (lane == 0 && s > 0 && seen < need && !alone) {
          alone = !wait_at_least(prog + s - 1, (unsigned)need, a.err);
          seen = (int)ld_acquire(prog + s - 1);
        }
        __syncwarp();
        const uint32_t dst = tc::smem_u32(ring + (n & (CH_NS - 1)) * CH_SLOT + lane);
        auto cp = [](uint32_t d, const double2* g) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(g) : "memory");
        };
        // column c: its block below (entries 32 - c .. 63 - c) is in its second half and, from 32 - c
        // on, its first; the diagonal block in its first
#pragma unroll
        for (int c = 0; c < BW; ++c) cp(dst + (c * LDB + BW) * 16, src + c * LDB + BW);
#pragma unroll
        for (int c = 0; c < BW; ++c) cp(dst + c * LDB * 16, src + c * LDB);
        if (t == 0) {
          cp(dst + CH_BLK * 16, AB + (long long)s * LDB + lane);
          if (lane == 0) cp(dst + (CH_BLK + BW) * 16, AB + (long long)s * LDB + BW);
        }
        const double2* gp = a.g + min(s + 1 + t * BW + lane, N - 1);
        for (int al = 0; al < a.ng; ++al, gp += N) cp(dst + (CH_BLK + LDB + al * BW) * 16, gp);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(&s_full[n & (CH_NS - 1)])) : "memory");
      }
    });
  } else if (wid == 18) {   // publisher: a step whose successor is finished too is left to that one
    sweeps([&](double2*, unsigned int* prog, int s, int ns) {
      if (lane == 0)
        for (int t = 0; t < ns; ++t, ++n) {
          tc::mbar_arrive(tc::smem_u32(&s_empty[n & (CH_NS - 1)]));
          wait_bar(s_done, CH_NX, n);
          if (t + 1 < ns && mbar_test(tc::smem_u32(&s_done[(n + 1) & (CH_NX - 1)]), (unsigned)((n + 1) / CH_NX) & 1u)) continue;
          st_release(prog + s, (unsigned int)(t + 1));
        }
    });
  } else if (grp == 4) {
    sweeps([&](double2*, unsigned int*, int s, int ns) {
      // velocity vectors g <- g - kappa conj(u) (u^T g), five at a time, and the stored reflector
      for (int t = 0; t < ns; ++t, ++n) {
        const int r0 = s + 1 + t * BW, L = min(BW, N - r0), xb = n & (CH_NX - 1);
        const double2* sl = ring + (n & (CH_NS - 1)) * CH_SLOT + CH_BLK + LDB + lane;
        wait_warp(s_full, CH_NS, n);
        wait_warp(s_sr, CH_NX, n);
        const double2 kap = s_sc[xb][0], bi = s_sc[xb][1];
        double2 uv = s_x[xb][lane];
        if (lane == 0) uv.x -= bi.x;
        const double2 ku = cmulc(uv, kap);
        double2* gp = a.g + r0 + lane;
        for (int j0 = 0; j0 < a.ng; j0 += 5, sl += 5 * BW) {
          double2 gv[5], p[5];
#pragma unroll
          for (int j = 0; j < 5; ++j) {
            gv[j] = lane < L ? sl[j * BW] : make_double2(0, 0);
            p[j] = cmul(uv, gv[j]);
          }
          // the five sums over the 32 rows: halves exchanged over lane bits 4, 3 and 2 (8 slots, 3 of
          // them empty), so that lane bits (4, 3, 2) = j end with sum j; then over bits 1 and 0
          const double2 z0 = make_double2(0, 0);
          const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
          const double2 e1 = shfl2_xor(p[1], 16), e2 = shfl2_xor(p[2], 16), e3 = shfl2_xor(p[3], 16);
          const double2 a0 = cadd(h4 ? p[4] : p[0], shfl2_xor(h4 ? p[0] : p[4], 16));
          const double2 a1 = h4 ? z0 : cadd(p[1], e1), a2 = h4 ? z0 : cadd(p[2], e2), a3 = h4 ? z0 : cadd(p[3], e3);
          const double2 b0 = cadd(h3 ? a2 : a0, shfl2_xor(h3 ? a0 : a2, 8));
          const double2 b1 = cadd(h3 ? a3 : a1, shfl2_xor(h3 ? a1 : a3, 8));
          double2 c = cadd(h2 ? b1 : b0, shfl2_xor(h2 ? b0 : b1, 4));
          c = cadd(c, shfl2_xor(c, 2));
          c = cadd(c, shfl2_xor(c, 1));
#pragma unroll
          for (int j = 0; j < 5; ++j, gp += N) {
            const double2 sg = shfl2(c, 4 * j);   // sum j sits in the lanes 4j .. 4j+3
            if (lane < L) *gp = cfms(ku, sg, gv[j]);
          }
        }
        arrive(s_empty, CH_NS, n);   // after the scalars: by then the first x has been read as well
        if (a.store) {
          // tau = -u_0 / beta, v = u / u_0
          const double2 u0 = make_double2(s_x[xb][0].x - bi.x, s_x[xb][0].y);
          double2 v = make_double2(lane == 0 ? 1.0 : 0.0, 0.0), tau = make_double2(0, 0);
          if (kap.x != 0.0 || kap.y != 0.0) {
            tau = cscale(u0, -bi.y);
            if (lane > 0) v = cscale(cmulc(u0, uv), s_rd[xb]);
          }
          if (lane < L) a.A[(r0 + lane - s - 1) + (long long)(N - 1 - s) * N] = v;
          if (lane == 0) a.tau2[tau2_offset(N, s) + t] = tau;
        }
        arrive(s_done, CH_NX, n);
      }
    });
  } else {
    double2 M[2][4] = {};
    const int ub = (LDB - 1) * i0 + qb;   // lane offset of D's mirrored elements: ub + 8 m + 4 (LDB - 1) r
    // z = M x over the warp's rows, the same in the 8 lanes of a row
    auto dot_rows = [&](const double2* x, double2(&z)[2]) {
      double2 xq[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) xq[m] = x[qb + 8 * m];
#pragma unroll
      for (int r = 0; r < 2; ++r)
        z[r] = cadd(cfma(M[r][1], xq[1], cmul(M[r][0], xq[0])), cfma(M[r][3], xq[3], cmul(M[r][2], xq[2])));
#pragma unroll
      for (int o = 4; o <= 16; o <<= 1)
#pragma unroll
        for (int r = 0; r < 2; ++r) z[r] = cadd(z[r], shfl2_xor(z[r], o));
    };
    // x of step n1 into s_x (lanes 0..3 of the group's warps: rows i0, i0 + 4), with its partial norm
    auto post_x = [&](int n1, double2 x0, double2 x1) {
      const int xn = n1 & (CH_NX - 1);
      double pn = fma(x1.x, x1.x, x1.y * x1.y);
      if (i0 > 0) pn = fma(x0.x, x0.x, fma(x0.y, x0.y, pn));
      pn += __shfl_xor_sync(0xffffffffu, pn, 1);
      pn += __shfl_xor_sync(0xffffffffu, pn, 2);
      if (lane < 4) {
        s_x[xn][i0] = x0;
        s_x[xn][i0 + 4] = x1;
      }
      if (lane == 0) s_np[xn][wg] = pn;
      bar_arrive(1 + (n1 & 1), 256);
      arrive(s_xr, CH_NX, n1);
    };
    sweeps([&](double2* AB, unsigned int*, int s, int ns) {
      for (int t = 0; t < ns; ++t, ++n) {
        const int r0 = s + 1 + t * BW, xb = n & (CH_NX - 1);
        const double2* sl = ring + (n & (CH_NS - 1)) * CH_SLOT;
        const int role = (n - grp) & 3;
        if (role == 0) {
          // ---- the block below, B1 <- B1 H
          wait_warp(s_full, CH_NS, n);
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int m = 0; m < 4; ++m) M[r][m] = sl[lb + BW + EM * m + 4 * r];
          arrive(s_empty, CH_NS, n);
          bar_sync(1 + (n & 1), 256);   // x
          double2 z[2], kap;
          double beta, ib, rd;
          const double2* xs = s_x[xb];
          const double* pn = s_np[xb];
          reflector_scalars(xs[0], (pn[0] + pn[1]) + (pn[2] + pn[3]), kap, beta, ib, rd);
          dot_rows(xs, z);
          // x is read again below rather than kept: registers
          asm volatile("" ::: "memory");
#pragma unroll
          for (int r = 0; r < 2; ++r) z[r] = cmul(kap, caxpy(-beta, shfl2(M[r][0], ig), z[r]));
          {
            double2 x0 = xs[qb];
            if (qb == 0) x0.x -= beta;
#pragma unroll
            for (int r = 0; r < 2; ++r) M[r][0] = cfmsc(x0, z[r], M[r][0]);
          }
          if (t + 1 < ns) post_x(n + 1, M[0][0], M[1][0]);
          if (wg == 0) {
            if (lane == 0) {
              s_sc[xb][0] = kap;
              s_sc[xb][1] = make_double2(beta, ib);
              s_rd[xb] = rd;
            }
            arrive(s_sr, CH_NX, n);
          }
          if (t + 1 < ns) {
#pragma unroll
            for (int m = 1; m < 4; ++m) {
              const double2 xm = xs[qb + 8 * m];
#pragma unroll
              for (int r = 0; r < 2; ++r) M[r][m] = cfmsc(xm, z[r], M[r][m]);
            }
            // partial x^H B of the next step: x of the own rows is column 0
            const double2 x0 = shfl2(M[0][0], ig), x1 = shfl2(M[1][0], ig);
            double2 p[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) p[m] = cfmac(x1, M[1][m], cmulc(x0, M[0][m]));
            // sums over the 4 lanes of a column group; lane (bit 0, bit 1) ends with m = 2 bit0 + bit1
            const bool b0 = lane & 1, b1 = lane & 2;
            double2 e0 = b0 ? p[2] : p[0], e1 = b0 ? p[3] : p[1];
            e0 = cadd(e0, shfl2_xor(b0 ? p[0] : p[2], 1));
            e1 = cadd(e1, shfl2_xor(b0 ? p[1] : p[3], 1));
            s_pw[grp][wg][qb + 16 * (lane & 1) + 4 * (lane & 2)] = cadd(b1 ? e1 : e0, shfl2_xor(b1 ? e0 : e1, 2));
            if (i0 == 0)
#pragma unroll
              for (int m = 0; m < 4; ++m) s_b0[grp][qb + 8 * m] = M[0][m];
          }
        } else if (role == 1) {
          const bool in0 = i0 < N - r0, in1 = i0 + 4 < N - r0;
          if (t > 0) {
            // ---- B <- H^H B, stored
            double2 xi[2];
            xi[0] = shfl2(M[0][0], ig);
            xi[1] = shfl2(M[1][0], ig);
            bar_sync(3 + grp, 128);   // s_pw, s_b0
            const double2(*pw)[BW] = s_pw[grp];
            const double2 w = cadd(cadd(pw[0][lane], pw[1][lane]), cadd(pw[2][lane], pw[3][lane]));
            const double2 br = s_b0[grp][lane];
            double2* dst = AB + (long long)(r0 - BW) * LDB + lb + BW;
            wait_warp(s_sr, CH_NX, n);
            const double beta = s_sc[xb][1].x;
            double2* wv = s_wv[wid];
            wv[lane] = cmulc(s_sc[xb][0], caxpy(-beta, br, w));
            __syncwarp();
            if (i0 == 0) xi[0].x -= beta;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              const double2 cw = wv[qb + 8 * m];
              double2 v0 = cfms(xi[0], cw, M[0][m]), v1 = cfms(xi[1], cw, M[1][m]);
              if (m == 0 && qb == 0) {   // the annihilated column
                v0 = make_double2(i0 == 0 ? beta : 0.0, 0.0);
                v1 = make_double2(0.0, 0.0);
              }
              if (in0) dst[EM * m] = v0;
              if (in1) dst[EM * m + 4] = v1;
            }
          } else {
            // first step: x is column s below its diagonal, which becomes (beta, 0, ..., 0)
            wait_warp(s_full, CH_NS, n);
            double2 x0 = make_double2(0, 0), x1 = x0;
            if (lane < 4) {
              x0 = sl[CH_BLK + 1 + i0];
              x1 = sl[CH_BLK + 5 + i0];
            }
            post_x(n, x0, x1);
            wait_warp(s_sr, CH_NX, n);
            double2* dst = AB + (long long)s * LDB + 1 + i0;
            if (lane < 4 && in0) dst[0] = make_double2(i0 == 0 ? s_sc[xb][1].x : 0.0, 0.0);
            if (lane < 4 && in1) dst[4] = make_double2(0.0, 0.0);
          }
          arrive(s_done, CH_NX, n);
        } else if (role == 2) {
          // ---- the diagonal block, D <- H^H D H
          const int yb = n & 3;
          wait_warp(s_full, CH_NS, n);
          // the stored lower triangle, the rest mirrored
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              const int d = i0 + 4 * r - (qb + 8 * m);
              M[r][m] = sl[d >= 0 ? lb + EM * m + 4 * r : ub + 8 * m + 4 * (LDB - 1) * r];
              M[r][m].y = d > 0 ? M[r][m].y : (d < 0 ? -M[r][m].y : 0.0);
            }
          arrive(s_empty, CH_NS, n);
          wait_warp(s_xr, CH_NX, n);
          double2 y[2];
          dot_rows(s_x[xb], y);
          if (lane < 4) {
            s_y[yb][i0] = y[0];
            s_y[yb][i0 + 4] = y[1];
            s_d0[yb][i0] = M[0][0];
            s_d0[yb][i0 + 4] = M[1][0];
          }
          bar_sync(3 + grp, 128);
          double2 yl = s_y[yb][lane];
          const double2 d0 = s_d0[yb][lane];
          double2 ul = s_x[xb][lane];
          wait_warp(s_sr, CH_NX, n);
          const double2 kap = s_sc[xb][0];
          const double beta = s_sc[xb][1].x;
          // lane = row: w = kappa y - 1/2 |kappa|^2 (u^H y) u, y = D u; then D <- D - u w^H - w u^H.  |kappa|^2 =
          // 1 / (beta^2 |u_0|^2), so the second term is 1/2 (u'^H y / |u_0|^2) u' with u' = u / beta
          if (lane == 0) ul.x -= beta;
          yl = caxpy(-beta, d0, yl);
          ul = cscale(ul, s_sc[xb][1].y);
          const double hk = 0.5 * s_rd[xb] * warp_sum(fma(ul.x, yl.x, ul.y * yl.y));
          double2* wv = s_wv[wid];
          wv[lane] = caxpy(-hk, ul, cmul(kap, yl));
          __syncwarp();
          double2 ui[2], wi[2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            ui[r] = s_x[xb][i0 + 4 * r];
            wi[r] = wv[i0 + 4 * r];
          }
          if (i0 == 0) ui[0].x -= beta;
          double2* dst = AB + (long long)r0 * LDB + lb;
          const bool in0 = i0 < N - r0, in1 = i0 + 4 < N - r0;
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            if (m > wg) break;   // above the diagonal for every row of the warp
            const double2 wq = wv[qb + 8 * m];
            double2 xm = s_x[xb][qb + 8 * m];
            if (m == 0 && qb == 0) xm.x -= beta;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const int d = i0 + 4 * r - (qb + 8 * m);
              double2 v = cfmsc(wq, ui[r], cfmsc(xm, wi[r], M[r][m]));
              if (d == 0) v.y = 0.0;
              if (d >= 0 && (r ? in1 : in0)) dst[EM * m + 4 * r] = v;
            }
          }
          arrive(s_done, CH_NX, n);
        }
      }
    });
  }
}

__global__ void k_band_to_tridiag(const double2* __restrict__ AB, long long N, double* __restrict__ d,
                                  double* __restrict__ e) {
  const long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (j >= N) return;
  d[j] = AB[j * LDB].x;
  if (j < N - 1) e[j] = AB[j * LDB + 1].x;
}

// Exciton vectors through stage 2: X <- Q2 X.  The reflectors of sweep s act on rows s + 1 + 32 t ..; a warp
// takes one vector through the 32 sweeps s0 .. s0 + 31 of a group, last sweep first, block t by block t: its 63
// rows are two numbers a lane (rows l and l + 32 of the window), of which sweep s0 + p uses the first where
// l >= p and the second where not, so nothing moves between the lanes.  Block t needs block t of the group
// behind (s0 + 32), whose rows start 32 further on.  One chain of dot products a block: N / 32 groups and as many
// blocks one after the other instead of N sweeps with a flag each: 8 vectors of N = 2916 14.6 -> 1.7 ms.
constexpr int BB_WARPS = 8;
__global__ void __launch_bounds__(32 * BB_WARPS, 2) k_bulge_back(const double2* __restrict__ A, long long N,
                                                                const double2* __restrict__ tau2, double2* X, int nvec,
                                                                unsigned int* prog, int* err) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long ng = (N - 1 + BW - 1) / BW;
  const int nch = (nvec + BB_WARPS - 1) / BB_WARPS;
  for (long long u = blockIdx.x; u < ng * nch; u += gridDim.x) {   // later sweeps first: no task waits for a later one
    const long long g = ng - 1 - u / nch, s0 = g * BW;
    const int c = (int)(u % nch) * BB_WARPS + wid;
    if (c >= nvec) continue;
    const int np = (int)min((long long)BW, N - 1 - s0);   // sweeps of the group
    const long long nblk = nsteps_of(N, s0), nnext = (g + 1 < ng) ? nsteps_of(N, s0 + BW) : 0;
    unsigned int* mine = prog + g * 32 + c;
    const long long toff = lane < np ? tau2_offset(N, s0 + lane) : 0;
    const int tn = lane < np ? (int)nsteps_of(N, s0 + lane) : 0;
    double2* xc = X + (long long)c * N + s0 + 1 + lane;
    auto row_ok = [&](long long r) { return s0 + 1 + r + lane < N; };
    double2 x0 = row_ok(0) ? __ldcg(xc) : make_double2(0, 0);
    for (long long t = 0; t < nblk; ++t) {
      const double2 tau = t < tn ? tau2[toff + t] : make_double2(0, 0);
      // v of sweep s0 + p in the window: element (lane - p) mod 32 of the stored reflector
      auto ldv = [&](int p) {
        const int i = (lane - p) & 31;
        return (p < np && s0 + p + 1 + t * BW + i < N) ? A[t * BW + i + (N - 1 - s0 - p) * N] : make_double2(0, 0);
      };
      double2 v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = ldv(31 - q);
      const long long need = min(t + 1, nnext);
      if (need > 0) {
        int bad = 0;
        if (lane == 0) bad = wait_at_least(prog + (g + 1) * 32 + c, (unsigned int)need, err) ? 0 : 1;
        if (__shfl_sync(0xffffffffu, bad, 0)) return;
      }
      double2 x1 = row_ok((t + 1) * BW) ? __ldcg(xc + (t + 1) * BW) : make_double2(0, 0);
#pragma unroll 1
      for (int p8 = 31; p8 > 0; p8 -= 8) {
        double2 vn[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) vn[q] = p8 >= 8 ? ldv(p8 - 8 - q) : make_double2(0, 0);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int p = p8 - q;
          const bool lo = lane >= p;
          const double2 xs = lo ? x0 : x1;
          const double2 sv = warp_sum2(cmulc(v[q], xs));   // v^H x
          const double2 tv = cmul(shfl2(tau, p), v[q]);
          const double2 xn = csub(xs, cmul(tv, sv));
          if (lo) x0 = xn;
          else x1 = xn;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = vn[q];
      }
      if (row_ok(t * BW)) xc[t * BW] = x0;
      if (t + 1 == nblk && row_ok((t + 1) * BW)) xc[(t + 1) * BW] = x1;
      x0 = x1;
      __syncwarp();
      if (lane == 0) st_release(mine, (unsigned int)(t + 1));
    }
  }
}

// ... and through stage 1: X <- Q1 X, the panels' block reflectors in reverse, X[k0:] -= V (T (V^H X[k0:])), all in
// one cooperative launch.  V from the panel's columns of A (unit at row k0+q, v below, zero above).  CTA b owns
// the 32-row tiles b, b + G, ... counted from the end of the matrix; per panel its share of V^H X, a grid
// barrier, the sum and the product with T (one CTA a vector, fixed order), a barrier, and its rows.  8 vectors of
// N = 2916 (91 panels): 6.5 -> 1.3 ms (three launches a panel, V read across its columns).
constexpr int BT_LD = 33;
constexpr size_t BT1_SMEM = (size_t)(32 * BT_LD + 2 * 32 * 32 + 32 * 32) * sizeof(double2);
__device__ __forceinline__ double2 panel_v(const double2* A, long long N, int j0, int k0, int q, long long r) {
  const long long rq = (long long)k0 + q;
  if (r < rq) return make_double2(0, 0);
  if (r == rq) return make_double2(1.0, 0.0);
  return A[r + (long long)(j0 + q) * N];
}
__global__ void __launch_bounds__(256, 1) k_bt1(const double2* __restrict__ A, long long N, const double2* __restrict__ Tbuf,
                                                double2* X, int nvec, double2* part, double2* Y, unsigned int* cnt,
                                                int* err) {
  extern __shared__ __align__(16) double2 bsm[];
  double2* sV = bsm;                    // [q][row]
  double2* sX = sV + 32 * BT_LD;        // [row][c]
  double2* sY = sX + 32 * 32;           // [q][c]
  double2* sP = sY + 32 * 32;
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, G = gridDim.x, b = blockIdx.x;
  const int npan = (int)((N - BW - 1 + BW - 1) / BW);
  unsigned int target = 0;
  for (int pnl = npan - 1; pnl >= 0; --pnl) {
    const int j0 = pnl * BW, k0 = j0 + BW;
    const int nref = (int)min((long long)BW, N - k0);
    const int ntile = (int)((N - k0 + 31) / 32), na = min(ntile, G);   // CTAs with rows
    const double2* T = Tbuf + (size_t)pnl * 1024;
    auto load = [&](int t) {   // tile t: rows N - 32 (t + 1) .. + 31, those from k0 on
      const long long r0 = N - 32LL * (t + 1);
      __syncthreads();
      for (int e = tid; e < 1024; e += 256) {
        const int i = e & 31, q = e >> 5;
        const long long r = r0 + i;
        sV[q * BT_LD + i] = (r >= k0 && q < nref) ? panel_v(A, N, j0, k0, q, r) : make_double2(0, 0);
        if (q < nvec) sX[i * 32 + (q ^ i)] = r >= k0 ? __ldcg(X + r + (long long)q * N) : make_double2(0, 0);
      }
      __syncthreads();
    };
    // share of V^H X: thread (q = lane, vectors wp + 8 u)
    double2 acc[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = make_double2(0, 0);
    for (int t = b; t < ntile; t += G) {
      load(t);
      for (int i = 0; i < 32; ++i) {
        const double2 v = sV[lane * BT_LD + i];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (wp + 8 * u < nvec) acc[u] = cfmac(v, sX[i * 32 + ((wp + 8 * u) ^ i)], acc[u]);
      }
    }
    if (b < na) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (wp + 8 * u < nvec) part[((size_t)(wp + 8 * u) * G + b) * 32 + lane] = acc[u];
    }
    if (!grid_sync(cnt, target += G, err)) return;
    // Y[:, c] = T sum of the shares
    for (int c = b; c < nvec; c += G) {
      double2 t = make_double2(0, 0);
      const double2* p = part + (size_t)c * G * 32 + lane;
      for (int i0 = wp; i0 < na; i0 += 64) {
        double2 pv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) pv[u] = i0 + 8 * u < na ? ldcg2(p + (size_t)(i0 + 8 * u) * 32) : make_double2(0, 0);
#pragma unroll
        for (int u = 0; u < 8; ++u) t = cadd(t, pv[u]);
      }
      sP[tid] = t;
      __syncthreads();
      if (wp == 0) {
#pragma unroll
        for (int u = 1; u < 8; ++u) t = cadd(t, sP[u * 32 + lane]);
        double2 y = make_double2(0, 0);   // (T P)[q] = sum_{l >= q} T[q][l] P[l]
        for (int l = 0; l < 32; ++l) {
          const double2 pl = shfl2(t, l);
          if (l >= lane) y = cfma(T[lane + 32 * l], pl, y);
        }
        Y[c * 32 + lane] = y;
      }
      __syncthreads();
    }
    if (!grid_sync(cnt, target += G, err)) return;
    if (b < na) {
      for (int e = tid; e < 32 * nvec; e += 256) sY[(e & 31) * 32 + (e >> 5)] = ldcg2(Y + e);
      for (int t = b; t < ntile; t += G) {
        if (t != b || ntile > G) load(t);   // else the tile is still here
        else __syncthreads();
        const long long r = N - 32LL * (t + 1) + lane;
        double2 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = make_double2(0, 0);
        for (int q = 0; q < 32; ++q) {
          const double2 v = sV[q * BT_LD + lane];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (wp + 8 * u < nvec) x[u] = cfma(v, sY[q * 32 + wp + 8 * u], x[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = wp + 8 * u;
          if (c < nvec && r >= k0) X[r + (long long)c * N] = csub(sX[lane * 32 + (c ^ lane)], x[u]);
        }
      }
    }
  }
}

}  // namespace

// Largest N whose panels fit the aggregate shared memory of the panel QR (one CTA per SM,
// at most PQ_MAX_R rows of the 32-wide panel each).
constexpr int PQ_MAX_R = 384;
constexpr long long LA_FOUR_FROM = 20000;   // N from which groups of four are used
constexpr int LOOKAHEAD = 4;   // largest number of panels applied per rank-2k update (K = 128)
// k_wfuse holds the K = 32 (group - 1) columns of the group in shared memory (220 KB at 4)
static_assert(LOOKAHEAD >= 1 && LOOKAHEAD <= 4, "look-ahead groups of 1 to 4 panels");
// Group size per reduction: the wider update pays off where the trailing matrices are large
// (config 2, N = 36864: fours 11.75 s, pairs 11.86 s per step); at N = 8100 the update rate does
// not rise and the corrections cost more (solve: fours 251 ms, pairs 247; N = 2304: 33.1 and 32.0).
static int lookahead_group(const wtbg_ctx* ctx) {
  return ctx->panel_group > 0 ? ctx->panel_group : (ctx->N >= LA_FOUR_FROM ? 4 : 2);
}
static bool two_stage_fits(wtbg_ctx* ctx, long long N) {
  if (ctx->nsm <= 0) cudaDeviceGetAttribute(&ctx->nsm, cudaDevAttrMultiProcessorCount, ctx->device);
  return N > BW + 1 && (N + ctx->nsm - 1) / ctx->nsm <= PQ_MAX_R;
}

// The reduction used for the current matrix: two-stage wherever it fits (auto).  Device time of a
// solve, one-stage against two-stage: N = 36 1.01 / 0.49 ms, 144 4.1 / 2.3, 576 17.4 / 10.4, 1156 36.8 /
// 22.0, 2304 83.7 / 47.6, 14400 2423 / 979 (the one-stage reduction is four launches per column, the
// two-stage one five per 32 columns and one for the chase).  Later steps brought the two-stage solve of N = 576 to
// 6.5 ms, of 2304 to 30, of 14400 to 854.
bool use_two_stage(wtbg_ctx* ctx) { return ctx->tri_mode != 1 && two_stage_fits(ctx, ctx->N); }

// Work buffers of the two-stage reduction for N (nband bands side by side for Q groups).
static int two_stage_buffers(wtbg_ctx* ctx, int nband) {
  const long long N = ctx->N;
  const int nsm = ctx->nsm > 0 ? ctx->nsm : 148;
  const long long npan = (N - BW - 1 + BW - 1) / BW;
  ENSURE(ctx->d, (size_t)N * 8);
  ENSURE(ctx->e, (size_t)N * 8);
  ENSURE(ctx->g, (size_t)N * 16 * NGMAX);
  const int la = lookahead_group(ctx);
  ENSURE(ctx->Wp, (size_t)N * 16 * 2 * la * BW);   // two groups: see run_stage1
  ENSURE(ctx->t2V, (size_t)N * 16 * 2 * la * BW);
  ENSURE(ctx->t2X, (size_t)8 * BW * N * 16);
  const long long wfg = std::min<long long>(nsm, (N + WF_TR - 1) / WF_TR);   // CTAs of k_wfuse
  ENSURE(ctx->t2G, (size_t)((wfg + 1) * (2 * la - 1) + 1) * 1024 * 16);
  ENSURE(ctx->t2T, (size_t)std::max<long long>(npan, 1) * 1024 * 16);
  ENSURE(ctx->t2P, (size_t)nsm * (16 + 2 * 16 * BW + 16 * BW * BW + 16 * BW * NGMAX) + 4096 +
                        (size_t)std::max<long long>(npan, 1) * 8);
  ENSURE(ctx->t2AB, (size_t)nband * (N + AB_PAD) * LDB * 16);
  ENSURE(ctx->t2prog, (size_t)nband * N * 4 + 512);
  ENSURE(ctx->triErr, 16);
  return 0;
}

// Panel QR on one cluster.  C CTAs of R = 8 NR rows with R >= 32 (CTA 0 holds the first 32 rows), as many
// CTAs as that allows: the column step gets shorter with fewer rows per thread.
using PanelClFn = void (*)(PanelArgs, int);
static PanelClFn panel_cl_fn(int nr) {
  switch (nr) {
    case 4: return k_panel_qr_cl<4>;
    case 6: return k_panel_qr_cl<6>;
    case 8: return k_panel_qr_cl<8>;
    case 10: return k_panel_qr_cl<10>;
    case 12: return k_panel_qr_cl<12>;
    case 14: return k_panel_qr_cl<14>;
    case 16: return k_panel_qr_cl<16>;
    case 18: return k_panel_qr_cl<18>;
    case 20: return k_panel_qr_cl<20>;
    case 22: return k_panel_qr_cl<22>;
    default: return k_panel_qr_cl<24>;
  }
}
// Shared memory that keeps a panel CTA alone on its SM while the rank-2k update runs beside it (the update
// takes 66 KB a CTA of the SM's 228).
constexpr size_t ALONE_SMEM = 168 * 1024;
static int launch_panel_cluster(wtbg_ctx* ctx, const PanelArgs& pa) {
  const long long m = pa.N - pa.k0;
  int C = 1;
  while (C < ctx->panel_cl_max && (long long)C * 32 < m) C *= 2;
  int nr = (int)((m + 8 * C - 1) / (8 * C));
  nr = std::max(4, (nr + 1) & ~1);
  PanelClFn fn = panel_cl_fn(nr);
  const size_t smem = std::max(pc_smem(nr), ALONE_SMEM);
  CK(cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if (C > 8) CK(cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(PC_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  CK(cudaLaunchKernelEx(&cfg, fn, pa, C));
  return 0;
}
// Largest cluster the device takes for the panel kernel (16 where a GPC has room for it, else 8) and the
// panel rows that gives.
static int panel_cluster_limits(wtbg_ctx* ctx) {
  if (ctx->panel_cl_max > 0) return 0;
  PanelClFn fn = panel_cl_fn(PC_MAX_NR);
  const size_t smem = std::max(pc_smem(PC_MAX_NR), ALONE_SMEM);
  CK(cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  CK(cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(PC_MAXC);
  cfg.blockDim = dim3(PC_THREADS);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = PC_MAXC;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int ncl = 0;
  if (cudaOccupancyMaxActiveClusters(&ncl, (const void*)fn, &cfg) != cudaSuccess) {
    cudaGetLastError();
    ncl = 0;
  }
  ctx->panel_cl_max = ncl > 0 ? PC_MAXC : 8;
  ctx->panel_cl_rows = (long long)ctx->panel_cl_max * 8 * PC_MAX_NR;
  return 0;
}

// Stage 1 (dense -> band) of the context's matrix; the band goes to slot `band` of ctx->t2AB.
// ng velocity vectors in ctx->g follow the reflectors.
static int run_stage1(wtbg_ctx* ctx, int ng, int band) {
  const long long N = ctx->N;
  cudaStream_t s = ctx->stream;
  const int nsm = ctx->nsm > 0 ? ctx->nsm : 148;
  const long long npan = (N - BW - 1 + BW - 1) / BW;
  const int SMAX = 8;
  double2* A = ctx->H.as<double2>();
  double2* g = ctx->g.as<double2>();
  double2* Vp = ctx->t2V.as<double2>();
  double2* Wp = ctx->Wp.as<double2>();
  double2* Xpart = ctx->t2X.as<double2>();
  const int la = std::min(LOOKAHEAD, lookahead_group(ctx));
  double2* red = ctx->t2G.as<double2>();                     // sums of k_wfuse, then its CTAs' shares
  double2* part = red + (size_t)(2 * la) * 1024;
  double2* Tbuf = ctx->t2T.as<double2>();
  char* pb = ctx->t2P.as<char>();
  double2* partW = reinterpret_cast<double2*>(pb + (size_t)nsm * 16);   // 16-byte aligned for any SM count
  double2* partG = partW + (size_t)2 * nsm * BW;
  double2* partVg = partG + (size_t)nsm * BW * BW;
  double2* alpha = partVg + (size_t)nsm * BW * NGMAX;
  unsigned int* cnt = reinterpret_cast<unsigned int*>(alpha + 2 * BW);   // barrier counters, two per panel
  int* err = ctx->triErr.as<int>();
  if (int r = panel_cluster_limits(ctx)) return r;
  CK(cudaMemsetAsync(cnt, 0, (size_t)std::max<long long>(npan, 1) * 8, s));
  CK(cudaFuncSetAttribute(k_hemm2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HM_SMEM));
  // profiling: event pairs around the panel QR, the Hermitian product and the rank-2k update
  // of every panel (read after the stage), and around the stage
  const bool prof = ctx->profiling != 0;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  if (prof) {
    for (auto& e : ev) CK(cudaEventCreate(&e));
    if (int r = ensure_events(ctx, 6 * (size_t)std::max<long long>(npan, 1))) return r;
    cudaEventRecord(ev[0], s);
  }
  auto mark = [&](long long pnl, int k) {
    if (prof) cudaEventRecord(ctx->evpool[6 * pnl + k], s);
  };
  // Panel QR of panel pnl into V (its 32 columns), then X = A22 V (split K) and W.  Inside a
  // look-ahead group (K > 0) A22 still lacks the updates of the group's K/32 earlier panels
  // (Vacc, Wacc) and the product is corrected by -Vacc C1 - Wacc C2.
  auto factor = [&](long long pnl, double2* V) -> int {
    const int j0 = (int)(pnl * BW), k0 = j0 + BW;
    const long long m = N - k0;
    const int nref = (int)std::min<long long>(BW, m);
    PanelArgs pa{};
    pa.A = A;
    pa.N = N;
    pa.j0 = j0;
    pa.k0 = k0;
    pa.jb = BW;
    pa.nref = nref;
    pa.Vp = V;
    pa.Tout = Tbuf + (size_t)pnl * 1024;
    pa.g = g;
    pa.ng = ng;
    pa.err = err;
    mark(pnl, 0);
    if (m <= ctx->panel_cl_rows && !ctx->panel_wide) {
      if (int r = launch_panel_cluster(ctx, pa)) return r;
    } else {
      // grid-wide: G CTAs of R rows (at most 64 CTAs while the rows fit: the panel is latency-bound,
      // and fewer CTAs make the grid barrier and the cross-CTA reductions cheaper; mode 5 as many as N = 56832 takes)
      const int R = ctx->panel_wide ? (int)std::max<long long>(8, (m + nsm - 1) / nsm)
                                    : (int)std::min<long long>(PQ_MAX_R, std::max<long long>(64, (m + 63) / 64));
      const int G = (int)((m + R - 1) / R);
      pa.R = R;
      pa.RS = R | 1;
      pa.partW = partW;
      pa.partG = partG;
      pa.partVg = partVg;
      pa.alpha = alpha;
      pa.cnt = cnt + pnl;
      const size_t psm = std::max((size_t)BW * (R | 1) * 16, ALONE_SMEM);
      CK(cudaFuncSetAttribute(k_panel_qr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psm));
      if (G > PQ_MAXG) return set_err(ctx, WTBG_ERR_UNSUPPORTED, "panel QR: more CTAs than the column reduction holds");
      void* args[] = {&pa};
      CK(cudaLaunchCooperativeKernel((const void*)k_panel_qr, dim3(G), dim3(PQ_THREADS), args, psm, s));
    }
    mark(pnl, 1);
    WTBG_COUNT(ctx, 1);
    return 0;
  };
  auto product = [&](long long pnl, const double2* V, const double2* Vacc, const double2* Wacc, double2* Wout, int K) -> int {
    const int k0 = (int)(pnl * BW) + BW;
    const long long m = N - k0;
    const int nIm = (int)((m + 63) / 64);
    int S = (int)std::min<long long>(SMAX, std::max<long long>(1, (4LL * nsm + nIm - 1) / nIm));
    S = std::min(S, nIm);
    const int chunkJ = (nIm + S - 1) / S;
    S = (nIm + chunkJ - 1) / chunkJ;
    mark(pnl, 2);
    k_hemm2<<<dim3(nIm, S), 256, HM_SMEM, s>>>(A, N, k0, V, nIm, chunkJ, Xpart);
    mark(pnl, 3);
    WfArgs wa{};
    wa.X = Xpart;
    wa.S = S;
    wa.N = N;
    wa.k0 = k0;
    wa.V = V;
    wa.T = Tbuf + (size_t)pnl * 1024;
    wa.Vacc = Vacc;
    wa.Wacc = Wacc;
    wa.W = Wout;
    wa.part = part;
    wa.red = red;
    wa.cnt = cnt + npan + pnl;
    wa.err = err;
    const long long ntile = (m + WF_TR - 1) / WF_TR, per = (ntile + nsm - 1) / nsm;
    wa.shares = (int)((ntile + per - 1) / per);
    const void* const wf[LOOKAHEAD] = {(const void*)k_wfuse<0>, (const void*)k_wfuse<1>, (const void*)k_wfuse<2>,
                                       (const void*)k_wfuse<3>};
    const size_t wsm = wf_smem(K / 32);
    CK(cudaFuncSetAttribute(wf[K / 32], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wsm));
    void* wargs[] = {&wa};
    CK(cudaLaunchCooperativeKernel(wf[K / 32], dim3((unsigned)std::min(wa.shares, nsm / ctx->nlane)), dim3(256), wargs, wsm, s));
    WTBG_COUNT(ctx, 2);
    CKL("two-stage panel");
    return 0;
  };
  // pending updates of kc columns of V, W on the 32 columns from c0
  auto strip = [&](long long c0, int kc, const double2* V, const double2* W) -> int {
    for (int q = 0; q < kc; q += 64) {   // as much as shared memory holds
      const int kq = std::min(64, kc - q);
      const size_t sss = ((size_t)2 * 32 * kq + (size_t)2 * 33 * kq) * 16;
      CK(cudaFuncSetAttribute(k_strip_update, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sss));
      k_strip_update<<<(int)((N - c0 + 31) / 32), 256, sss, s>>>(A, N, c0, kq, V + (size_t)q * N, W + (size_t)q * N);
      WTBG_COUNT(ctx, 1);
    }
    return 0;
  };
  // Panels in look-ahead groups of la (up to LOOKAHEAD): panel j of a group first gets the pending
  // updates of the group's earlier panels on its own 32 columns (strip), is factored, and forms
  // its product from the matrix that still lacks those updates (corrected); one rank-2k update
  // with K = 32 x (panels in the group) then applies the whole group to the trailing matrix.
  // The QR of the next group's first panel, a latency chain on one cluster or 64 CTAs, needs only its own 32
  // columns: they are updated first (strip), and the rank-2k update of the rest runs beside it.  V and W
  // of the two groups in turn.  Solve: N = 1156 14.6 -> 14.3 ms, 2304 32.0 -> 30.7, 3600 60.5 -> 57.0,
  // 8100 247 -> 236, 14400 870 -> 843.
  std::vector<double> her2k_flops(npan, 0.0);
  bool factored = false;
  for (long long p0 = 0, grp = 0; p0 < npan; p0 += la, ++grp) {
    const int gsz = (int)std::min<long long>(la, npan - p0);
    double2* Vg = Vp + (size_t)(grp & 1) * la * BW * N;
    double2* Wg = Wp + (size_t)(grp & 1) * la * BW * N;
    for (int j = 0; j < gsz; ++j) {
      const long long pnl = p0 + j;
      const int K = BW * j;
      double2* V = Vg + (size_t)K * N;
      if (j > 0) {
        mark(pnl - 1, 4);
        if (int r = strip(pnl * BW, K, Vg, Wg)) return r;   // the panel's first column (= the previous panel's k0)
        mark(pnl - 1, 5);
        her2k_flops[pnl - 1] = 8.0 * (double)(N - pnl * BW) * 32 * 2 * K;
      }
      if (j > 0 || !factored)
        if (int r = factor(pnl, V)) return r;
      if (int r = product(pnl, V, Vg, Wg, Wg + (size_t)K * N, K)) return r;
    }
    const long long pl = p0 + gsz - 1;
    const long long kl = (pl + 1) * BW;
    const long long ml = N - kl;
    const int Kg = 32 * (gsz - 1) + (int)std::min<long long>(BW, ml);
    factored = pl + 1 < npan;
    if (factored) {
      if (int r = strip(kl, Kg, Vg, Wg)) return r;
      if (int r = factor(pl + 1, Vp + (size_t)((grp + 1) & 1) * la * BW * N)) return r;
    }
    mark(pl, 4);   // with profiling the events keep the two apart
    if (int r = launch_her2k_v(ctx, A, N, Wg, Vg, N, 0, Kg, factored ? kl + BW : kl, factored)) return r;
    mark(pl, 5);
    const double mu = (double)(factored ? ml - BW : ml);
    her2k_flops[pl] = mu * (mu + 1.0) * 0.5 * 16.0 * Kg;
  }
  k_band_extract<<<(unsigned)(N + AB_PAD), BW * 2, 0, s>>>(A, N, ctx->t2AB.as<double2>() + (size_t)band * (N + AB_PAD) * LDB);
  WTBG_COUNT(ctx, 1);
  CKL("k_band_extract");
  if (prof) {
    cudaEventRecord(ev[1], s);
    CK(cudaEventSynchronize(ev[1]));
    float t = 0.f;
    cudaEventElapsedTime(&t, ev[0], ev[1]);
    ctx->stats.stage1_ms += t;
    ctx->stats.tri_ms += t;
    for (long long pnl = 0; pnl < npan; ++pnl) {
      const double m = (double)(N - (pnl + 1) * BW), nref = std::min(m, (double)BW);
      float a = 0.f, b = 0.f, c = 0.f;
      cudaEventElapsedTime(&a, ctx->evpool[6 * pnl + 0], ctx->evpool[6 * pnl + 1]);
      cudaEventElapsedTime(&b, ctx->evpool[6 * pnl + 2], ctx->evpool[6 * pnl + 3]);
      cudaEventElapsedTime(&c, ctx->evpool[6 * pnl + 4], ctx->evpool[6 * pnl + 5]);
      ctx->stats.panel_ms += a;
      ctx->stats.hemm_ms += b;
      ctx->stats.hemm_flops += 8.0 * m * m * nref;
      ctx->stats.her2k_ms += c;   // rank-2k updates (K = 64 per pair) and the look-ahead strips
      ctx->stats.her2k_flops += her2k_flops[pnl];
      ctx->stats.her2k_launches += 1;
    }
    for (auto& e : ev) cudaEventDestroy(e);
  }
  return 0;
}

// Stage 2 (band -> tridiagonal) of nband bands of ctx->t2AB in one persistent launch; the
// tridiagonal forms go to dd/ee ([nband][N] each).  With store (one band only; ctx->tau must
// hold ceil_sum(N-1) entries) the ng velocity vectors follow the reflectors and the reflectors
// are kept for the eigenvector back-transform; without, only the band is reduced.
static int run_stage2(wtbg_ctx* ctx, int nband, int ng, bool store, double* dd, double* ee) {
  if (store && (nband != 1 || ctx->tau.bytes < (size_t)std::max<long long>(ceil_sum(ctx->N - 1), 1) * 16))
    return set_err(ctx, WTBG_ERR_STATE, "two-stage: reflector storage not sized");
  const long long N = ctx->N;
  cudaStream_t s = ctx->stream;
  const int nsm = ctx->nsm > 0 ? ctx->nsm : 148;
  double2* AB = ctx->t2AB.as<double2>();
  unsigned int* prog = ctx->t2prog.as<unsigned int>();
  const bool prof = ctx->profiling != 0;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  if (prof) {
    for (auto& e : ev) CK(cudaEventCreate(&e));
    cudaEventRecord(ev[0], s);
  }
  CK(cudaMemsetAsync(prog, 0, (size_t)nband * N * 4, s));
  BulgeArgs ba;
  ba.AB = AB;
  ba.N = N;
  ba.A = ctx->H.as<double2>();
  ba.tau2 = ctx->tau.as<double2>();
  ba.g = ctx->g.as<double2>();
  ba.ng = store ? ng : 0;
  ba.prog = prog;
  ba.err = ctx->triErr.as<int>();
  ba.store = store ? 1 : 0;
  ba.nprob = nband;
  ba.ab_stride = (N + AB_PAD) * LDB;
  ba.prog_stride = N;
  const long long nsweep = (long long)nband * (N - 1);
  if (ctx->bulge_warp_mode) {   // one warp per sweep
    const size_t bsm = (size_t)BG_WARPS * BG_WARP_TILE * 16;
    CK(cudaFuncSetAttribute(k_bulge, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsm));
    int per = 1;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_bulge, 32 * BG_WARPS, bsm));
    const int gb = (int)std::max<long long>(1, std::min<long long>((long long)nsm * std::max(per, 1),
                                                                    (nsweep + BG_WARPS - 1) / BG_WARPS));
    void* args[] = {&ba};
    CK(cudaLaunchCooperativeKernel((const void*)k_bulge, dim3(gb), dim3(32 * BG_WARPS), args, bsm, s));
  } else {   // one CTA per sweep
    CK(cudaFuncSetAttribute(k_chase, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CH_SMEM));
    const int gb = (int)std::max<long long>(1, std::min<long long>(nsm, nsweep));
    void* args[] = {&ba};
    CK(cudaLaunchCooperativeKernel((const void*)k_chase, dim3(gb), dim3(CH_THREADS), args, CH_SMEM, s));
  }
  for (int q = 0; q < nband; ++q)
    k_band_to_tridiag<<<(int)((N + 255) / 256), 256, 0, s>>>(AB + (size_t)q * (N + AB_PAD) * LDB, N, dd + (size_t)q * N,
                                                              ee + (size_t)q * N);
  WTBG_COUNT(ctx, 1 + nband);
  CKL("two-stage bulge chasing");
  if (prof) {
    cudaEventRecord(ev[1], s);
    CK(cudaEventSynchronize(ev[1]));
    float t = 0.f;
    cudaEventElapsedTime(&t, ev[0], ev[1]);
    ctx->stats.stage2_ms += t;
    ctx->stats.tri_ms += t;
    for (auto& e : ev) cudaEventDestroy(e);
  }
  return 0;
}

static std::mutex& spin_mutex(int device) {
  static std::mutex m[64];   // device ordinals; two that share one only wait for each other
  return m[(unsigned)device % 64u];
}
SpinSection::SpinSection(wtbg_ctx* ctx) : ctx_(ctx) { spin_mutex(ctx->device).lock(); }
SpinSection::~SpinSection() {
  cudaStreamSynchronize(ctx_->stream);   // an error stays with the stream: the caller's next call returns it
  spin_mutex(ctx_->device).unlock();
}

int run_tridiagonalise2(wtbg_ctx* ctx) {
  SpinSection section(ctx);
  const long long N = ctx->N;
  cudaStream_t s = ctx->stream;
  if (int r = two_stage_buffers(ctx, 1)) return r;
  ENSURE(ctx->tau, (size_t)std::max<long long>(ceil_sum(N - 1), 1) * 16);
  CK(cudaMemsetAsync(ctx->triErr.p, 0, 4, s));
  double2* g = ctx->g.as<double2>();
  // velocity vectors g (as the one-stage reduction)
  const int ng = ctx->have_velocity ? (ctx->temp_on ? 10 : 5) : 0;
  ctx->ng = ctx->have_velocity ? ng : 5;
  if (ctx->have_velocity && ctx->temp_on) {
    if (int r = fill_g_vectors(ctx, g)) return r;
  } else if (ctx->have_velocity) {
    CK(cudaMemcpyAsync(g, ctx->h.p, (size_t)N * 16 * 5, cudaMemcpyDeviceToDevice, s));
  } else {
    CK(cudaMemsetAsync(g, 0, (size_t)N * 16 * 5, s));
  }
  if (int r = run_stage1(ctx, ng, 0)) return r;
  if (int r = run_stage2(ctx, 1, ng, true, ctx->d.as<double>(), ctx->e.as<double>())) return r;
  ctx->tri_two = true;
  return 0;
}

// Q groups of the exciton band structure (eigenvalues only): group_begin sizes the work
// buffers for nq bands, group_add runs stage 1 of the matrix just built into band slot i, and
// group_finish chases all nq bands in one persistent launch; the tridiagonal forms of the group
// land in dd/ee ([nq][N] each).
int two_stage_group_begin(wtbg_ctx* ctx, int nq) {
  if (int r = two_stage_buffers(ctx, nq)) return r;
  ENSURE(ctx->t2de, (size_t)2 * nq * ctx->N * 8);
  CK(cudaMemsetAsync(ctx->triErr.p, 0, 4, ctx->stream));
  return 0;
}
int two_stage_group_add(wtbg_ctx* ctx, int slot, int nq) {
  if (int r = two_stage_buffers(ctx, nq)) return r;   // the panel buffers of a further lane
  return run_stage1(ctx, 0, slot);
}
// Q points whose stage 1 runs side by side, each on its own stream with its own matrix and buffers.  Stage 1 of
// a small matrix is a chain of kernels that leave most of the device idle (the panel QR takes 16 SMs or 64), and at
// large N the panels of one run beside the products of another.  The kernels that spin on a grid barrier are all
// resident at once: k_wfuse takes nsm / lanes CTAs, and the grid-wide panel QR (64 CTAs up to N = 9216) runs only
// where there are two lanes; four where every panel goes to a cluster.  Other contexts of the device are kept
// out meanwhile (SpinSection).  A path of 12 Q points of N = 576 27.8 ->
// 13.3 ms, 6 of 1156 34.8 -> 20.9, 4 of 2304 58.4 -> 38.2 (two lanes 43.8), 3 of 5625 240 -> 214, of 8100 526 -> 486.
int two_stage_lanes(wtbg_ctx* ctx, long long N, int nq) {
  const int nsm = ctx->nsm > 0 ? ctx->nsm : 148;
  if (ctx->profiling || ctx->panel_wide || nq < 2 || N > 9216 || nsm < 128) return 1;
  if (panel_cluster_limits(ctx)) return 1;
  const int n = std::min(nq, N - BW <= ctx->panel_cl_rows ? 4 : 2);
  size_t freeb = 0, totb = 0;
  if (cudaMemGetInfo(&freeb, &totb) != cudaSuccess) return 1;
  const size_t need = (size_t)(n - 1) * ((size_t)N * N * 16 + (size_t)N * 16 * BW * 32 + (64u << 20));
  return need <= (freeb + lane_bytes(ctx)) / 2 ? n : 1;   // what the lanes hold from the last call counts as free
}
int two_stage_group_finish(wtbg_ctx* ctx, int nq, double** dd, double** ee) {
  *dd = ctx->t2de.as<double>();
  *ee = *dd + (size_t)nq * ctx->N;
  if (int r = run_stage2(ctx, nq, 0, false, *dd, *ee)) return r;
  ctx->tri_two = false;   // no reflectors kept: exciton vectors need a wtbg_bse_solve
  return 0;
}

// Exciton vectors through both stages: X <- Q1 (Q2 X), Q2 the bulge-chasing reflectors in
// reverse, Q1 the panels' block reflectors in reverse.
int run_backtransform2(wtbg_ctx* ctx, double2* X, int nvec) {
  SpinSection section(ctx);
  const long long N = ctx->N;
  cudaStream_t s = ctx->stream;
  const int nsm = ctx->nsm > 0 ? ctx->nsm : 148;
  unsigned int* prog = ctx->t2prog.as<unsigned int>();
  int* err = ctx->triErr.as<int>();
  const long long ng = (N - 1 + BW - 1) / BW;
  CK(cudaMemsetAsync(prog, 0, (size_t)(ng + 1) * 32 * 4, s));   // and the barrier counter of k_bt1
  CK(cudaMemsetAsync(err, 0, 4, s));
  const double2* A = ctx->H.as<double2>();
  long long NN = N;
  {
    int per = 1;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_bulge_back, 32 * BB_WARPS, 0));
    const long long tasks = ng * ((nvec + BB_WARPS - 1) / BB_WARPS);
    const int gb = (int)std::max<long long>(1, std::min<long long>((long long)nsm * std::max(per, 1), tasks));
    const double2* tau2 = ctx->tau.as<double2>();
    void* args[] = {(void*)&A, (void*)&NN, (void*)&tau2, (void*)&X, (void*)&nvec, (void*)&prog, (void*)&err};
    CK(cudaLaunchCooperativeKernel((const void*)k_bulge_back, dim3(gb), dim3(32 * BB_WARPS), args, 0, s));
  }
  {
    const int gt = (int)std::max<long long>(1, std::min<long long>(nsm, (N - BW + 31) / 32));
    ENSURE(ctx->t2G, (size_t)(gt + 1) * 1024 * 16);
    double2* Y = ctx->t2G.as<double2>();
    double2* part = Y + 1024;
    const double2* T = ctx->t2T.as<double2>();
    unsigned int* cnt = prog + ng * 32;
    CK(cudaFuncSetAttribute(k_bt1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BT1_SMEM));
    void* args[] = {(void*)&A, (void*)&NN, (void*)&T, (void*)&X, (void*)&nvec, (void*)&part, (void*)&Y, (void*)&cnt, (void*)&err};
    CK(cudaLaunchCooperativeKernel((const void*)k_bt1, dim3(gt), dim3(256), args, BT1_SMEM, s));
  }
  WTBG_COUNT(ctx, 2);
  CKL("two-stage back-transform");
  int herr = 0;
  CK(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (herr) return set_err(ctx, WTBG_ERR_CUDA, "back-transform: a sweep wait timed out");
  return 0;
}
