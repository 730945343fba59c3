// pb_cg_small.cu -- PCG with point Jacobi or no preconditioner on vectors that fit the
// registers of one CTA per SM, all iterations in one cooperative launch.
//
// The loop is KSP_pCG's (src/pcg.f90:224-892), as run_pcg's kernels compute it.  A 65,536-row
// iteration moves 5 MB, all of it in L2, so five launches of 2 to 7 us each (two of them
// ending in a ticket over 592 CTAs) were its whole cost.  Here a CTA keeps its rows' x, r
// and p in registers and an iteration has two grid-wide sums:
//   1. p = s + beta p for the own rows and, recomputed from s and the old p, for the
//      neighbours (so no barrier lies between the update and the product); q = A p; <p, q>
//   2. r -= alpha q, s = D^-1 r, written for the neighbours; <s, r> and <r, r>
// Every CTA then computes the same step lengths and stop test from the same sums.
//
// Grid sum without a counter: a CTA stores each 64-bit partial as two 64-bit words of 32
// value bits and a 32-bit tag (the iteration number), so a word is either this iteration's or
// visibly not.  Up to kCgDirect CTAs read all CTAs' words until the tags match, one L2 round
// trip after the last store; of more, CTA 0 does and stores the total in kCgCopies lines for
// the others, because lines that many CTAs poll hold up the stores into them.  Only the second sum also publishes the vectors: p and s are gathered
// after it, and what the first sum orders (s may be overwritten) rests on loads whose values
// went into it.  The two sums of an iteration use different words, so a CTA can only
// overwrite words that every CTA has finished reading.  Waits are bounded; one that runs
// out sets *err and ends the CTA, whose missing words then end the others the same way.
#include "pb_cg_small.cuh"
#include "pb_device.cuh"

namespace pb {

namespace {

constexpr int kCgThreads = 512;
constexpr int kCgWarps = kCgThreads / 32;
constexpr int kCgMaxElems = 4;             // rows per thread
constexpr unsigned kCgWaitLimit = 1u << 21;
// Up to this many CTAs read one another's words, beyond it CTA 0 hands the total back.  Five-point
// stencil, us an iteration, read directly / through CTA 0: 16 CTAs 5.7 / 7.0, 32 5.7 / 6.8, 64 6.4 /
// 6.8, 96 7.5 / 6.9, 128 8.6 / 6.8.
constexpr int kCgDirect = 32;

// Both words of a value in one access; each word is single-copy atomic by itself, and each
// carries its tag.
__device__ __forceinline__ ulonglong2 ld_words(const unsigned long long* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_words(unsigned long long* p, unsigned long long x, unsigned long long y) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y) : "memory");
}

// Sums K per-thread values over the grid; every thread of every CTA gets the same bits.
// words: 2 K per CTA, then the total's copies, 2 K words in a line each.  PUBLISH: the CTA's
// vector stores are visible to every CTA that has the sum.  False when a wait ran out.
template <int K, bool PUBLISH>
__device__ __forceinline__ bool grid_sum(double (&v)[K], unsigned long long* words, unsigned tag,
                                         double (*wsum)[kCgWarps], double (*csum)[8], int* sbad) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, G = gridDim.x;
  unsigned long long* tot = words + (size_t)((G * 2 * K + kCgLine - 1) & ~(kCgLine - 1));
  auto put = [&](unsigned long long* w, double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    st_words(w, (b & 0xffffffff00000000ull) | tag, (b << 32) | tag);
  };
  // waits for K values in consecutive words; false when it gave up
  auto get = [&](const unsigned long long* w, double (&x)[K]) -> bool {
    ulonglong2 u[K];
#pragma unroll
    for (int k = 0; k < K; ++k) u[k] = ld_words(w + 2 * k);
    for (unsigned it = 0;; ++it) {
      bool pending = false;
#pragma unroll
      for (int k = 0; k < K; ++k) pending |= (unsigned)u[k].x != tag || (unsigned)u[k].y != tag;
      if (!pending) break;
      if (it >= kCgWaitLimit) return false;
#pragma unroll
      for (int k = 0; k < K; ++k) u[k] = ld_words(w + 2 * k);
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
      x[k] = __longlong_as_double((long long)((u[k].x & 0xffffffff00000000ull) | (u[k].y >> 32)));
    return true;
  };
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double x = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
    if (lane == 0) wsum[k][warp] = x;
  }
  __syncthreads();
  if (warp < K) {    // warp k stores this CTA's k-th sum
    double x = lane < kCgWarps ? wsum[warp][lane] : 0.0;
#pragma unroll
    for (int o = kCgWarps / 2; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
    if (lane == 0) {
      if (PUBLISH) __threadfence();   // the block barrier above put the CTA's stores before it
      put(words + (size_t)blockIdx.x * 2 * K + 2 * warp, x);
    }
  }
  const bool direct = G <= kCgDirect;
  if (direct || blockIdx.x == 0) {
    const int nw = (G + 31) >> 5;   // warps that read: at most 8 (G <= 256)
    if (warp < nw) {
      double x[K];
#pragma unroll
      for (int k = 0; k < K; ++k) x[k] = 0.0;
      const bool bad = t < G && !get(words + (size_t)t * 2 * K, x);
      if (PUBLISH) __threadfence();
#pragma unroll
      for (int k = 0; k < K; ++k) {
        double y = x[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(kFull, y, o);
        if (lane == 0) csum[k][warp] = y;
      }
      if (__any_sync(kFull, bad) && lane == 0) *sbad = 1;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double y = 0.0;
      for (int w = 0; w < nw; ++w) y += csum[k][w];
      v[k] = y;
    }
    if (!direct && t < kCgCopies && *sbad == 0) {
      if (PUBLISH) __threadfence();
#pragma unroll
      for (int k = 0; k < K; ++k) put(tot + t * kCgLine + 2 * k, v[k]);
    }
  } else {
    if (t == 0) {
      double x[K];
#pragma unroll
      for (int k = 0; k < K; ++k) x[k] = 0.0;
      if (!get(tot + (blockIdx.x % kCgCopies) * kCgLine, x)) *sbad = 1;
      if (PUBLISH) __threadfence();
#pragma unroll
      for (int k = 0; k < K; ++k) csum[k][0] = x[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = csum[k][0];
  }
  const bool ok = *sbad == 0;
  __syncthreads();
  return ok;
}

template <class T, int E, bool DIA>
__global__ void __launch_bounds__(kCgThreads, 1) k_cg_small(CgSmallArgs<T> a) {
  if (a.st->done) return;
  __shared__ double wsum[2][kCgWarps], csum[2][8];
  __shared__ int sbad, offs[kDiaMaxDiag];
  const int t = threadIdx.x, n = a.A.n;
  const int row0 = blockIdx.x * (E * kCgThreads) + t;
  if (t == 0) sbad = 0;
  if (DIA && t < a.A.ndiag) offs[t] = a.A.d_off[t];
  __syncthreads();
  T x[E], r[E], p[E], s[E], q[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int i = row0 + e * kCgThreads;
    x[e] = i < n ? a.x[i] : T(0);
    r[e] = i < n ? a.r[i] : T(0);
    p[e] = i < n ? a.p[i] : T(0);
    s[e] = i < n ? a.s[i] : T(0);
    q[e] = T(0);
  }
  // the scalars of KState, the same in every thread of the grid
  const double bnorm = a.st->bnorm;
  double rho0 = a.st->rho0, alpha = a.st->alpha, beta = a.st->beta, gamma = a.st->gamma, rho1 = a.st->rho1,
         rnorm = a.st->rnorm;
  const int itrmax = a.st->itrmax;
  int itr = a.st->itr, done = 0, niter = 0, iret = 0, diverged = 0, breakdown = 0;
  const T *pold = a.p;
  T* pnew = a.p2;
  unsigned long long *w1 = a.slots, *w2 = a.slots + cg_small_slots(gridDim.x) / 2;
  bool ok = true;
  for (int k = 0; k < a.maxit && !done; ++k) {
    const unsigned tag = a.tag0 + (unsigned)k + 1u;
    const T al = (T)alpha, be = (T)beta;
#pragma unroll
    for (int e = 0; e < E; ++e) {   // x += alpha p; p = s + beta p
      const int i = row0 + e * kCgThreads;
      x[e] = x[e] + al * p[e];
      p[e] = s[e] + be * p[e];
      if (i < n) pnew[i] = p[e];
    }
    double pq[1] = {0.0};
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int i = row0 + e * kCgThreads;
      T sum = T(0);
      if (i < n) {
        // every load of a batch is issued before the first is used: one L2 round trip per
        // batch (a counted loop made it one per entry, half of the iteration)
        constexpr int U = 8;
        const int w = DIA ? a.A.ndiag : __ldg(a.A.s_w + (i >> 5));
        const int off = DIA ? 0 : __ldg(a.A.s_off + (i >> 5)) + (i & 31);
        const T* dv = DIA ? a.A.d_val + (int64_t)(i & ~31) * w + (i & 31) : a.A.s_val + off;
        for (int d0 = 0; d0 < w; d0 += U) {
          int c[U];
          T v[U], sv[U], pv[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const bool on = d0 + u < w;
            if constexpr (DIA) {
              c[u] = i + (on ? offs[d0 + u] : 0);
              c[u] = c[u] < 0 ? 0 : (c[u] >= n ? n - 1 : c[u]);   // out of the matrix: the stored value is zero
            } else {
              c[u] = on ? __ldg(a.A.s_col + off + 32 * (d0 + u)) : i;
            }
            v[u] = on ? __ldg(dv + 32 * (d0 + u)) : T(0);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const bool on = d0 + u < w;
            sv[u] = on ? __ldcg(a.s + c[u]) : T(0);
            pv[u] = on ? __ldcg(pold + c[u]) : T(0);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) sum += v[u] * (sv[u] + be * pv[u]);
        }
        pq[0] += (double)(p[e] * sum);
      }
      q[e] = sum;
    }
    if (!(ok = grid_sum<1, false>(pq, w1, tag, wsum, csum, &sbad))) break;
    gamma = pq[0];
    alpha = rho0 / gamma;
    const T na = (T)(-alpha);
    double d2[2] = {0.0, 0.0};
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int i = row0 + e * kCgThreads;
      r[e] = na * q[e] + r[e];
      s[e] = r[e];
      if (i < n) {
        if (a.dinv) s[e] = r[e] * __ldg(a.dinv + i);
        a.s[i] = s[e];
        d2[0] += (double)(s[e] * r[e]);
        d2[1] += (double)(r[e] * r[e]);
      }
    }
    if (!(ok = grid_sum<2, true>(d2, w2, tag, wsum, csum, &sbad))) break;
    // EPI_CG_DOT2's logic
    rho1 = d2[0];
    rnorm = sqrt(d2[1]);
    const double rel = rnorm / bnorm;
    if (rel < a.rtol) {
      done = 1; niter = min(itrmax, itr); iret = itrmax <= itr ? 1 : 0;
    } else if (rel > 1.0e8) {
      done = 1; diverged = 1; niter = min(itrmax, itr); iret = itrmax <= itr ? 1 : 0;
    } else if (!isfinite(rel) || !isfinite(rho1)) {
      done = 1; breakdown = 1; niter = min(itrmax, itr); iret = PARCEL_B_E_BREAKDOWN;
    } else {
      beta = rho1 / rho0;
      rho0 = rho1;
      if (itr + 1 > itrmax) {
        done = 1; niter = itrmax; iret = 1;
      } else {
        if (blockIdx.x == 0 && t == 0) a.hist[itr] = rnorm / bnorm;
        ++itr;
      }
    }
    T* o = const_cast<T*>(pold);
    pold = pnew;
    pnew = o;
  }
  if (!ok) {
    if (t == 0) atomicExch(a.err, 1);
    return;
  }
  // the second sum of the last iteration: no CTA reads p or s any more
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int i = row0 + e * kCgThreads;
    if (i < n) {
      a.x[i] = x[e];
      a.r[i] = r[e];
      a.p[i] = p[e];
    }
  }
  if (blockIdx.x == 0 && t == 0) {
    KState* st = a.st;
    st->rho0 = rho0; st->rho1 = rho1; st->gamma = gamma; st->alpha = alpha; st->beta = beta;
    st->tmp[0] = -alpha; st->rnorm = rnorm; st->itr = itr;
    st->niter = niter; st->iret = iret; st->diverged = diverged; st->breakdown = breakdown;
    st->done = done;
  }
}

template <class T, int E, bool DIA>
void launch(const CgSmallArgs<T>& a, int grid, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kCgThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  PB_CUDA(cudaLaunchKernelEx(&cfg, k_cg_small<T, E, DIA>, a));
}

inline int elems(int64_t n) {   // rows per thread: the fewest that need at most one CTA per SM
  const int64_t cap = (int64_t)std::min(num_sms(), 256) * kCgThreads;
  for (int e = 1; e <= kCgMaxElems; e *= 2)
    if (n <= cap * e) return e;
  return 0;
}

}  // namespace

// Which matrices take the launch.  Its 512 threads per SM walk their rows alone and gather two
// vectors per entry, so it wins while an iteration is launches and latency and loses once it is
// bandwidth: per iteration, one launch against three kernels (200 iterations, one B200, point
// Jacobi): 20,000 rows of 100 entries 23.3 / 24.9 us, 60,000 of 27 20.2 / 20.9, 300,000 of 9 29.1 /
// 32.1; 60,000 of 100 38.3 / 32.8, 150,000 of 27 37.9 / 32.5, 300,000 of 27 68.8 / 50.8, 150,000
// of 100 103 / 49.6.
constexpr int64_t kCgMaxEntries = 2000000;
constexpr int64_t kCgShortRow = 12;

template <class T>
int cg_small_grid(int64_t n, int64_t nnz) {
  if (nnz > kCgMaxEntries && nnz > kCgShortRow * n) return 0;
  const int e = elems(n);
  return e ? (int)((n + (int64_t)e * kCgThreads - 1) / ((int64_t)e * kCgThreads)) : 0;
}

template <class T>
void cg_small(const CgSmallArgs<T>& a, cudaStream_t st) {
  const int e = elems(a.A.n), g = cg_small_grid<T>(a.A.n, a.A.nnz);
  PB_CHECK(g > 0 && (a.A.d_val || a.A.s_val), PARCEL_B_E_ARG, "short-vector CG on %d rows", a.A.n);
#define CG_E(E_)                                                                    \
  if (a.A.d_val) launch<T, E_, true>(a, g, st); else launch<T, E_, false>(a, g, st);
  if (e == 1) { CG_E(1) } else if (e == 2) { CG_E(2) } else { CG_E(4) }
#undef CG_E
}

template int cg_small_grid<double>(int64_t, int64_t);
template int cg_small_grid<float>(int64_t, int64_t);
template void cg_small<double>(const CgSmallArgs<double>&, cudaStream_t);
template void cg_small<float>(const CgSmallArgs<float>&, cudaStream_t);

}  // namespace pb
