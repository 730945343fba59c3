// pb_ilu.cu -- block-Jacobi ILU(0) and D-ILU on B200.
//
// Reference algorithms (restated, not translated):
//   * blocks: contiguous row ranges from divide_region (src/common.f90:125-182);
//   * ILU(0): IKJ factorisation of each block's in-block submatrix, L unit-diagonal,
//     U with its diagonal (src/matrix.f90:7970-8072, 8249-8392); sweeps
//     solve_LU_crs (matrix.f90:8548-8747);
//   * D-ILU: K = (D+L) D^-1 (D+U) with D matched to the diagonal (ILUD) or the row sum
//     (MLUD) (DILU_DInv_crs, matrix.f90:3482-3648); sweeps solve_ILU_crs
//     (matrix.f90:4987-5163).
// The reference runs each block's sweeps sequentially on one OpenMP thread (CPU) or one
// cuSPARSE csrsv2 solve per process (src/CUDA/src/cusparse.cu:712-787).
//
// B200 design.  Rows of every block are grouped into wavefront levels (row i depends on
// the in-block rows it couples to with a smaller index), and the library stores every
// Krylov vector in a permuted, level-major layout where each level is contiguous and
// starts on a 16-byte boundary.  The plan and the layout are made on the device.  One CTA sweeps
// one block (many small blocks: a warp for one, two or four).  A producer warp streams groups
// of levels, packed coefficients and input-vector slice, into a ring of shared-memory stages
// with bulk asynchronous copies (cp.async.bulk + mbarrier); the consumer warps
// solve the level's rows from shared memory, keeping the last W levels of the solution in
// a shared-memory ring, so a level step costs shared-memory latency and one named
// barrier.  The arithmetic of every row is the reference's: same operands, same order.
#include <algorithm>
#include <cub/device/device_scan.cuh>
#include <climits>
#include <cmath>
#include <memory>
#include <numeric>
#include <type_traits>

#include "pb_device.cuh"
#include "pb_epilogue.cuh"
#include "pb_ilu.cuh"

namespace pb {

namespace {

// the plan looks for later levels when a ring of the early ones (gap + 1 of mean width) would
// hold more than this many rows: below it the ring fits beside the stages as it is
constexpr int64_t kTightenRing = 2048;

inline int align4(int x) { return (x + 3) & ~3; }
inline int64_t align16(int64_t x) { return (x + 15) & ~int64_t(15); }

void divide_region(int r, int np, long idown, long iup, long* lo, long* hi) {
  if (iup == idown) { *lo = idown; *hi = iup; return; }
  long region = iup - idown + 1, blk = region / np, over = region % np;
  if (r < over) { *lo = idown + blk * r + r; *hi = *lo + blk; }
  else { *lo = idown + blk * r + over; *hi = *lo + blk - 1; }
}

}  // namespace

void ilu_block_rows(int b, int nb, int n, int* lo, int* hi) {
  long l, h;
  divide_region(b, nb, 1, n, &l, &h);
  *lo = (int)(l - 1);
  *hi = (int)h;
}

// How a plan's sweep runs for values of one size: 2 grouped, 1 general with its ring in shared
// memory, 0 general without, -1 too wide for it; ring: entries of the grouped sweep's ring.
struct SweepForm {
  int rank;
  int64_t ring;
};
static SweepForm sweep_form(const IluPlan& P, int tsize);

// ------------------------------------------------------------------ wavefront plan
// Levels: row x waits for every in-block row y < x coupled to it in either direction
// (a lower entry of x, or an upper entry (y, x) of y), so one level order serves the
// forward and the backward sweep.  The dependency window W is the largest level gap of any
// coupling + 1.
//
// k_plan_levels: one CTA per block walks the block's rows PR at a time.  Levels of earlier rows
// are final; among the rows at hand, every row takes the largest level of what it waits for plus
// one until nothing changes.  The equations are acyclic and the levels only grow, so the
// reads of rows that change at the same time do no harm.  Rows that each wait for the row before
// them, as along a grid line, are taken in one prefix maximum per warp, and a row's neighbour in
// the plane before is final already, so a stencil's chunk takes few rounds.  What a round
// costs is block barriers and shared-memory latency: a row's couplings within the chunk are
// listed in shared memory once, and those that the other row lists as well (all, in a symmetric
// pattern) are read and not also pushed.  Where couplings make longer chains (a random band) a
// chunk gives up the rounds, after fewer of them than the chunk before if that did, and its warps
// take turns instead, each until its 32 rows are final.
// Everything that is not a chain is done for all rows at once by other kernels: gaps, positions.
// With positions and gaps inside one CTA or warp a block, two passes over the levels where the
// gap was 1 already, and a round per row on chains, the plan of few blocks took longer than on
// the host (copies of the structure and of the maps included): 160^3 in one block 71 ms on the
// host, 106 ms so, 17 ms now; 1,024 x 1,024 triangulated 13.7, 21.1, 4.0 ms; 100,000
// rows tridiagonal 2.1, 74.9, 3.0 ms; a random band of 9 in a million rows 16.7, about 390, 128
// ms (of a set-up of 1.4 s).
//
// When the early levels' gap makes the ring too long, they are moved as late as the rows'
// dependents allow, rows without dependents left where they are (every row with dependents to
// one below its lowest dependent): the same kernel on the mirrored order (LATE) finds every
// row's distance from the last level.  The number of levels and the validity of the order are
// unchanged (the longest chain has no slack); what changes is the largest gap.  A block that
// starts in the middle of a grid plane has rows that could start at once but are only needed
// a hundred levels later; with the levels taken as early as possible the ring of a
// 12,000-row block of a 61 x 53 x 47 stencil would hold 58 levels, tightened it holds 2, as for
// a block of whole planes, and the grouped sweep takes it instead of the general one, which
// gathers coupled values from global memory: applications back to back 147 -> 33 us there (16
// blocks; 119 -> 26 us inside a solve), 247 -> 53 us on 97 x 89 x 83 in 48 blocks.  The late
// levels are kept where they get the sweep a better form (sweep_form), or a grouped sweep a
// shorter ring: a shorter gap alone can come with levels so wide that the ring is longer, or that
// no sweep takes them (rows all over a chain whose only dependents are at its end move into one
// level).
constexpr int kPlanRounds = 48;
constexpr int kPlanRetry = 8;
constexpr int kPlanList = 16;      // couplings of a row within its chunk, each way, that are listed
constexpr int kPlanFar = 4;        // couplings to later chunks kept in registers
constexpr int kPlanBatch = 8;      // entries of a row loaded at once

struct PlanStat {
  int kmax, missing;   // missing: a block without a diagonal entry, or INT_MAX
};

// A block's early levels make its ring too long, and another order can help.
__host__ __device__ inline bool plan_loose(int gap, int rows, int nlev) {
  return gap > 1 && (int64_t)(gap + 1) * rows > kTightenRing * (int64_t)nlev;
}

// val: levels out (LATE: distances from the last level).  far (zeroed): scratch, one int per
// row.  wid (zeroed): level widths, block b's from its first row on.  LATE: lev, nlev and gap of
// the early levels, dep: rows that have dependents; blocks that are not loose are left out.
template <bool LATE, int PR>
__global__ void __launch_bounds__(PR, PR == 1024 ? 1 : 4)
    k_plan_levels(const int* __restrict__ starts, const int* __restrict__ rp, const int* __restrict__ ci, int rbase,
                  int cbase, int* val, int* far, int* wid, const int* __restrict__ lev,
                  const unsigned char* __restrict__ dep, const int* __restrict__ gap, int* nlev, PlanStat* stat) {
  extern __shared__ unsigned short plan_smem[];
  unsigned short(*before)[PR] = reinterpret_cast<unsigned short(*)[PR]>(plan_smem);
  unsigned short(*after)[PR] = before + kPlanList;
  __shared__ volatile int cur[PR];   // level of the chunk's rows
  __shared__ int push[PR];           // forced on them by couplings only the other row lists
  __shared__ unsigned short nbef[PR];   // listed couplings; kPlanList + 1: the row is read
  __shared__ int s_max, s_kmax;
  const int b = blockIdx.x, t = threadIdx.x;
  const int lo = starts[b], hi = starts[b + 1], m = hi - lo;
  if (LATE && !plan_loose(gap[b], m, nlev[b])) return;
  const int last = LATE ? nlev[b] - 1 : 0;
  if (t == 0) s_max = s_kmax = 0;
  auto row_of = [&](int u) { return LATE ? hi - 1 - u : lo + u; };   // u-th row of the walk
  auto walk_of = [&](int c) { return LATE ? hi - 1 - c : c - lo; };
  int kmax = 0, maxlev = 0, rounds = kPlanRounds;
  bool missing = false;
  for (int base = 0; base < m; base += PR) {
    const int u = base + t;
    const bool on = u < m;
    const int i = on ? row_of(u) : 0;
    const int a = on ? rp[i] - rbase : 0, z = on ? rp[i + 1] - rbase : 0;
    int L0 = on ? __ldcg(far + i) : 0;
    if (LATE && on && !dep[i]) L0 = last - lev[i];
    int nb = 0, na = 0, nf = 0, kl = 0, ku = 0, farc[kPlanFar];
    bool diag = false;
    // f(walk position) for every in-block entry off the diagonal
    auto entries = [&](int from, int to, int self, auto&& f) {
      for (int j0 = from; j0 < to; j0 += kPlanBatch) {
        int c[kPlanBatch];
#pragma unroll
        for (int e = 0; e < kPlanBatch; ++e) c[e] = j0 + e < to ? ci[j0 + e] - cbase : -1;
#pragma unroll
        for (int e = 0; e < kPlanBatch; ++e)
          if (c[e] >= lo && c[e] < hi && c[e] != self) f(walk_of(c[e]));
      }
    };
    for (int j0 = a; j0 < z; j0 += kPlanBatch) {
      int c[kPlanBatch], lv[kPlanBatch];
#pragma unroll
      for (int e = 0; e < kPlanBatch; ++e) c[e] = j0 + e < z ? ci[j0 + e] - cbase : -1;
#pragma unroll
      for (int e = 0; e < kPlanBatch; ++e) {
        const bool done = c[e] >= lo && c[e] < hi && walk_of(c[e]) < base;
        lv[e] = done ? __ldcg(val + c[e]) : -1;
      }
#pragma unroll
      for (int e = 0; e < kPlanBatch; ++e) {
        if (c[e] < lo || c[e] >= hi) continue;
        if (c[e] == i) { diag = true; continue; }
        const int v = walk_of(c[e]);
        L0 = max(L0, lv[e] + 1);
        if (v < u) {
          ++kl;
          if (v >= base) {
            if (nb < kPlanList) before[nb][t] = (unsigned short)(v - base);
            ++nb;
          }
        } else {
          ++ku;
          if (v < base + PR) {
            if (na < kPlanList) after[na][t] = (unsigned short)(v - base);
            ++na;
          } else {
#pragma unroll
            for (int q = 0; q < kPlanFar; ++q)
              if (q == nf) farc[q] = c[e];
            ++nf;
          }
        }
      }
    }
    kmax = max(kmax, max(kl, ku));
    missing |= on && !diag;
    const bool listed = nb <= kPlanList && na <= kPlanList;
    cur[t] = -1;
    push[t] = L0;
    nbef[t] = listed ? nb : kPlanList + 1;
    __syncthreads();
    if (listed) {   // drop the couplings that the other row reads
      int k = 0;
      for (int e = 0; e < na; ++e) {
        const int v = after[e][t], n = nbef[v];
        bool seen = n > kPlanList;   // it reads its whole row
        if (seen) {
          seen = false;
          entries(rp[row_of(base + v)] - rbase, rp[row_of(base + v) + 1] - rbase, -1, [&](int w) { seen |= w == u; });
        } else {
          for (int q = 0; q < n; ++q) seen |= before[q][v] == t;
        }
        if (!seen) after[k++][t] = (unsigned short)v;
      }
      na = k;
    }
    // how many rows before this one in the warp each wait for the one before them
    bool link = false;
    for (int e = 0; listed && e < nb; ++e) link |= before[e][t] == t - 1;
    const int run = __clz(~(__ballot_sync(kFull, link && (t & 31) != 0) << (31 - (t & 31))));
    const int longest = __reduce_max_sync(kFull, run);
    int mine = -1, changed, left = rounds;
    auto round = [&]() -> int {   // whole warps
      int L = on ? max(mine, *(volatile int*)&push[t]) : -1;
      if (listed) {
        for (int e = 0; e < nb; ++e) L = max(L, cur[before[e][t]] + 1);
      } else {
        entries(a, z, i, [&](int v) { if (v >= base && v < u) L = max(L, cur[v - base] + 1); });
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        if (o > longest) break;   // the same in every lane
        const int up = __shfl_up_sync(kFull, L, o);
        if (o <= run) L = max(L, up + o);
      }
      if (!on || L <= mine) return 0;
      mine = L;
      cur[t] = L;
      if (listed) {
        for (int e = 0; e < na; ++e) atomicMax(&push[after[e][t]], L + 1);
      } else {
        entries(a, z, i, [&](int v) { if (v > u && v < base + PR) atomicMax(&push[v - base], L + 1); });
      }
      return 1;
    };
    do changed = __syncthreads_or(round()); while (changed && --left > 0);
    rounds = changed ? kPlanRetry : kPlanRounds;
    if (changed) {   // a long chain: the warps in order, each until its rows are final
      for (int w = 0; w < PR / 32; ++w) {
        if ((t >> 5) == w) {
          int c;
          do {
            c = round();
            __syncwarp();
          } while (__any_sync(kFull, c));
        }
        __syncthreads();
      }
    }
    if (on) {
      val[i] = mine;
      maxlev = max(maxlev, mine);
      atomicAdd(wid + lo + (LATE ? last - mine : mine), 1);
      if (nf <= kPlanFar) {
#pragma unroll
        for (int q = 0; q < kPlanFar; ++q)
          if (q < nf) atomicMax(far + farc[q], mine + 1);
      } else {
        entries(a, z, i, [&](int v) { if (v >= base + PR) atomicMax(far + row_of(v), mine + 1); });
      }
    }
    __syncthreads();
  }
  if (LATE) return;
  atomicMax(&s_max, maxlev);
  atomicMax(&s_kmax, kmax);
  if (missing) atomicMin(&stat->missing, b);
  __syncthreads();
  if (t == 0) {
    nlev[b] = s_max + 1;
    atomicMax(&stat->kmax, s_kmax);
  }
}

__device__ __forceinline__ int plan_block(const int* __restrict__ starts, int nb, int i) {
  int a = 0, z = nb - 1;   // the last block that starts at or before row i
  while (a < z) {
    const int mid = (a + z + 1) >> 1;
    if (starts[mid] <= i) a = mid; else z = mid - 1;
  }
  return a;
}

// Largest level difference of a coupling of each block (gap, zeroed); dep, if given: the rows
// that have dependents.  only: the blocks that are loose by it (with nlev) are looked at.
__global__ void k_plan_gap(int n, int nb, const int* __restrict__ starts, const int* __restrict__ rp,
                           const int* __restrict__ ci, int rbase, int cbase, const int* __restrict__ val,
                           int* gap, unsigned char* __restrict__ dep, const int* __restrict__ only,
                           const int* __restrict__ nlev) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int b = plan_block(starts, nb, i), lo = starts[b], hi = starts[b + 1];
    if (only && !plan_loose(only[b], hi - lo, nlev[b])) continue;
    const int L = val[i];
    int g = 0;
    for (int j = rp[i] - rbase; j < rp[i + 1] - rbase; ++j) {
      const int c = ci[j] - cbase;
      if (c < lo || c >= hi || c == i) continue;
      if (dep) dep[min(c, i)] = 1;
      else g = max(g, abs(val[c] - L));
    }
    if (!dep && g > *(volatile int*)(gap + b)) atomicMax(gap + b, g);
  }
}

// Blocks whose late levels have the smaller gap take them (once the host has chosen that plan).
__global__ void k_plan_take(int n, int nb, const int* __restrict__ starts, const int* __restrict__ gap,
                            const int* __restrict__ gap_late, const int* __restrict__ nlev,
                            const int* __restrict__ late, int* __restrict__ lev) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int b = plan_block(starts, nb, i);
    if (plan_loose(gap[b], starts[b + 1] - starts[b], nlev[b]) && gap_late[b] < gap[b])
      lev[i] = nlev[b] - 1 - late[i];
  }
}

// Block b's level widths from wid (wid_late where its late levels are taken), from its first row
// on, to width[blvl[b]..].
__global__ void k_plan_widths(const int* __restrict__ starts, const int* __restrict__ blvl,
                              const int* __restrict__ wid, const int* __restrict__ wid_late,
                              const int* __restrict__ gap, const int* __restrict__ gap_late,
                              int* __restrict__ width) {
  const int b = blockIdx.x, lo = starts[b], l0 = blvl[b], n = blvl[b + 1] - l0;
  const bool late = wid_late && plan_loose(gap[b], starts[b + 1] - lo, n) && gap_late[b] < gap[b];
  for (int l = threadIdx.x; l < n; l += blockDim.x) width[l0 + l] = (late ? wid_late : wid)[lo + l];
}

// Positions: the rows of a level in natural order.  A segment is a run of one block's rows; its
// counters, one per level of the block, end as the position where the segment's rows of the
// level start: counted per segment, then summed over the segments of a block, level by level.
struct PlanSeg {
  int row0, row1;   // rows [row0, row1)
  int64_t ctr;      // first counter
};

__global__ void k_plan_count(int nseg, const PlanSeg* __restrict__ seg, const int* __restrict__ lev, int* ctr) {
  const int s = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (s >= nseg) return;
  const PlanSeg S = seg[s];
  for (int i = S.row0 + lane; i < S.row1; i += 32) atomicAdd(ctr + S.ctr + lev[i], 1);
}

__global__ void k_plan_scan(int totlev, int nb, const int* __restrict__ blvl, const int* __restrict__ blk_seg,
                            const PlanSeg* __restrict__ seg, const int* __restrict__ lst, int* __restrict__ ctr) {
  const int gl = blockIdx.x * blockDim.x + threadIdx.x;
  if (gl >= totlev) return;
  const int b = plan_block(blvl, nb, gl), l = gl - blvl[b], nl = blvl[b + 1] - blvl[b];
  const int s0 = blk_seg[b], ns = blk_seg[b + 1] - s0;
  int* c = ctr + seg[s0].ctr + l;   // a block's segments have their counters one after another
  int at = lst[gl];
  for (int s = 0; s < ns; s += 8) {
    int w[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) w[u] = s + u < ns ? c[(int64_t)(s + u) * nl] : 0;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (s + u < ns) {
        c[(int64_t)(s + u) * nl] = at;
        at += w[u];
      }
  }
}

// One warp per segment takes 32 rows at a time; rows of one level among them are ranked by
// lane, and the level's counter is where it goes on.
__global__ void k_plan_pos(int nseg, const PlanSeg* __restrict__ seg, const int* __restrict__ lev, int* ctr,
                           int* __restrict__ pos, int* __restrict__ rowAt) {
  const int s = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (s >= nseg) return;
  const PlanSeg S = seg[s];
  int* nx = ctr + S.ctr;
  int L = S.row0 + lane < S.row1 ? lev[S.row0 + lane] : -1;
  for (int base = S.row0; base < S.row1; base += 32) {
    const int i = base + lane;
    const int Ln = i + 32 < S.row1 ? lev[i + 32] : -1;   // on its way while this step runs
    const unsigned same = __match_any_sync(kFull, L);
    const int lead = __ffs(same) - 1, rank = __popc(same & ((1u << lane) - 1u));
    int at = 0;
    if (lane == lead && L >= 0) {   // one lane per level, this warp alone on the counters
      at = *(volatile int*)(nx + L);
      *(volatile int*)(nx + L) = at + __popc(same);
    }
    at = __shfl_sync(kFull, at, lead) + rank;
    if (L >= 0) {
      pos[i] = at;
      rowAt[at] = i;
    }
    __syncwarp();
    L = Ln;
  }
}

static int row_grid(int n) { return std::max(1, std::min((n + 255) / 256, 8 * num_sms())); }

template <bool LATE>
static void plan_levels(const DevMat<double>& A, int nb, int max_rows, const int* starts, int* val, int* far, int* wid,
                        const int* lev, const unsigned char* dep, const int* gap, int* nlev, PlanStat* stat) {
  auto go = [&](auto kern, int pr) {
    const size_t smem = sizeof(unsigned short) * 2 * kPlanList * pr;
    PB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<nb, pr, smem, stream()>>>(starts, A.rowptr, A.col, A.rbase, A.cbase, val, far, wid, lev, dep, gap, nlev, stat);
    PB_CUDA(cudaGetLastError());
  };
  // more than two blocks per SM: narrower CTAs, several to an SM
  if (max_rows <= 256 || nb > 2 * num_sms()) go(k_plan_levels<LATE, 256>, 256);
  else go(k_plan_levels<LATE, 1024>, 1024);
}

// pos and rowAt from the levels and their starts.
static void plan_positions(int nb, const std::vector<int>& starts, const std::vector<int>& blk_lvl, const int* d_blvl,
                           const int* d_lst, int totlev, const int* lev, int* pos, int* rowAt) {
  cudaStream_t st = stream();
  std::vector<PlanSeg> seg;
  std::vector<int> blk_seg(nb + 1, 0);
  seg.reserve(nb);
  int64_t ctrs = 0;
  for (int b = 0; b < nb; ++b) {
    blk_seg[b] = (int)seg.size();
    const int nl = blk_lvl[b + 1] - blk_lvl[b];
    const int len = std::max(1024, nl);   // so there are never more counters than rows and levels together
    for (int r = starts[b]; r < starts[b + 1]; r += len) {
      seg.push_back(PlanSeg{r, std::min(r + len, starts[b + 1]), ctrs});
      ctrs += nl;
    }
  }
  blk_seg[nb] = (int)seg.size();
  const int ns = (int)seg.size(), grid = (ns + 7) / 8;
  DBuf dseg, ctr;
  dseg.alloc(sizeof(PlanSeg) * seg.size(), false);
  h2d(dseg.p, seg.data(), sizeof(PlanSeg) * seg.size());
  ctr.alloc(sizeof(int) * (size_t)ctrs, ns > nb);
  if (ns > nb) {
    DBuf dbs;
    dbs.alloc(sizeof(int) * blk_seg.size(), false);
    h2d(dbs.p, blk_seg.data(), sizeof(int) * blk_seg.size());
    k_plan_count<<<grid, 256, 0, st>>>(ns, dp<PlanSeg>(dseg), lev, dp<int>(ctr));
    PB_CUDA(cudaGetLastError());
    k_plan_scan<<<(totlev + 255) / 256, 256, 0, st>>>(totlev, nb, d_blvl, dp<int>(dbs), dp<PlanSeg>(dseg), d_lst,
                                                      dp<int>(ctr));
    PB_CUDA(cudaGetLastError());
  } else {   // a segment per block: its counters are the level starts
    d2d(ctr.p, d_lst, sizeof(int) * (size_t)totlev);
  }
  k_plan_pos<<<grid, 256, 0, st>>>(ns, dp<PlanSeg>(dseg), lev, dp<int>(ctr), pos, rowAt);
  PB_CUDA(cudaGetLastError());
}

// What depends on the levels' widths and gaps: level starts (multiples of 4, in block order) and the
// sizes of ring and layout.
static void plan_layout(IluPlan& P, const std::vector<int>& width, const std::vector<int>& gap) {
  int64_t total = 0;
  for (int w : width) total += align4(w);
  PB_CHECK(total <= INT_MAX - 3, PARCEL_B_E_ARG, "the permuted layout of %d rows exceeds 2^31 entries", P.n);
  P.lvl_start.resize(width.size());
  P.lvl_end.resize(width.size());
  int cursor = 0, maxw = 0;
  for (size_t l = 0; l < width.size(); ++l) {
    P.lvl_start[l] = cursor;
    P.lvl_end[l] = cursor + width[l];
    maxw = std::max(maxw, width[l]);
    cursor = align4(cursor + width[l]);
  }
  P.np = (int)total;   // the last level is padded as well
  P.maxWp = align4(maxw);
  P.W = *std::max_element(gap.begin(), gap.end()) + 1;
}

bool ilu_build_plan(const DevMat<double>& A, const BlockSplit& blocks, Tighten tighten, int tsize, IluPlan& P,
                    DBuf& pos, DBuf& rowAt, DBuf& lev) {
  cudaStream_t st = stream();
  const int n = A.n, nb = blocks.nb;
  P.n = n;
  P.nb = nb;
  P.blk_lo.resize(nb);
  P.blk_hi.resize(nb);
  std::vector<int> starts(nb + 1, n);
  int max_rows = 0;
  for (int b = 0; b < nb; ++b) {
    blocks.rows(b, n, &P.blk_lo[b], &P.blk_hi[b]);
    starts[b] = P.blk_lo[b];
    max_rows = std::max(max_rows, P.blk_hi[b] - P.blk_lo[b]);
  }
  const size_t ib = sizeof(int) * (size_t)n;
  DBuf dstarts(sizeof(int) * (nb + 1)), far(ib), wid(ib), dnlev(sizeof(int) * nb), dgap(sizeof(int) * nb),
      dstat(sizeof(PlanStat));
  lev.alloc(ib, false);
  PlanStat h{0, INT_MAX};
  h2d(dstarts.p, starts.data(), sizeof(int) * (nb + 1));
  h2d(dstat.p, &h, sizeof(h));
  plan_levels<false>(A, nb, max_rows, dp<int>(dstarts), dp<int>(lev), dp<int>(far), dp<int>(wid), nullptr, nullptr,
                     nullptr, dp<int>(dnlev), dp<PlanStat>(dstat));
  k_plan_gap<<<row_grid(n), 256, 0, st>>>(n, nb, dp<int>(dstarts), A.rowptr, A.col, A.rbase, A.cbase, dp<int>(lev),
                                          dp<int>(dgap), nullptr, nullptr, nullptr);
  PB_CUDA(cudaGetLastError());
  std::vector<int> nlev(nb), gap(nb);
  PB_CUDA(cudaMemcpyAsync(nlev.data(), dnlev.p, sizeof(int) * nb, cudaMemcpyDeviceToHost, st));
  PB_CUDA(cudaMemcpyAsync(gap.data(), dgap.p, sizeof(int) * nb, cudaMemcpyDeviceToHost, st));
  d2h(&h, dstat.p, sizeof(h));
  PB_CHECK(h.missing == INT_MAX, PARCEL_B_E_ZERO_PIVOT,
           "block-Jacobi block %d has a row without an in-block diagonal entry", h.missing);
  P.kmax = h.kmax;
  P.max_levels = *std::max_element(nlev.begin(), nlev.end());
  P.blk_lvl.assign(nb + 1, 0);
  for (int b = 0; b < nb; ++b) P.blk_lvl[b + 1] = P.blk_lvl[b] + nlev[b];
  const int totlev = P.blk_lvl[nb];
  DBuf dblvl(sizeof(int) * (nb + 1)), dwidth(sizeof(int) * std::max(totlev, 1));
  h2d(dblvl.p, P.blk_lvl.data(), sizeof(int) * (nb + 1));
  std::vector<int> width(totlev);
  auto widths = [&](const int* wid_late, const int* gap_late) {
    k_plan_widths<<<nb, 256, 0, st>>>(dp<int>(dstarts), dp<int>(dblvl), dp<int>(wid), wid_late, dp<int>(dgap), gap_late,
                                      dp<int>(dwidth));
    PB_CUDA(cudaGetLastError());
    d2h(width.data(), dwidth.p, sizeof(int) * totlev);
  };
  widths(nullptr, nullptr);
  plan_layout(P, width, gap);
  bool loose = false, moved = false;
  for (int b = 0; b < nb; ++b) loose |= plan_loose(gap[b], starts[b + 1] - starts[b], nlev[b]);
  if (loose && tighten != Tighten::no) {
    DBuf dep(n), wid_late(ib), gap_late(sizeof(int) * nb), late;
    late.alloc(ib, false);
    far.zero_fill();
    k_plan_gap<<<row_grid(n), 256, 0, st>>>(n, nb, dp<int>(dstarts), A.rowptr, A.col, A.rbase, A.cbase, dp<int>(lev),
                                            dp<int>(dgap), dp<unsigned char>(dep), dp<int>(dgap), dp<int>(dnlev));
    PB_CUDA(cudaGetLastError());
    plan_levels<true>(A, nb, max_rows, dp<int>(dstarts), dp<int>(late), dp<int>(far), dp<int>(wid_late), dp<int>(lev),
                      dp<unsigned char>(dep), dp<int>(dgap), dp<int>(dnlev), nullptr);
    k_plan_gap<<<row_grid(n), 256, 0, st>>>(n, nb, dp<int>(dstarts), A.rowptr, A.col, A.rbase, A.cbase, dp<int>(late),
                                            dp<int>(gap_late), nullptr, dp<int>(dgap), dp<int>(dnlev));
    PB_CUDA(cudaGetLastError());
    std::vector<int> g2(nb);
    d2h(g2.data(), gap_late.p, sizeof(int) * nb);
    bool any = false;
    for (int b = 0; b < nb; ++b)
      if (plan_loose(gap[b], starts[b + 1] - starts[b], nlev[b]) && g2[b] < gap[b]) {
        gap[b] = g2[b];
        any = true;
      }
    if (any) {
      IluPlan Q = P;
      widths(dp<int>(wid_late), dp<int>(gap_late));
      plan_layout(Q, width, gap);
      const SweepForm f = sweep_form(P, tsize), g = sweep_form(Q, tsize);
      moved = g.rank > f.rank || (tighten == Tighten::shorter && g.rank == 2 && f.rank == 2 && g.ring < f.ring);
      if (moved) {
        P = std::move(Q);
        k_plan_take<<<row_grid(n), 256, 0, st>>>(n, nb, dp<int>(dstarts), dp<int>(dgap), dp<int>(gap_late),
                                                 dp<int>(dnlev), dp<int>(late), dp<int>(lev));
        PB_CUDA(cudaGetLastError());
      }
    }
  }
  pos.alloc(ib, false);
  rowAt.alloc(sizeof(int) * (size_t)P.np, false);
  PB_CUDA(cudaMemsetAsync(rowAt.p, 0xFF, sizeof(int) * (size_t)P.np, st));   // padding: -1
  DBuf dlst(sizeof(int) * std::max(totlev, 1));
  h2d(dlst.p, P.lvl_start.data(), sizeof(int) * totlev);
  plan_positions(nb, starts, P.blk_lvl, dp<int>(dblvl), dp<int>(dlst), totlev, dp<int>(lev), dp<int>(pos),
                 dp<int>(rowAt));
  sync();   // the temporaries above are released on return
  return tighten == Tighten::no ? loose : moved;
}

// Largest chunk, and the most consumer threads of the grouped sweep, for records of K couplings
// of tsize bytes.  A thread holds two rows' operands.  With 512 consumers and the producer warp an
// SM partition has five warps and a thread 96 registers, with 480 four warps and 128, with 352
// three and 168.  At 96 the wide records spilled 172 to 1,164 bytes: 15-point stencil, 96^3 in 24
// blocks (seven couplings, levels of up to 372 rows), 264 us per application, 168 at 128 registers
// (178 before rows were staged ahead); double-double 13-point, 48 x 48 x 96 in 8 blocks (levels of
// up to 540 rows), 20 iterations 14.5 ms at 96, 9.7 at 128, 8.9 at 168.  Narrower records fit 96
// registers and keep the longer chunk.
constexpr int grp_rows(int tsize, int K) {
  if (tsize == 16 && K <= 6) return K > 4 ? 352 : (K > 2 ? 480 : kIluChunk);
  return tsize == 8 && (K == 7 || K == 8) ? 480 : kIluChunk;
}

// The plan's chunks (a level split at `rows` rows), in block order; K couplings per row in
// their records.  blk_chunk: nb + 1.
static std::vector<IluChunk> plan_chunks(const IluPlan& P, int rows, int K, std::vector<int>& blk_chunk) {
  size_t n = 0;
  for (size_t l = 0; l < P.lvl_start.size(); ++l) n += (P.lvl_end[l] - P.lvl_start[l] + rows - 1) / rows;
  std::vector<IluChunk> ch(n);
  blk_chunk.assign(P.nb + 1, 0);
  int c = 0;
  for (int b = 0; b < P.nb; ++b) {
    blk_chunk[b] = c;
    for (int gl = P.blk_lvl[b]; gl < P.blk_lvl[b + 1]; ++gl) {
      const int w = P.lvl_end[gl] - P.lvl_start[gl];
      for (int o = 0; o < w; o += rows) {
        IluChunk& C = ch[c++];
        C.start = P.lvl_start[gl] + o;
        C.w = std::min(rows, w - o);
        C.wpad = align4(C.w);
        C.KL = C.KU = K;
        C.lvl = gl - P.blk_lvl[b];
        C.off_in_level = o;
        C.blk = b;
        C.offF = 0;
        C.offB = 0;
      }
    }
  }
  blk_chunk[P.nb] = c;
  return ch;
}

// ------------------------------------------------------------------ factorisation
// In-block column range of natural row i (columns sorted): [first, last) positions.
__device__ __forceinline__ void inblock_range(const int* rp, const int* ci, int rbase, int cbase,
                                              int i, int lo, int hi, int* ja, int* jz, int* jd) {
  int a = rp[i] - rbase, z = rp[i + 1] - rbase;
  int s = z, e = z, d = -1;
  for (int j = a; j < z; ++j) {
    int c = ci[j] - cbase;
    if (c >= lo && s == z) s = j;
    if (c >= hi) { e = j; break; }
    if (c == i) d = j;
  }
  if (s > e) s = e;
  *ja = s; *jz = e; *jd = d;
}

// ILU(0) IKJ factorisation of every block, level by level; one CTA per block.
// ILU_LU_crs (matrix.f90:7970-8072).  Explicit roundings keep the reference's
// two-rounding a - b*c.
//
// A row of at most kFacCap entries is staged in registers: its columns and values in one
// batch of loads, then for each lower in-block entry (increasing column) the pivot row in
// one batch; the eliminations run on the registers in the reference's order and the row
// is written back once.  Longer rows (or pivot rows) take the entry-by-entry path.
constexpr int kFacCap = 8;

// Levels [start, end) in the iteration layout; block b has levels blvl[b] .. blvl[b + 1] - 1.
struct LevelTab {
  const int *blvl, *start, *end;
};

__device__ __forceinline__ void ilu0_row_generic(const int* rp, const int* ci, int rbase, int cbase, int i, int lo, int hi,
                                 double* lu) {
  int ia, iz, idg;
  inblock_range(rp, ci, rbase, cbase, i, lo, hi, &ia, &iz, &idg);
  for (int kc = ia; kc < iz; ++kc) {
    int k = ci[kc] - cbase;
    if (k > i - 1) break;
    int ka, kz, kk;
    inblock_range(rp, ci, rbase, cbase, k, lo, hi, &ka, &kz, &kk);
    double lik = __ddiv_rn(lu[kc], lu[kk]);
    lu[kc] = lik;
    for (int jc = kc + 1; jc < iz; ++jc) {
      int j = ci[jc] - cbase;
      for (int kj = kk; kj < kz; ++kj) {
        int cj = ci[kj] - cbase;
        if (cj == j) { lu[jc] = __dsub_rn(lu[jc], __dmul_rn(lik, lu[kj])); break; }
        if (cj > j) break;
      }
    }
  }
}

__global__ void k_ilu0_factor(LevelTab tab, const int* __restrict__ blk_lo, const int* __restrict__ blk_hi,
                              const int* __restrict__ rowAt, const int* __restrict__ rp,
                              const int* __restrict__ ci, int rbase, int cbase, double* lu) {
  const int b = blockIdx.x;
  const int lo = blk_lo[b], hi = blk_hi[b];
  for (int l = tab.blvl[b]; l < tab.blvl[b + 1]; ++l) {
    const int e = tab.end[l];
    for (int p = tab.start[l] + threadIdx.x; p < e; p += blockDim.x) {
      const int i = rowAt[p];
      const int a = rp[i] - rbase, z = rp[i + 1] - rbase;
      if (z - a > kFacCap) {
        ilu0_row_generic(rp, ci, rbase, cbase, i, lo, hi, lu);
        continue;
      }
      int col[kFacCap];
      double val[kFacCap];
#pragma unroll
      for (int e = 0; e < kFacCap; ++e) {
        col[e] = e < z - a ? ci[a + e] - cbase : INT_MAX;
        val[e] = e < z - a ? lu[a + e] : 0.0;
      }
      // pivot rows must fit as well; otherwise the whole row goes the generic way.  Their
      // bounds are kept for the eliminations.
      bool fits = true;
      int pa[kFacCap], pz[kFacCap];
#pragma unroll
      for (int e = 0; e < kFacCap; ++e) {
        const int k = col[e];
        pa[e] = 0;
        pz[e] = 0;
        if (k >= lo && k < i) {
          pa[e] = rp[k] - rbase;
          pz[e] = rp[k + 1] - rbase;
          if (pz[e] - pa[e] > kFacCap) fits = false;
        }
      }
      if (!fits) {
        ilu0_row_generic(rp, ci, rbase, cbase, i, lo, hi, lu);
        continue;
      }
      // e walks the row; the register arrays are only ever indexed by unrolled loops
      for (int e = 0; e < z - a; ++e) {
        int k = INT_MAX, ka = 0, kz = 0;
        double ve = 0.0;
#pragma unroll
        for (int q = 0; q < kFacCap; ++q)
          if (q == e) { k = col[q]; ve = val[q]; ka = pa[q]; kz = pz[q]; }
        if (k < lo || k >= i) continue;   // lower in-block entries only, increasing column
        int kcol[kFacCap];
        double kval[kFacCap];
#pragma unroll
        for (int f = 0; f < kFacCap; ++f) {
          kcol[f] = f < kz - ka ? ci[ka + f] - cbase : INT_MAX;
          kval[f] = f < kz - ka ? lu[ka + f] : 0.0;
        }
        double ukk = 0.0;
#pragma unroll
        for (int f = 0; f < kFacCap; ++f)
          if (kcol[f] == k) ukk = kval[f];
        const double lik = __ddiv_rn(ve, ukk);
        // l_ik replaces a_ik; the in-block entries after it lose l_ik u_kj where row k
        // has column j (> k)
#pragma unroll
        for (int g = 0; g < kFacCap; ++g) {
          if (g == e) val[g] = lik;
          const int j = col[g];
#pragma unroll
          for (int f = 0; f < kFacCap; ++f)
            if (g > e && kcol[f] == j && j > k && j < hi) val[g] = __dsub_rn(val[g], __dmul_rn(lik, kval[f]));
        }
      }
#pragma unroll
      for (int e = 0; e < kFacCap; ++e)
        if (e < z - a) lu[a + e] = val[e];
    }
    __syncthreads();
  }
}

__global__ void k_dilu_diag(LevelTab tab, const int* __restrict__ blk_lo, const int* __restrict__ blk_hi,
                            const int* __restrict__ rowAt, const int* __restrict__ rp,
                            const int* __restrict__ ci, const double* __restrict__ va, int rbase,
                            int cbase, int mlud, double* D, double* Dinv) {
  const int b = blockIdx.x;
  const int lo = blk_lo[b], hi = blk_hi[b];
  for (int l = tab.blvl[b]; l < tab.blvl[b + 1]; ++l) {
    const int e = tab.end[l];
    for (int p = tab.start[l] + threadIdx.x; p < e; p += blockDim.x) {
      int k = rowAt[p];
      int ia, iz, idg;
      inblock_range(rp, ci, rbase, cbase, k, lo, hi, &ia, &iz, &idg);
      double d = va[idg];
      for (int jr = ia; jr < idg; ++jr) {
        int kr = ci[jr] - cbase;
        int ra, rz, rd;
        inblock_range(rp, ci, rbase, cbase, kr, lo, hi, &ra, &rz, &rd);
        double dk = D[kr];
        for (int i = ra; i < rz; ++i) {
          int rc = ci[i] - cbase;
          if (!mlud) {
            if (rc == k) { d = __dsub_rn(d, __ddiv_rn(__dmul_rn(va[jr], va[i]), dk)); break; }
          } else if (kr < rc) {
            d = __dsub_rn(d, __ddiv_rn(__dmul_rn(va[jr], va[i]), dk));
          }
        }
      }
      D[k] = d;
      Dinv[k] = __ddiv_rn(1.0, d);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ packing
// Packed chunk layout (bytes, every section 16-byte aligned):
//   header int[8] = {start, w, wpad, K, lvl, off_in_level, 0, 0}
//   header int[6] = ring offset of the chunk's first row: (lvl % W) * maxWp + off_in_level
//   diag   T[wpad]          forward: 1 (ILU(0)) or D^-1 (D-ILU); backward: 1/U_kk or D^-1
//   val    T[K * wpad]      entry k of row p at k*wpad + p
//   slot   int[K * wpad]    ring slot (or permuted position) of the coupled row, -1 = none
template <class T>
__host__ __device__ inline int64_t chunk_bytes(int wpad, int K) {
  return kIluHeader + (int64_t)wpad * sizeof(T) * (1 + K) + (int64_t)4 * K * wpad;
}

template <class T>
__global__ void k_ilu_pack(const IluChunk* __restrict__ ch, int nchunks,
                           const int* __restrict__ blk_lo, const int* __restrict__ blk_hi,
                           const int* __restrict__ blk_lvl, const int* __restrict__ lvl_start,
                           const int* __restrict__ rowAt, const int* __restrict__ pos,
                           const int* __restrict__ lev, const int* __restrict__ rp,
                           const int* __restrict__ ci, int rbase, int cbase,
                           const double* __restrict__ vL,    // values of L entries
                           const double* __restrict__ vU,    // values of U entries
                           const double* __restrict__ Dinv,  // D-ILU only
                           int dilu, int ring, int W, int maxWp,
                           unsigned char* packF, unsigned char* packB) {
  for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
    const IluChunk C = ch[c];
    const int lo = blk_lo[C.blk], hi = blk_hi[C.blk];
    unsigned char* f = packF + C.offF;
    unsigned char* g = packB + C.offB;
    if (threadIdx.x == 0) {
      int* hf = (int*)f;
      int* hb = (int*)g;
      hf[0] = C.start; hf[1] = C.w; hf[2] = C.wpad; hf[3] = C.KL; hf[4] = C.lvl;
      hf[5] = C.off_in_level; hf[6] = (C.lvl % W) * maxWp + C.off_in_level; hf[7] = 0;
      hb[0] = C.start; hb[1] = C.w; hb[2] = C.wpad; hb[3] = C.KU; hb[4] = C.lvl;
      hb[5] = C.off_in_level; hb[6] = (C.lvl % W) * maxWp + C.off_in_level; hb[7] = 0;
    }
    T* dF = (T*)(f + kIluHeader);
    T* valF = dF + C.wpad;
    int* slF = (int*)(valF + (size_t)C.KL * C.wpad);
    T* dB = (T*)(g + kIluHeader);
    const int zslot = ring ? W * maxWp : -1;   // ring mode: a slot that always holds 0
    T* valB = dB + C.wpad;
    int* slB = (int*)(valB + (size_t)C.KU * C.wpad);
    for (int p = threadIdx.x; p < C.wpad; p += blockDim.x) {
      if (p >= C.w) {
        dF[p] = (T)0; dB[p] = (T)0;
        for (int k = 0; k < C.KL; ++k) { valF[k * C.wpad + p] = (T)0; slF[k * C.wpad + p] = zslot; }
        for (int k = 0; k < C.KU; ++k) { valB[k * C.wpad + p] = (T)0; slB[k * C.wpad + p] = zslot; }
        continue;
      }
      int i = rowAt[C.start + p];
      int ia, iz, idg;
      inblock_range(rp, ci, rbase, cbase, i, lo, hi, &ia, &iz, &idg);
      auto slot_of = [&](int cnat) -> int {
        int q = pos[cnat];
        if (!ring) return q;
        int l = lev[cnat];
        return (l % W) * maxWp + (q - lvl_start[blk_lvl[C.blk] + l]);
      };
      // forward: strictly lower in-block entries, increasing column
      int k = 0;
      for (int j = ia; j < idg; ++j, ++k) {
        valF[k * C.wpad + p] = (T)vL[j];
        slF[k * C.wpad + p] = slot_of(ci[j] - cbase);
      }
      for (; k < C.KL; ++k) { valF[k * C.wpad + p] = (T)0; slF[k * C.wpad + p] = zslot; }
      dF[p] = dilu ? (T)Dinv[i] : (T)1;
      // backward: strictly upper in-block entries; ILU(0) increasing column
      // (solve_LU_crs), D-ILU decreasing column (solve_ILU_crs runs Ustart down to Uend)
      k = 0;
      if (!dilu) {
        for (int j = idg + 1; j < iz; ++j, ++k) {
          valB[k * C.wpad + p] = (T)vU[j];
          slB[k * C.wpad + p] = slot_of(ci[j] - cbase);
        }
        dB[p] = (T)(1.0 / vU[idg]);   // reciprocal of U_kk: the sweep multiplies
      } else {
        for (int j = iz - 1; j > idg; --j, ++k) {
          valB[k * C.wpad + p] = (T)vU[j];
          slB[k * C.wpad + p] = slot_of(ci[j] - cbase);
        }
        dB[p] = (T)Dinv[i];
      }
      for (; k < C.KU; ++k) { valB[k * C.wpad + p] = (T)0; slB[k * C.wpad + p] = zslot; }
    }
  }
}

// ------------------------------------------------------------------ grouped sweep
// The fast sweep streams GROUPS of consecutive chunks (levels, or 512-row pieces of a
// level) of one block: one bulk copy of the group's packed record plus one of its slice of
// the input vector fills one shared-memory stage, so the consumers wait on a stage
// barrier once per group and, between levels, pass only the level barrier.  The rows of a
// group are contiguous in the permuted layout ([sstart, sstart + sspan)).  Group record:
//   int4 hdr              {nchunks, sstart, xoff, 0}: xoff is the byte offset of the input
//                         slice in the stage
//   int4 cd[kGrpMax]      per chunk in sweep order, ready to add: {byte offset of the first
//                         row's record in the stage, rows - 1, ring byte offset of the first
//                         row, byte offset of the first row in the input slice}
//   row records           one per position of the span, `stride` bytes apart:
//                           T dg        1/U_kk or D^-1 (backward sweep, forward D-ILU only)
//                           T val[K]    coupled coefficients in the reference's order
//                           u16 slot[K] ring byte offsets of the coupled rows (the ring's
//                                       zero slot for padding)
//                         padded to an odd number of T-sized words, so that the 32 lanes
//                         of a warp reading consecutive records hit distinct banks.
// The stage holds T xin[sspan] (the input slice) after the records, 16-byte aligned.
// Positions without a row (level padding) have no record contents.
constexpr int kGrpMax = 31;
constexpr int kGrpHdr = 16 + kGrpMax * 16;

__host__ __device__ constexpr int rec_words(int tsize, bool has_dg, int K) {
  return ((has_dg ? 1 : 0) + K + (2 * K + tsize - 1) / tsize) | 1;
}
__host__ __device__ constexpr int rec_stride(int tsize, bool has_dg, int K) {
  return rec_words(tsize, has_dg, K) * tsize;
}

// Where a row's value sits in the shared-memory ring: the last W levels, or the whole block
// by position (W = 0), whichever is smaller.
struct RingMap {
  int W, maxWp;
  __host__ __device__ int at(int lvl, int off_in_level, int off_in_block) const {
    return W > 0 ? (lvl % W) * maxWp + off_in_level : off_in_block;
  }
};

// Sweep coefficients of the packed records: L and U entries by position in the natural
// matrix, and the diagonal factors of row nat (diagonal entry jd).
template <class T>
struct FpSrc {
  const double *vL, *vU, *Dinv;   // Dinv: D-ILU only
  __device__ T low(int j) const { return (T)vL[j]; }
  __device__ T up(int j) const { return (T)vU[j]; }
  __device__ T fwd(int nat) const { return (T)Dinv[nat]; }
  // ILU(0): the reciprocal of U_kk, the sweep multiplies
  __device__ T bwd(int nat, int jd) const { return Dinv ? (T)Dinv[nat] : (T)(1.0 / vU[jd]); }
};
struct DdSrc {
  const double *ah, *al, *dih, *dil;   // al and dil null: low parts zero
  __device__ dd low(int j) const { return dd{ah[j], al ? al[j] : 0.0}; }
  __device__ dd up(int j) const { return low(j); }
  __device__ dd fwd(int nat) const { return dd{dih[nat], dil ? dil[nat] : 0.0}; }
  __device__ dd bwd(int nat, int) const { return fwd(nat); }
};

// Coefficient and ring value of a padding entry.  The sums add a zero product; the
// double-double ones leave the entry out, and a factor of one keeps it on the short product.
template <class T> __device__ __forceinline__ T pad_coef() { return T(0); }
template <> __device__ __forceinline__ dd pad_coef<dd>() { return dd{1.0, 0.0}; }

// Packs the group records of the grouped sweep (layout above): one CTA per group;
// gi[g] = {first chunk, end chunk, sstart, sspan}, goff[g] = byte offsets of the forward
// and backward records.
template <class T, class Src>
__global__ void k_ilu_pack_grp(const int4* __restrict__ gi, const int64_t* __restrict__ goff, int ngroups,
                               const IluChunk* __restrict__ ch, const int* __restrict__ blk_lo,
                               const int* __restrict__ blk_hi, const int* __restrict__ blk_lvl,
                               const int* __restrict__ lvl_start, const int* __restrict__ rowAt,
                               const int* __restrict__ pos, const int* __restrict__ lev,
                               const int* __restrict__ rp, const int* __restrict__ ci, int rbase, int cbase,
                               Src src, int dilu, RingMap ring, int zslot, int K,
                               unsigned char* packF, unsigned char* packB) {
  const int sz = (int)sizeof(T);
  const int strF = rec_stride(sz, dilu != 0, K), strB = rec_stride(sz, true, K);
  for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
    const int4 G = gi[g];
    const int c0 = G.x, c1 = G.y, sstart = G.z, sspan = G.w;
    const int nch = c1 - c0;
    const int blk = ch[c0].blk;
    const int lo = blk_lo[blk], hi = blk_hi[blk];
    const int bstart = lvl_start[blk_lvl[blk]];   // the block's first position
    unsigned char* f = packF + goff[2 * g];
    unsigned char* bk = packB + goff[2 * g + 1];
    const int xF = kGrpHdr + (int)(((int64_t)sspan * strF + 15) & ~int64_t(15));
    const int xB = kGrpHdr + (int)(((int64_t)sspan * strB + 15) & ~int64_t(15));
    for (int t = threadIdx.x; t < kGrpHdr / 16; t += blockDim.x) {
      int4 hf = make_int4(0, 0, 0, 0), hb = make_int4(0, 0, 0, 0);
      if (t == 0) {
        hf = make_int4(nch, sstart, xF, 0);
        hb = make_int4(nch, sstart, xB, 0);
      } else if (t - 1 < nch) {
        auto desc = [&](const IluChunk& c, int str) {
          return make_int4(kGrpHdr + (c.start - sstart) * str, c.w - 1,
                           ring.at(c.lvl, c.off_in_level, c.start - bstart) * sz, (c.start - sstart) * sz);
        };
        hf = desc(ch[c0 + t - 1], strF);   // forward: increasing level
        hb = desc(ch[c1 - t], strB);       // backward: decreasing level
      }
      reinterpret_cast<int4*>(f)[t] = hf;
      reinterpret_cast<int4*>(bk)[t] = hb;
    }
    for (int i = threadIdx.x; i < sspan; i += blockDim.x) {
      unsigned char* rf = f + kGrpHdr + (size_t)i * strF;
      unsigned char* rb = bk + kGrpHdr + (size_t)i * strB;
      T* valF = reinterpret_cast<T*>(rf + (dilu ? sz : 0));
      unsigned short* slF = reinterpret_cast<unsigned short*>(rf + (dilu ? sz : 0) + K * sz);
      T* valB = reinterpret_cast<T*>(rb + sz);
      unsigned short* slB = reinterpret_cast<unsigned short*>(rb + sz + K * sz);
      const int nat = rowAt[sstart + i];
      if (nat < 0) continue;   // level padding: never read
      int ia, iz, idg;
      inblock_range(rp, ci, rbase, cbase, nat, lo, hi, &ia, &iz, &idg);
      auto slot_of = [&](int cnat) -> int {
        const int l = lev[cnat], q = pos[cnat];
        return ring.at(l, q - lvl_start[blk_lvl[blk] + l], q - bstart) * sz;
      };
      // forward: strictly lower in-block entries, increasing column
      int k = 0;
      for (int j = ia; j < idg; ++j, ++k) {
        valF[k] = src.low(j);
        slF[k] = (unsigned short)slot_of(ci[j] - cbase);
      }
      for (; k < K; ++k) { valF[k] = pad_coef<T>(); slF[k] = (unsigned short)zslot; }
      if (dilu) *reinterpret_cast<T*>(rf) = src.fwd(nat);
      // backward: strictly upper in-block entries; ILU(0) increasing column
      // (solve_LU_crs), D-ILU decreasing column (solve_ILU_crs runs Ustart down to Uend)
      k = 0;
      if (!dilu) {
        for (int j = idg + 1; j < iz; ++j, ++k) {
          valB[k] = src.up(j);
          slB[k] = (unsigned short)slot_of(ci[j] - cbase);
        }
      } else {
        for (int j = iz - 1; j > idg; --j, ++k) {
          valB[k] = src.up(j);
          slB[k] = (unsigned short)slot_of(ci[j] - cbase);
        }
      }
      *reinterpret_cast<T*>(rb) = src.bwd(nat, idg);
      for (; k < K; ++k) { valB[k] = pad_coef<T>(); slB[k] = (unsigned short)zslot; }
    }
  }
}

// ------------------------------------------------------------------ the sweep kernel
constexpr int kIluProducerWarps = 1;
constexpr int kIluConsumerThreads = 256;
constexpr int kIluThreads = 32 * kIluProducerWarps + kIluConsumerThreads;
constexpr unsigned kWaitLimit = 1u << 20;   // polls of one mbarrier wait before giving up
constexpr int kIluKUnroll = 4;            // coupled entries gathered per step

// What the producer needs per chunk, in the order it streams them:
// {packed offset / 16, first permuted row, packed bytes, vector-slice bytes}.
struct ProdDesc { int off16, start, cbytes, vbytes; };

template <class T>
struct IluSolveArgs {
  const ProdDesc* tabF;   // per chunk, forward order
  const ProdDesc* tabB;   // per chunk, forward order (read backwards)
  const int* blk_chunk;
  const unsigned char* packF;
  const unsigned char* packB;
  const T* r;
  T* y;
  T* s;
  int W, maxWp, stage_bytes, nstages, ring_elems;
  const int* gate;
  int* err;
};

constexpr int kBarLevel = 1;                      // consumers, once per chunk
constexpr int kBarTurn = 2;                       // consumers -> producer: forward sweep written
constexpr int kBarStage0 = 3;                     // consumers -> producer: stage s free (id 3 + s)
constexpr int kGrpMaxStages = 12;                 // named barrier ids 3..14

// Producer descriptor of one group: {packed offset / 16, record bytes, first permuted
// position, vector-slice bytes}.
struct GrpDesc { int off16, cbytes, start, vbytes; };

template <class T>
struct GrpArgs {
  const GrpDesc* tabF;   // per group, forward order
  const GrpDesc* tabB;   // per group, forward order (the backward sweep walks it backwards)
  const int* blk_grp;    // nb + 1
  const unsigned char* packF;
  const unsigned char* packB;
  const T* r;
  T* y;
  T* s;
  int stage_bytes, nstages, ring_elems;
  const int* gate;
  int* err;
};

__device__ __forceinline__ void named_bar_arrive(int id, int nthreads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Operands of the row a consumer thread owns in one chunk, staged in registers one chunk
// ahead.  Every chunk carries exactly KM coupled entries per row (shorter rows point at the
// ring's zero slot), and a thread past the chunk's last row repeats that row (the same
// loads, the same result stored to the same place), so the level step has no branch and no
// predicate.
template <class T, int KM>
struct GOps {
  T x, dg, v[KM];
  uint32_t g[KM];       // ring byte offsets of the coupled rows
  uint32_t w;           // ring byte offset of the row
  uint32_t xo;          // byte offset of the row in the group's vector slice
};

// The K 16-bit ring offsets of a row record, read as whole T-sized words (no bank conflicts).
template <class T, int KM>
__device__ __forceinline__ void load_slots(const unsigned char* sp, uint32_t (&g)[KM]) {
  constexpr int PER = (int)sizeof(T) / 2;   // offsets per word
#pragma unroll
  for (int k0 = 0; k0 < KM; k0 += PER) {
    uint32_t w[PER / 2];
    if constexpr (sizeof(T) == 16) {
      const uint4 v = *reinterpret_cast<const uint4*>(sp + 2 * k0);
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else if constexpr (sizeof(T) == 8) {
      const uint2 v = *reinterpret_cast<const uint2*>(sp + 2 * k0);
      w[0] = v.x; w[1] = v.y;
    } else {
      w[0] = *reinterpret_cast<const uint32_t*>(sp + 2 * k0);
    }
#pragma unroll
    for (int k = k0; k < KM && k < k0 + PER; ++k) g[k] = (k & 1) ? w[(k - k0) / 2] >> 16 : w[(k - k0) / 2] & 0xffffu;
  }
}

template <class T, bool HAS_DG, int KM>
__device__ __forceinline__ void gload(GOps<T, KM>& o, const int4& c, const unsigned char* sp, int xoff, int p) {
  constexpr int SZ = (int)sizeof(T);
  constexpr int STR = rec_stride(SZ, HAS_DG, KM);
  constexpr int VOFF = HAS_DG ? SZ : 0;
  const int i = min(p, c.y);
  const unsigned char* rec = sp + c.x + i * STR;
  o.xo = (uint32_t)(c.w + i * SZ);
  o.w = (uint32_t)(c.z + i * SZ);
  load_slots<T, KM>(rec + VOFF + KM * SZ, o.g);
  o.x = *reinterpret_cast<const T*>(sp + xoff + o.xo);
#pragma unroll
  for (int k = 0; k < KM; ++k) o.v[k] = *reinterpret_cast<const T*>(rec + VOFF + k * SZ);
  if constexpr (HAS_DG) o.dg = *reinterpret_cast<const T*>(rec);
}

// zslot: the ring offset of a padding entry.
template <class T, bool DILU, bool FWD, int KM>
__device__ __forceinline__ T gsolve(const GOps<T, KM>& c, const T (&dv)[KM], uint32_t zslot) {
  if constexpr (std::is_same<T, dd>::value) {
    // ddsolve_ILU_crs (ddmatrix.f90:4310-4680): products s_c a in the loop's order, padding
    // entries left out (adding a zero would renormalise)
    static_assert(DILU, "the double-double sweep is D-ILU");
    dd v[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) v[k] = dd_mul(dv[k], c.v[k]);
    dd z = FWD ? c.x : dd{0.0, 0.0};
#pragma unroll
    for (int k = 0; k < KM; ++k) {
      const dd t = FWD ? dd_sub(z, v[k]) : dd_add(z, v[k]);
      const bool on = c.g[k] != zslot;
      z.hi = on ? t.hi : z.hi;
      z.lo = on ? t.lo : z.lo;
    }
    return FWD ? dd_mul(z, c.dg) : dd_sub(c.x, dd_mul(c.dg, z));
  } else {
    T acc = (FWD || !DILU) ? c.x : T(0);
#pragma unroll
    for (int k = 0; k < KM; ++k) {
      if (FWD) acc = acc - c.v[k] * dv[k];
      else if (DILU) acc = acc + dv[k] * c.v[k];
      else acc = acc - dv[k] * c.v[k];
    }
    if (FWD) return DILU ? c.dg * acc : acc;
    if (DILU) return c.x - c.dg * acc;
    return acc * c.dg;
  }
}

// Consumer side of one sweep over groups [g0, g0 + ng) of the sequence (NG groups over both
// sweeps).  Per chunk: gather the coupled values from the ring, load the next chunk's
// operands (through its descriptor, read one chunk earlier still) and finish the row, then
// pass the level barrier.  What a level costs is the instructions a warp issues between two
// barriers: about 50 a warp and level, 317 cycles, 6.8 cycles each of which 1.9 wait for a fixed
// latency, 1.5 for shared memory and 1.5 at the barrier (counters, 128^3 in 64 blocks).  So
// descriptors come ready to add, the group's bookkeeping runs once per group and threads
// without a row repeat the last one instead of branching around the work (a warp-uniform
// branch per level cost 14 us of the 86 below).  Measured, applications back to back, 128^3
// convection-diffusion, 64 blocks, 2 x 256 levels: 126 us with the descriptors and records read in
// one dependent chain under predicates, 86 us so (119 -> 70 us in FP32; 160^3 D-ILU, 80 blocks,
// 170 -> 124 us; four 1,024-row blocks of a 16^3 grid, 18.5 -> 10.3 us); inside a solve, where the
// vectors come from L2, 125 -> 77 us.  The level's own chain (gather 29 cycles, four dependent FMAs
// 36, store and barrier about 45) is a third of what remains.  A
// stage that never landed sets the abort flag; every consumer reads it after the barrier that follows a
// stage wait, so all return together (`arrived` tells how far each released stages).
template <class T, bool DILU, bool FWD, int KM>
__device__ __forceinline__ void gsweep(const GrpArgs<T>& a, uint64_t* full, volatile int* sflags,
                                       const unsigned char* stages, unsigned char* ring, int NC, int g0, int ng,
                                       int NG, int p, T* vout, int* arrived) {
  constexpr bool HAS_DG = DILU || !FWD;
  const int NST = a.nstages;
  const uint32_t zslot = (uint32_t)((a.ring_elems - 1) * (int)sizeof(T));
  if (ng <= 0) return;
  int g = g0, st = g0 % NST, ph = (g0 / NST) & 1, j = 0, nch = 0, xoff = 0;
  const unsigned char* sp = nullptr;
  unsigned char *out = nullptr, *nout = nullptr;   // the staged and the next group's output slice
  int4 h = make_int4(0, 0, 0, 0);                   // descriptor of chunk j of the group
  enum { RUN = 0, CHECK = 1, LAST = 2 };
  int state = RUN;
  // Waits for group g's stage and loads its first chunk into o.
  auto enter = [&](GOps<T, KM>& o) {
    // warp-uniform outcome, so the aligned barrier instructions below never diverge
    if (!__all_sync(kFull, mbar_wait(&full[st], ph, kWaitLimit))) {
      atomicExch(a.err, 3);
      sflags[0] = 1;
      return;
    }
    sp = stages + (size_t)st * a.stage_bytes;
    const int4 gh = *reinterpret_cast<const int4*>(sp);
    nch = gh.x;
    xoff = gh.z;
    nout = reinterpret_cast<unsigned char*>(vout + gh.y);
    gload<T, HAS_DG, KM>(o, reinterpret_cast<const int4*>(sp)[1], sp, xoff, p);
    h = reinterpret_cast<const int4*>(sp)[2];
    j = 1;
  };
  // One level: c is staged, n receives the next chunk.
  auto step = [&](const GOps<T, KM>& c, GOps<T, KM>& n) -> bool {
    T dv[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) dv[k] = *reinterpret_cast<const T*>(ring + c.g[k]);
    if (j < nch) {
      gload<T, HAS_DG, KM>(n, h, sp, xoff, p);
      ++j;
      h = reinterpret_cast<const int4*>(sp)[1 + j];   // past the last chunk: read, not used
    } else {
      // every operand of the group is in this thread's registers: release the stage
      if (g + NST < NG) named_bar_arrive(kBarStage0 + st, NC + 32);
      *arrived = ++g;
      if (++st == NST) { st = 0; ph ^= 1; }
      if (g < g0 + ng) {
        enter(n);
        state = CHECK;
      } else {
        state = LAST;
      }
    }
    const T r = gsolve<T, DILU, FWD, KM>(c, dv, zslot);
    *reinterpret_cast<T*>(ring + c.w) = r;
    *reinterpret_cast<T*>(out + c.xo) = r;
    named_bar_sync(kBarLevel, NC);
    if (state != RUN) {
      if (state == LAST || sflags[0]) return false;
      state = RUN;
      out = nout;
    }
    return true;
  };
  GOps<T, KM> A, B;
  enter(A);
  out = nout;
  named_bar_sync(kBarLevel, NC);
  if (sflags[0]) return;
  while (step(A, B) && step(B, A)) {
  }
}

// One CTA per block: NC consumer threads (a multiple of 32, at least the widest chunk, at
// most MAXC) and a producer warp.
template <class T, bool DILU, int KM, int MAXC>
__global__ void __launch_bounds__(MAXC + 32, 1) k_ilu_sweep_grp(GrpArgs<T> a) {
  if (gated(a.gate)) return;
  const int NC = blockDim.x - 32, NT = blockDim.x;
  extern __shared__ __align__(128) unsigned char smem[];
  const int NST = a.nstages;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  volatile int* sflags = reinterpret_cast<volatile int*>(full + kGrpMaxStages);
  T* ring = reinterpret_cast<T*>(smem + 128);
  unsigned char* stages =
      reinterpret_cast<unsigned char*>(ring) + (((size_t)a.ring_elems * sizeof(T) + 127) & ~size_t(127));
  const int b = blockIdx.x;
  const int c0 = a.blk_grp[b], c1 = a.blk_grp[b + 1];
  const int nGF = c1 - c0, NG = 2 * nGF;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NST; ++i) mbar_init(&full[i], 1);
    sflags[0] = 0;
    ring[a.ring_elems - 1] = pad_coef<T>();   // the padding slot; every other entry is written before it is read
    mbar_fence_init();
  }
  __syncthreads();
  if ((int)threadIdx.x >= NC) {
    // Producer warp: lane 0 fills stage g % NST with group g once the consumers have
    // released the stage (named barrier kBarStage0 + stage: a hardware wait, no polling).
    // A backward group's slice of y can only be copied once the forward sweep has
    // written it (barrier kBarTurn), so before that only its record is copied.
    const bool lead = (int)threadIdx.x == NC;
    int issued = 0;     // groups whose copies were issued
    bool turned = false;
    auto desc = [&](int g) -> GrpDesc { return g < nGF ? a.tabF[c0 + g] : a.tabB[c1 - 1 - (g - nGF)]; };
    auto turn = [&]() {
      named_bar_sync(kBarTurn, NT);
      turned = true;
      if (lead)
        for (int g = nGF; g < issued; ++g) {
          const GrpDesc d = desc(g);
          bulk_g2s(stages + (size_t)(g % NST) * a.stage_bytes + d.cbytes, a.y + d.start, (unsigned)d.vbytes,
                   &full[g % NST]);
        }
    };
    for (int g = 0; g < NG; ++g) {
      if (g == nGF + NST && !turned) turn();
      if (g >= NST) named_bar_sync(kBarStage0 + g % NST, NT);
      if (sflags[0]) continue;   // aborted: keep the barrier sequence, issue nothing
      if (lead) {
        const GrpDesc d = desc(g);
        const int st = g % NST;
        unsigned char* dst = stages + (size_t)st * a.stage_bytes;
        const bool fwd = g < nGF;
        mbar_arrive_expect_tx(&full[st], (unsigned)(d.cbytes + d.vbytes));
        bulk_g2s(dst, (fwd ? a.packF : a.packB) + (size_t)d.off16 * 16, (unsigned)d.cbytes, &full[st]);
        if (fwd) bulk_g2s(dst + d.cbytes, a.r + d.start, (unsigned)d.vbytes, &full[st]);
        else if (turned) bulk_g2s(dst + d.cbytes, a.y + d.start, (unsigned)d.vbytes, &full[st]);
      }
      issued = g + 1;
    }
    if (!turned) turn();
    // wait (bounded) for the last copy into every stage, so that no bulk copy is still
    // writing into this CTA's shared memory when it exits
    if (lead)
      for (int g = max(0, issued - NST); g < issued; ++g) mbar_wait(&full[g % NST], (g / NST) & 1, kWaitLimit);
    return;
  }
  const int p = threadIdx.x;
  unsigned char* ringb = reinterpret_cast<unsigned char*>(ring);
  int arrived = 0;   // groups (sequence index) whose stage this thread has released
  gsweep<T, DILU, true, KM>(a, full, sflags, stages, ringb, NC, 0, nGF, NG, p, a.y, &arrived);
  // forward result written: make it visible to the producer's bulk copies
  fence_proxy_async_global();
  if (sflags[0]) {
    // aborted: complete the producer's barrier sequence (blocking syncs, in its order)
    for (int g = arrived; g < nGF; ++g)
      if (g + NST < NG) named_bar_sync(kBarStage0 + g % NST, NT);
    arrived = max(arrived, nGF);
    named_bar_sync(kBarTurn, NT);
  } else {
    named_bar_arrive(kBarTurn, NT);
    gsweep<T, DILU, false, KM>(a, full, sflags, stages, ringb, NC, nGF, nGF, NG, p, a.s, &arrived);
  }
  if (sflags[0])
    for (int g = arrived; g < NG; ++g)
      if (g + NST < NG) named_bar_sync(kBarStage0 + g % NST, NT);
}

template <class T, bool DILU, bool RING>
__global__ void __launch_bounds__(kIluThreads, 1) k_ilu_solve(IluSolveArgs<T> a) {
  if (gated(a.gate)) return;
  extern __shared__ __align__(128) unsigned char smem[];
  const int NST = a.nstages;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + NST;
  volatile int* sflags = reinterpret_cast<volatile int*>(empty + NST);   // [0] abort, [1] consumed
  T* ring = reinterpret_cast<T*>(smem + ((16 * NST + 16 + 127) & ~127));
  unsigned char* stages =
      reinterpret_cast<unsigned char*>(ring) + (((size_t)a.ring_elems * sizeof(T) + 127) & ~size_t(127));

  const int b = blockIdx.x;
  const int c0 = a.blk_chunk[b], c1 = a.blk_chunk[b + 1];
  const int nc = c1 - c0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool producer = warp < kIluProducerWarps;
  const int ctid = threadIdx.x - 32 * kIluProducerWarps;
  int issued = 0;   // producer lane 0: copies issued so far (over both phases)

  if (threadIdx.x == 0) {
    for (int i = 0; i < NST; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    sflags[0] = 0;
    sflags[1] = 0;
    mbar_fence_init();
  }
  if (RING) {
    for (int i = threadIdx.x; i < a.ring_elems; i += blockDim.x) ring[i] = T(0);
  }
  __syncthreads();

  for (int phase = 0; phase < 2; ++phase) {
    const bool fwd = phase == 0;
    const unsigned char* pack = fwd ? a.packF : a.packB;
    const T* vin = fwd ? a.r : a.y;
    T* vout = fwd ? a.y : a.s;
    const int gbase = phase * nc;
    if (producer) {
      // The whole warp walks the chunk list: 32 descriptors per coalesced load, prefetched
      // one batch ahead and broadcast with shuffles; lane 0 issues the bulk copies.
      const ProdDesc* tab = fwd ? a.tabF : a.tabB;
      auto fetch = [&](int i) -> ProdDesc {
        if (i >= nc) return ProdDesc{0, 0, 0, 0};
        return tab[fwd ? c0 + i : c1 - 1 - i];
      };
      ProdDesc cur = fetch(lane);
      int pst = gbase % NST, puse = gbase / NST;   // stage and reuse count of chunk gbase
      for (int i0 = 0; i0 < nc; i0 += 32) {
        ProdDesc nxt = fetch(i0 + 32 + lane);
        const int kmax = min(32, nc - i0);
        bool stop = false;
        for (int k = 0; k < kmax; ++k) {
          ProdDesc d;
          d.off16 = __shfl_sync(kFull, cur.off16, k);
          d.start = __shfl_sync(kFull, cur.start, k);
          d.cbytes = __shfl_sync(kFull, cur.cbytes, k);
          d.vbytes = __shfl_sync(kFull, cur.vbytes, k);
          if (lane == 0) {
            const int st = pst, use = puse;
            if (++pst == NST) { pst = 0; ++puse; }
            if (sflags[0]) {
              stop = true;
            } else if (use > 0 && !mbar_wait(&empty[st], (use - 1) & 1, kWaitLimit)) {
              atomicExch(a.err, 2);
              sflags[0] = 1;
              stop = true;
            } else {
              unsigned char* dst = stages + (size_t)st * a.stage_bytes;
              mbar_arrive_expect_tx(&full[st], (unsigned)(d.cbytes + d.vbytes));
              bulk_g2s(dst, pack + (size_t)d.off16 * 16, (unsigned)d.cbytes, &full[st]);
              bulk_g2s(dst + d.cbytes, vin + d.start, (unsigned)d.vbytes, &full[st]);
              ++issued;
            }
          }
          stop = __shfl_sync(kFull, stop, 0);
          if (stop) break;
        }
        if (stop) break;
        cur = nxt;
      }
    } else {
      for (int i = 0; i < nc; ++i) {
        const int g = gbase + i;
        const int st = g % NST;
        const bool ok = mbar_wait(&full[st], (g / NST) & 1, kWaitLimit);
        if (!ok) {
          atomicExch(a.err, 3);
          sflags[0] = 1;
        } else {
          const unsigned char* sp = stages + (size_t)st * a.stage_bytes;
          const int* hdr = reinterpret_cast<const int*>(sp);
          const int start = hdr[0], w = hdr[1], wpad = hdr[2], K = hdr[3], lvl = hdr[4], off = hdr[5];
          const T* dg = reinterpret_cast<const T*>(sp + kIluHeader);
          const T* val = dg + wpad;
          const int* slot = reinterpret_cast<const int*>(val + (size_t)K * wpad);
          const T* xin = reinterpret_cast<const T*>(sp + chunk_bytes<T>(wpad, K));
          const T* dep = RING ? ring : vout;
          T* rslot = ring + (size_t)(lvl % a.W) * a.maxWp + off;
          for (int p = ctid; p < w; p += kIluConsumerThreads) {
            T out;
            // Gather the K coupled values first (independent loads), then accumulate in
            // the reference's order.
            T dv[kIluKUnroll], av[kIluKUnroll];
            T acc = (fwd || !DILU) ? xin[p] : T(0);
            for (int k0 = 0; k0 < K; k0 += kIluKUnroll) {
#pragma unroll
              for (int u = 0; u < kIluKUnroll; ++u) {
                const int k = k0 + u;
                dv[u] = T(0);
                av[u] = T(0);
                if (k < K) {
                  const int sl = slot[k * wpad + p];
                  av[u] = val[k * wpad + p];
                  if (RING || sl >= 0) dv[u] = dep[sl];
                }
              }
#pragma unroll
              for (int u = 0; u < kIluKUnroll; ++u) {
                if (k0 + u < K) {
                  if (fwd) acc = acc - av[u] * dv[u];
                  else if (DILU) acc = acc + dv[u] * av[u];
                  else acc = acc - dv[u] * av[u];
                }
              }
            }
            if (fwd) out = DILU ? dg[p] * acc : acc;
            else if (DILU) out = xin[p] - dg[p] * acc;
            else out = acc * dg[p];
            if (RING) rslot[p] = out;
            vout[start + p] = out;
          }
        }
        named_bar_sync(1, kIluConsumerThreads);
        if (ctid == 0) {
          if (ok) mbar_arrive(&empty[st]);
          sflags[1] = g + 1;
        }
        if (sflags[0]) break;   // uniform: read after the barrier
      }
      if (fwd) fence_proxy_async_global();
    }
    __syncthreads();
    if (sflags[0]) break;
  }
  // After an abort, wait (bounded) for copies that were issued but never consumed so no
  // bulk copy is still writing into this CTA's shared memory when it exits.
  if (sflags[0] && threadIdx.x == 0) {
    for (int g = sflags[1]; g < issued; ++g) mbar_wait(&full[g % NST], (g / NST) & 1, kWaitLimit);
  }
}

// ------------------------------------------------------------------ many small blocks
// A block of a few dozen rows (the 4^3 boxes of a stencil-format matrix: 64 rows on 10
// levels) gives the grouped sweep's one CTA per block too little work for its set-up and
// its 20 dependent level steps; with tens of thousands of blocks the CTAs then run one after
// another.  Here one warp sweeps one block: the rows of a level on the lanes (the levels are
// contiguous in the iteration layout), __syncwarp between levels (it orders the warp's global
// writes before the next level's reads).  The records sit in the iteration layout, K entries
// per row: forward the strictly lower in-block couplings in increasing column, backward the
// strictly upper ones (ILU(0) increasing, D-ILU decreasing column), so each row sums in the
// order of the grouped sweep, with the same expressions.
constexpr int kSmallMaxRows = 1024;   // largest block the warp sweep takes
constexpr int kSmallThreads = 256;

template <class T>
__global__ void k_ilu_small_pack(int n, int nb, const int* __restrict__ blk_lo, const int* __restrict__ blk_hi,
                                 const int* __restrict__ pos, const int* __restrict__ rp, const int* __restrict__ ci,
                                 int rbase, int cbase, const double* __restrict__ vL, const double* __restrict__ vU,
                                 const double* __restrict__ Dinv, int dilu, int K, int* __restrict__ cF,
                                 T* __restrict__ vF, T* __restrict__ dF, int* __restrict__ cB, T* __restrict__ vB,
                                 T* __restrict__ dB, const int2* __restrict__ box, int KC,
                                 unsigned short* __restrict__ hF, unsigned short* __restrict__ hB) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int a = 0, z = nb - 1;   // block of row i: the last b with blk_lo[b] <= i
    while (a < z) {
      const int mid = (a + z + 1) >> 1;
      if (blk_lo[mid] <= i) a = mid; else z = mid - 1;
    }
    int ia, iz, idg;
    inblock_range(rp, ci, rbase, cbase, i, blk_lo[a], blk_hi[a], &ia, &iz, &idg);
    const int64_t p = pos[i];
    // entry k of a sweep's record: permuted column (unstaged records) or position in the
    // block's stretch (staged ones; 32 bits where it is the only one), -1 and 0xffff for none
    auto put = [&](int* c, unsigned short* h, int k, int q) {
      if (h && K == 1) reinterpret_cast<int*>(h)[p] = q < 0 ? -1 : q - box[a].x;
      else if (h) h[p * KC + k] = q < 0 ? (unsigned short)0xffff : (unsigned short)(q - box[a].x);
      else c[p * K + k] = q;
    };
    int k = 0;
    for (int j = ia; j < idg; ++j, ++k) {
      put(cF, hF, k, pos[ci[j] - cbase]);
      vF[p * K + k] = (T)vL[j];
    }
    for (; k < K; ++k) { put(cF, hF, k, -1); vF[p * K + k] = T(0); }
    dF[p] = dilu ? (T)Dinv[i] : T(1);
    k = 0;
    if (!dilu) {
      for (int j = idg + 1; j < iz; ++j, ++k) {
        put(cB, hB, k, pos[ci[j] - cbase]);
        vB[p * K + k] = (T)vU[j];
      }
      dB[p] = (T)(1.0 / vU[idg]);
    } else {
      for (int j = iz - 1; j > idg; --j, ++k) {
        put(cB, hB, k, pos[ci[j] - cbase]);
        vB[p * K + k] = (T)vU[j];
      }
      dB[p] = (T)Dinv[i];
    }
    for (; k < K; ++k) { put(cB, hB, k, -1); vB[p * K + k] = T(0); }
  }
}

// The columns of one row's record (what its gathers wait for), loaded a level ahead.
template <int K>
struct SmallCols {
  int p;        // permuted row, -1: none
  int c[K];
};

template <int K>
__device__ __forceinline__ void small_cols(SmallCols<K>& o, int p, const int* __restrict__ cc) {
  o.p = p;
  if (p < 0) return;
#pragma unroll
  for (int k = 0; k < K; ++k) o.c[k] = cc[(int64_t)p * K + k];
}

// Row p of one sweep: its values, its input x[p] (r forward, y backward) and its diagonal
// factor load beside the gathers of the coupled values, so the row costs one round trip.
template <class T, bool DILU, bool FWD, int K>
__device__ __forceinline__ void small_row(const SmallCols<K>& o, const T* __restrict__ vv, const T* __restrict__ dd,
                                          const T* x, const T* g, T* out) {
  const int p = o.p;
  T v[K], gv[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    v[k] = vv[(int64_t)p * K + k];
    gv[k] = o.c[k] >= 0 ? g[o.c[k]] : T(0);
  }
  const T xp = x[p], dp_ = dd[p];
  T acc = (FWD || !DILU) ? xp : T(0);
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (o.c[k] >= 0) {
      if (FWD) acc = acc - v[k] * gv[k];
      else if (DILU) acc = acc + gv[k] * v[k];
      else acc = acc - gv[k] * v[k];
    }
  if (FWD) out[p] = DILU ? dp_ * acc : acc;
  else out[p] = DILU ? xp - dp_ * acc : acc * dp_;
}

// LPB lanes per block, 32 / LPB blocks per warp; y and s are written and re-read across
// levels (no __restrict__ on them).  Each lane loads its next level's columns before it
// works on the current level, so a level costs one dependent round trip.
template <class T, bool DILU, int K, int LPB>
__global__ void __launch_bounds__(kSmallThreads, K <= 3 ? 4 : (K <= 4 ? 3 : 2))
k_ilu_small(int nb, const int* __restrict__ blvl, const int* __restrict__ lo, const int* __restrict__ hi,
            const int* __restrict__ cF, const T* __restrict__ vF, const T* __restrict__ dF,
            const int* __restrict__ cB, const T* __restrict__ vB, const T* __restrict__ dB,
            const T* __restrict__ r, T* y, T* s, const int* gate) {
  if (gated(gate)) return;
  constexpr int BPW = 32 / LPB;
  const int lane = threadIdx.x & 31, sub = lane / LPB, li = lane % LPB;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int ngroups = (nb + BPW - 1) / BPW;
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < ngroups; w += nwarps) {
    const int b = w * BPW + sub;
    const int l0 = b < nb ? blvl[b] : 0, l1 = b < nb ? blvl[b + 1] : 0;
    const int nlev = l1 - l0;
    int maxlev = nlev;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) maxlev = max(maxlev, __shfl_xor_sync(0xffffffffu, maxlev, o));
    auto first_row = [&](int t, bool fwd) -> int {   // this lane's first row of step t, or -1
      if (t >= nlev) return -1;
      const int l = fwd ? l0 + t : l1 - 1 - t;
      const int p = lo[l] + li;
      return p < hi[l] ? p : -1;
    };
    SmallCols<K> cur, nxt;
    // forward: y = D^-1 (r - L y) (D-ILU) or r - L y (ILU(0), unit L)
    small_cols<K>(cur, first_row(0, true), cF);
    for (int t = 0; t < maxlev; ++t) {
      small_cols<K>(nxt, first_row(t + 1, true), cF);
      if (cur.p >= 0) {
        small_row<T, DILU, true, K>(cur, vF, dF, r, y, y);
        const int e = hi[l0 + t];
        for (int p = cur.p + LPB; p < e; p += LPB) {   // levels wider than LPB
          SmallCols<K> o;
          small_cols<K>(o, p, cF);
          small_row<T, DILU, true, K>(o, vF, dF, r, y, y);
        }
      }
      __syncwarp();
      cur = nxt;
    }
    // backward from the forward result y
    small_cols<K>(cur, first_row(0, false), cB);
    for (int t = 0; t < maxlev; ++t) {
      small_cols<K>(nxt, first_row(t + 1, false), cB);
      if (cur.p >= 0) {
        small_row<T, DILU, false, K>(cur, vB, dB, y, s, s);
        const int e = hi[l1 - 1 - t];
        for (int p = cur.p + LPB; p < e; p += LPB) {
          SmallCols<K> o;
          small_cols<K>(o, p, cB);
          small_row<T, DILU, false, K>(o, vB, dB, y, s, s);
        }
      }
      __syncwarp();
      cur = nxt;
    }
  }
}

// The same sweep with a block's data staged in shared memory.  A block's rows occupy one
// stretch [P0, P0 + S) of the iteration layout (its levels one after another, each starting
// on a multiple of 4), so the block's lanes copy the stretch's right-hand side, records and
// diagonal factors into the block's own area of shared memory with 16-byte asynchronous
// copies, all in flight at once.  Both sweeps run on shared memory, the solution overwriting
// the right-hand side in place (a level reads only rows of other levels, which are final),
// and each row of s is stored as it is finished.  The backward records are copied over the
// forward ones once the forward sweep is done: a smaller area per block lets more blocks be
// in flight on an SM, which is what the sweep waits on.  Same records, same expressions, same
// order as k_ilu_small.
// The staged records hold a coupling as its 16-bit position in the stretch, a row's entries
// padded to two or a multiple of four (small_kc): 8 bytes of indices per row and sweep instead of
// 12 for a 7-point stencil, read in one load, and a 4^3 box takes 3.9 KB instead of 4.3.  One coupling,
// as in lines of a grid, is 32 bits as it stands: the same 4 bytes as two positions, and a level
// does not wait for them to be unpacked.  64,000 lines of 64 rows, ILU(0) / D-ILU: 589 / 435 us per
// application (598 / 443 with 32-bit columns; 653 / 562 with one position padded to four, which
// also leaves room for fewer blocks on an SM; 665 / 486 padded to two).
constexpr int kStageWarps = 4;
__host__ __device__ constexpr int small_kc(int K) { return K <= 2 ? 2 : (K + 3) & ~3; }
constexpr int kStageBoxBytes = 12 * 1024;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// The lanes of a group copy `bytes` (a multiple of 16; both addresses 16-byte aligned).
__device__ __forceinline__ void group_stage(void* dst, const void* src, int bytes, int li, int lanes) {
  char* d = static_cast<char*>(dst);
  const char* g = static_cast<const char*>(src);
  for (int o = li * 16; o < bytes; o += lanes * 16) cp_async16(d + o, g + o);
}

// The positions of row q's K couplings, negative for none.
template <int K>
__device__ __forceinline__ void small_at(int (&c)[K], const unsigned short* Cc, int q) {
  if constexpr (K == 1) {
    c[0] = reinterpret_cast<const int*>(Cc)[q];
  } else {
    constexpr int KC = small_kc(K), W = KC / 2;
    unsigned w[W];
    if constexpr (KC == 2) {
      w[0] = reinterpret_cast<const unsigned*>(Cc)[q];
    } else {
#pragma unroll
      for (int k = 0; k < W; k += 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(Cc + q * KC + 2 * k);
        w[k] = v.x;
        w[k + 1] = v.y;
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const unsigned h = (k & 1) ? w[k / 2] >> 16 : w[k / 2] & 0xffffu;
      c[k] = h == 0xffffu ? -1 : (int)h;
    }
  }
}

// CG's step around the preconditioner: r += c q before the sweep, <s, r> and <r, r> after it.
// The fused sweep reads q beside r (which it reads anyway) and writes r back; s is in shared
// memory when its products are formed.  Apart they were three launches that moved five
// vectors more.
template <class T>
struct SmallCg {
  const T* q = nullptr;
  T* r = nullptr;           // updated in place
  const double* c = nullptr;
  Red red{};
};

// LPB lanes per block, 32 / LPB blocks per warp (as k_ilu_small), each block with its own
// area of box_bytes; blockDim.x / 32 warps per CTA.
template <class T, bool DILU, int K, int LPB, bool CG>
__global__ void __launch_bounds__(kStageWarps * 32)
k_ilu_small_staged(int nb, const int2* __restrict__ box, const int* __restrict__ blvl, const int* __restrict__ lo,
                   const int* __restrict__ hi, const unsigned short* __restrict__ cF, const T* __restrict__ vF,
                   const T* __restrict__ dF, const unsigned short* __restrict__ cB, const T* __restrict__ vB,
                   const T* __restrict__ dB, const T* r, T* __restrict__ s, const int* gate, int span,
                   int levcap, int box_bytes, SmallCg<T> cg) {
  if (gated(gate)) return;
  double acc2[2] = {0.0, 0.0};   // <s, r>, <r, r>
  const T cgc = CG ? (T)*cg.c : T(0);
  constexpr int BPW = 32 / LPB, KC = small_kc(K);
  extern __shared__ __align__(16) unsigned char stage_smem[];
  const int lane = threadIdx.x & 31, sub = lane / LPB, li = lane % LPB;
  const int wib = threadIdx.x >> 5, wpc = blockDim.x >> 5;
  // this block's area: T arrays first (each a multiple of 16 bytes, span being a multiple of
  // 4), then the int arrays; V and Cc hold the forward records, then the backward ones
  T* X = reinterpret_cast<T*>(stage_smem + ((size_t)wib * BPW + sub) * box_bytes);
  T* Fd = X + span;
  T* Bd = DILU ? Fd : Fd + span;   // D-ILU: both sweeps scale by the same D^-1
  T* V = Fd + span + (DILU ? 0 : span);   // after Fd (D-ILU) or after Bd (ILU(0))
  unsigned short* Cc = reinterpret_cast<unsigned short*>(V + (size_t)span * K);
  int* Lo = reinterpret_cast<int*>(Cc + (size_t)span * KC);
  int* Hi = Lo + levcap;
  const int nwarps = gridDim.x * wpc;
  const int ngroups = (nb + BPW - 1) / BPW;
  for (int w = blockIdx.x * wpc + wib; w < ngroups; w += nwarps) {
    const int b = w * BPW + sub;
    int P0 = 0, S = 0, l0 = 0, nlev = 0;
    if (b < nb) {
      const int2 bx = box[b];   // stretch: first position, length (host-checked: <= span)
      P0 = bx.x;
      S = bx.y;
      l0 = blvl[b];
      nlev = blvl[b + 1] - l0;  // host-checked: <= levcap
    }
    int maxlev = nlev;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) maxlev = max(maxlev, __shfl_xor_sync(0xffffffffu, maxlev, o));
    if (b < nb) {
      if (!CG) group_stage(X, r + P0, S * (int)sizeof(T), li, LPB);
      group_stage(V, vF + (int64_t)P0 * K, S * K * (int)sizeof(T), li, LPB);
      group_stage(Fd, dF + P0, S * (int)sizeof(T), li, LPB);
      group_stage(Cc, cF + (int64_t)P0 * KC, S * KC * 2, li, LPB);
      if (!DILU) group_stage(Bd, dB + P0, S * (int)sizeof(T), li, LPB);
      for (int t = li; t < nlev; t += LPB) {
        Lo[t] = lo[l0 + t] - P0;
        Hi[t] = hi[l0 + t] - P0;
      }
    }
    cp_async_commit();
    if (CG && b < nb) {   // r += c q while the copies are under way (16 bytes at a time: S is a multiple of 4)
      constexpr int E = 16 / (int)sizeof(T);
      for (int o = li * E; o < S; o += LPB * E) {
        const uint4 ru = *reinterpret_cast<const uint4*>(cg.r + P0 + o);
        const uint4 qu = __ldcs(reinterpret_cast<const uint4*>(cg.q + P0 + o));
        T rv[E], qv[E];
        memcpy(rv, &ru, 16);
        memcpy(qv, &qu, 16);
#pragma unroll
        for (int e = 0; e < E; ++e) {
          rv[e] = cgc * qv[e] + rv[e];
          X[o + e] = rv[e];
          acc2[1] += (double)(rv[e] * rv[e]);
        }
        uint4 wu;
        memcpy(&wu, rv, 16);
        *reinterpret_cast<uint4*>(cg.r + P0 + o) = wu;
      }
    }
    cp_async_wait<0>();   // this lane's copies
    __syncwarp();         // and everyone's
    // forward: y = D^-1 (r - L y) (D-ILU) or r - L y (ILU(0), unit L)
    for (int t = 0; t < maxlev; ++t) {
      if (t < nlev) {
        const int e = Hi[t];
        for (int q = Lo[t] + li; q < e; q += LPB) {
          T acc = X[q];
          int cc[K];
          small_at<K>(cc, Cc, q);
#pragma unroll
          for (int k = 0; k < K; ++k)
            if (cc[k] >= 0) acc = acc - V[q * K + k] * X[cc[k]];
          X[q] = DILU ? Fd[q] * acc : acc;
        }
      }
      __syncwarp();
    }
    // the forward records are no longer read (the barrier above): the backward ones replace them
    if (b < nb) {
      group_stage(V, vB + (int64_t)P0 * K, S * K * (int)sizeof(T), li, LPB);
      group_stage(Cc, cB + (int64_t)P0 * KC, S * KC * 2, li, LPB);
    }
    cp_async_commit();
    // CG: the new r again, on its way (from L2) while the backward sweep runs
    constexpr int E16 = 16 / (int)sizeof(T), RK = 3;
    uint4 rk[RK];
    if (CG) {
#pragma unroll
      for (int u = 0; u < RK; ++u) {
        const int o = (li + u * LPB) * E16;
        if (o < S) rk[u] = *reinterpret_cast<const uint4*>(cg.r + P0 + o);   // this lane's own stores
      }
    }
    cp_async_wait<0>();
    __syncwarp();
    // backward from the forward result
    for (int t = 0; t < maxlev; ++t) {
      if (t < nlev) {
        const int tl = nlev - 1 - t;
        const int e = Hi[tl];
        for (int q = Lo[tl] + li; q < e; q += LPB) {
          const T xp = X[q], d = Bd[q];
          T acc = DILU ? T(0) : xp;
          int cc[K];
          small_at<K>(cc, Cc, q);
#pragma unroll
          for (int k = 0; k < K; ++k) {
            if (cc[k] >= 0) {
              if (DILU) acc = acc + X[cc[k]] * V[q * K + k];
              else acc = acc - X[cc[k]] * V[q * K + k];
            }
          }
          const T o = DILU ? xp - d * acc : acc * d;
          X[q] = o;
          if (!CG) s[P0 + q] = o;
        }
      }
      __syncwarp();
    }
    if (CG && b < nb) {
      auto finish = [&](int o, const uint4& ru) {
        T rv[E16], sv[E16];
        memcpy(rv, &ru, 16);
#pragma unroll
        for (int e = 0; e < E16; ++e) {
          sv[e] = X[o + e];
          acc2[0] += (double)(sv[e] * rv[e]);
        }
        uint4 wu;
        memcpy(&wu, sv, 16);
        *reinterpret_cast<uint4*>(s + P0 + o) = wu;
      };
#pragma unroll
      for (int u = 0; u < RK; ++u) {
        const int o = (li + u * LPB) * E16;
        if (o < S) finish(o, rk[u]);
      }
      for (int o = (li + RK * LPB) * E16; o < S; o += LPB * E16)
        finish(o, *reinterpret_cast<const uint4*>(cg.r + P0 + o));
      __syncwarp();   // X is the next block's right-hand side
    }
  }
  if constexpr (CG) reduce_and_finish_wide<2>(acc2, cg.red);
}

// ------------------------------------------------------------------ host side
static int sweep_smem_budget() {
  int dev_smem = 0;
  PB_CUDA(cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx().device));
  return std::min(dev_smem, 220 * 1024);
}

// Couplings per row of the records: the matrix's largest number rounded up to a supported one.
static int record_couplings(int kmax) {
  for (int c : {1, 2, 3, 4, 6, 8})
    if (kmax <= c) return c;
  return kmax;
}

// The general sweep's ring of the last W levels, and the most it takes of shared memory.
constexpr int64_t kGeneralRing = 64 * 1024;
static int64_t general_ring_bytes(const IluPlan& P, int tsize) {
  return ((int64_t)P.W * std::max(4, P.maxWp) + 1) * tsize;
}
// Shared memory of the general sweep with `stages` stages of a widest chunk.
static int64_t general_smem(const IluPlan& P, int tsize, int K, bool ring, int stages) {
  const int64_t ring_alloc = ring ? ((general_ring_bytes(P, tsize) + 127) & ~int64_t(127)) : 0;
  const int64_t wpad = align4(std::min(P.maxWp, grp_rows(tsize, K)));
  const int64_t stage = (kIluHeader + wpad * tsize * (1 + K) + 4 * K * wpad + wpad * tsize + 127) & ~int64_t(127);
  return ((16 * stages + 16 + 127) & ~127) + ring_alloc + stages * stage;
}

// Whether the grouped sweep takes plan P with kuni couplings per row and sweep, and its ring: the
// last W levels or the largest block by position, whichever is smaller; its byte offsets are
// 16-bit and two stages of a widest chunk must fit beside it.  elems: the zero slot included.
static bool grp_fits(const IluPlan& P, int tsize, int kuni, RingMap& ring, int64_t& elems) {
  if (kuni > 8) return false;
  int max_span = 0;
  for (int b = 0; b < P.nb; ++b)
    max_span = std::max(max_span, align4(P.lvl_end[P.blk_lvl[b + 1] - 1]) - P.lvl_start[P.blk_lvl[b]]);
  const int maxWp = std::max(4, P.maxWp);
  const int64_t by_level = (int64_t)P.W * maxWp;
  ring = by_level <= max_span ? RingMap{P.W, maxWp} : RingMap{0, 0};
  elems = std::min<int64_t>(by_level, max_span) + 1;
  const int64_t ring_alloc = (elems * tsize + 127) & ~int64_t(127);
  const int64_t widest = kGrpHdr + align4(std::min(P.maxWp, grp_rows(tsize, kuni))) * (int64_t)(rec_stride(tsize, true, kuni) + tsize) + 256;
  return elems * tsize <= 65536 && 128 + ring_alloc + 2 * widest <= sweep_smem_budget();
}

// The double-double sweep without staged records (pb_ddcg.cu) has no stages; its ring is larger.
static SweepForm sweep_form(const IluPlan& P, int tsize) {
  const bool is_dd = tsize == (int)sizeof(dd);
  const int K = record_couplings(P.kmax);
  RingMap ring;
  int64_t elems = 0;
  if (!(is_dd && (K > 6 || P.nb >= 8 * num_sms())) && grp_fits(P, tsize, K, ring, elems)) return SweepForm{2, elems};
  const int64_t bytes = general_ring_bytes(P, tsize);
  if (is_dd) return SweepForm{bytes <= kDdRingBytes ? 1 : 0, bytes};
  const bool with_ring = bytes <= kGeneralRing;
  if (general_smem(P, tsize, K, with_ring, 2) > sweep_smem_budget()) return SweepForm{-1, bytes};
  return SweepForm{with_ring ? 1 : 0, bytes};
}

// Lays out the grouped sweep of plan P (chunks ch, kuni couplings per row and sweep) if it fits:
// ring, groups, stages and the producer tables.
template <class T>
static bool grp_layout(const IluPlan& P, const std::vector<IluChunk>& ch, const std::vector<int>& blk_chunk, int kuni,
                       IluDev<T>& D, RingMap& ring) {
  const int budget = sweep_smem_budget();
  const int maxw = std::min(P.maxWp, grp_rows((int)sizeof(T), kuni));
  int64_t elems = 0;
  if (!grp_fits(P, (int)sizeof(T), kuni, ring, elems)) return false;
  const int64_t ring_alloc = (elems * (int64_t)sizeof(T) + 127) & ~int64_t(127);
  D.ring_elems = (int)elems;
  // consumer threads: one row per thread, as many warps as the widest chunk needs: every warp more
  // lengthens the level barrier
  D.nc = std::max(32, (maxw + 31) & ~31);
  // Groups of consecutive chunks of one block, each at most kGrpMax chunks and about a
  // quarter of the stage budget (a chunk larger than that forms a group of its own).
  const int64_t sz = sizeof(T);
  const int64_t strF = rec_stride((int)sz, D.dilu, kuni), strB = rec_stride((int)sz, true, kuni);
  auto grp_bytes = [&](int64_t span) {   // backward record (the larger) + vector slice
    return kGrpHdr + ((span * strB + 15) & ~int64_t(15)) + span * sz;
  };
  // at least two stages; four when a quarter still holds a widest chunk
  const int64_t target = (budget - 128 - ring_alloc) / 4;
  std::vector<int4> gi;
  std::vector<int> blk_grp(P.nb + 1, 0);
  int64_t max_stage = 0;
  for (int b = 0; b < P.nb; ++b) {
    blk_grp[b] = (int)gi.size();
    int c = blk_chunk[b];
    while (c < blk_chunk[b + 1]) {
      const int sstart = ch[c].start;
      int e = c + 1;
      auto span_to = [&](int ce) { return (int64_t)align4(ch[ce - 1].start + ch[ce - 1].w) - sstart; };
      while (e < blk_chunk[b + 1] && e - c < kGrpMax && grp_bytes(span_to(e + 1)) <= target) ++e;
      const int64_t span = span_to(e);
      gi.push_back(make_int4(c, e, sstart, (int)span));
      max_stage = std::max(max_stage, grp_bytes(span));
      c = e;
    }
  }
  blk_grp[P.nb] = (int)gi.size();
  const int ng = (int)gi.size();
  std::vector<int64_t> goff(2 * (size_t)std::max(ng, 1), 0);
  std::vector<GrpDesc> tf(ng), tb(ng);
  int64_t oF = 0, oB = 0;
  for (int g = 0; g < ng; ++g) {
    const int64_t span = gi[g].w;
    const int64_t cbF = kGrpHdr + ((span * strF + 15) & ~int64_t(15));
    const int64_t cbB = kGrpHdr + ((span * strB + 15) & ~int64_t(15));
    goff[2 * g] = oF;
    goff[2 * g + 1] = oB;
    PB_CHECK(oF / 16 < INT32_MAX && oB / 16 < INT32_MAX, PARCEL_B_E_UNSUPPORTED,
             "packed preconditioner larger than 32 GiB");
    tf[g] = GrpDesc{(int)(oF / 16), (int)cbF, gi[g].z, (int)(span * sz)};
    tb[g] = GrpDesc{(int)(oB / 16), (int)cbB, gi[g].z, (int)(span * sz)};
    oF += align16(cbF);
    oB += align16(cbB);
  }
  D.packF_bytes = std::max<int64_t>(oF, 16);
  D.packB_bytes = std::max<int64_t>(oB, 16);
  D.stage_bytes = (int)((max_stage + 127) & ~int64_t(127));
  const int64_t room = budget - 128 - ring_alloc;
  D.nstages = (int)std::min<int64_t>(kGrpMaxStages, room / D.stage_bytes);
  PB_CHECK(D.nstages >= 2, PARCEL_B_E_UNSUPPORTED,
           "block-Jacobi level too wide for shared memory (stage %d bytes)", D.stage_bytes);
  D.smem_bytes = (int)(128 + ring_alloc + (int64_t)D.nstages * D.stage_bytes);
  D.ngroups = ng;
  D.tabF.alloc(sizeof(GrpDesc) * std::max(ng, 1));
  D.tabB.alloc(sizeof(GrpDesc) * std::max(ng, 1));
  h2d(D.tabF.p, tf.data(), sizeof(GrpDesc) * ng);
  h2d(D.tabB.p, tb.data(), sizeof(GrpDesc) * ng);
  D.blk_grp.alloc(sizeof(int) * (P.nb + 1));
  h2d(D.blk_grp.p, blk_grp.data(), sizeof(int) * (P.nb + 1));
  D.ginfo.alloc(sizeof(int4) * std::max(ng, 1));
  h2d(D.ginfo.p, gi.data(), sizeof(int4) * ng);
  D.goff.alloc(sizeof(int64_t) * goff.size());
  h2d(D.goff.p, goff.data(), sizeof(int64_t) * goff.size());
  return true;
}

// ------------------------------------------------------------------ diagonal recurrences
// D-ILU (ILUD): D_k = a_kk - sum over the lower in-block entries of (a_kr a_rk) / D_r.
// ILU(0) of a matrix without triangles (no entry of row k right of the diagonal meets row i's
// pattern except at the diagonal, as in 5- and 7-point stencils): U_ii = a_ii - sum of
// (a_ik / U_kk) a_ki, and L_ik = a_ik / U_kk; everything right of the diagonal stays.  Only the
// recurrence is sequential, so one parallel pass collects its operands in level order (the
// products a_kr a_rk, or both factors) and the recurrence reads them by position, the next
// level's while the current one is worked on, with the diagonals of earlier levels in a
// shared-memory ring (the sweep's).  Searching the transposed entries inside the recurrence
// made every level several dependent loads.  Operands + recurrence, before the split and now:
// D-ILU of 160^3 in 80 blocks 3.6 -> 0.55 + 0.25 ms, ILU(0) of 128^3 2.0 -> 0.35 + 0.21 ms,
// double-double D-ILU of 80^3 1.3 ms -> 0.1 + 0.27 ms.
// The operations and their order are those of the general kernels.
enum { FAC_DILU = 0, FAC_ILU0 = 1 };
// Lower couplings per row: three of the 5- and 7-point stencils, four of a 9-point one under
// D-ILU.  Wider stencils have triangles, so ILU(0) could not take this path; D-ILU on them keeps
// the general kernel because no solve here needed more instances (not measured).
constexpr int kFacMaxK = 4;
constexpr int kFacThreads = 512;

__device__ __forceinline__ double fac_val(const double* h, const double*, int j, double) { return h[j]; }
__device__ __forceinline__ dd fac_val(const double* h, const double* l, int j, dd) { return dd{h[j], l ? l[j] : 0.0}; }
__device__ __forceinline__ double fac_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ dd fac_mul(dd a, dd b) { return dd_mul(a, b); }
__device__ __forceinline__ double fac_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ dd fac_sub(dd a, dd b) { return dd_sub(a, b); }
__device__ __forceinline__ double fac_div(double a, double b) { return __ddiv_rn(a, b); }
// ddDILU_DInv_crs replaces a zero D by 1e-100
__device__ __forceinline__ dd fac_div(dd a, dd b) {
  return dd_div(a, (b.hi == 0.0 && b.lo == 0.0) ? dd{1.0e-100, 0.0} : b);
}

// Operands of position q: x (the diagonal entry), K couplings (c, and c2 for ILU(0)) at
// k * np + q with the ring index of the coupled row, -1 for none.  *other is set when the
// matrix needs the general kernel (unsorted rows or no diagonal entry; triangles under ILU(0)).
template <class S, int MODE>
__global__ void k_fac_operands(int np, int nb, int K, const int* __restrict__ rowAt, const int* __restrict__ pos,
                               const int* __restrict__ lev, const int* __restrict__ blo, const int* __restrict__ bhi,
                               const int* __restrict__ blvl, const int* __restrict__ lst, const int* __restrict__ rp,
                               const int* __restrict__ ci, int rbase, int cbase, const double* __restrict__ vh,
                               const double* __restrict__ vl, RingMap ring, S* __restrict__ x, S* __restrict__ c,
                               S* __restrict__ c2, int* __restrict__ slot, int* __restrict__ other) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < np; q += gridDim.x * blockDim.x) {
    const int i = rowAt[q];
    if (i < 0) continue;
    int a = 0, z = nb - 1;   // block of row i: the last b with blo[b] <= i
    while (a < z) {
      const int mid = (a + z + 1) >> 1;
      if (blo[mid] <= i) a = mid; else z = mid - 1;
    }
    const int lo = blo[a], hi = bhi[a], l0 = blvl[a], bstart = lst[l0];
    const int ra = rp[i] - rbase, rz = rp[i + 1] - rbase;
    bool bad = false, diag = false;
    int k = 0, prev = -1;
    for (int j = ra; j < rz; ++j) {
      const int r = ci[j] - cbase;
      bad |= r <= prev;
      prev = r;
      if (r == i) {
        x[q] = fac_val(vh, vl, j, S{});
        diag = true;
      }
      if (r < lo || r >= i) continue;
      // the transposed entry a_ri, and (ILU(0)) whether row r's other entries meet row i's
      int ja = -1;
      const int sa = rp[r] - rbase, sz = rp[r + 1] - rbase;
      for (int s = sa; s < sz; ++s) {
        const int cc = ci[s] - cbase;
        if (cc == i) ja = s;
        if (MODE == FAC_ILU0 && cc > r && cc < hi && cc != i)
          for (int m = ra; m < rz; ++m) bad |= ci[m] - cbase == cc;
      }
      const int64_t o = (int64_t)k * np + q;
      if (k < K) {
        int sl = -1;
        if (ja >= 0) {
          const S v = fac_val(vh, vl, j, S{}), t = fac_val(vh, vl, ja, S{});
          if (MODE == FAC_DILU) {
            c[o] = fac_mul(v, t);
          } else {
            c[o] = v;
            c2[o] = t;
          }
          const int l = lev[r], pr = pos[r];
          sl = ring.at(l, pr - lst[l0 + l], pr - bstart);
        }
        slot[o] = sl;
      }
      ++k;
    }
    for (; k < K; ++k) slot[(int64_t)k * np + q] = -1;
    if (bad || !diag) *other = 1;
  }
}

template <class S, int MODE, int K>
struct FacOps {
  S x, c[K], c2[MODE == FAC_ILU0 ? K : 1];
  int sl[K], nat, ring;
};

// One CTA per block; diag: D or U_ii by natural row.
template <class S, int MODE, int K>
__global__ void __launch_bounds__(kFacThreads, 1) k_fac_sweep(int np, LevelTab tab, const int* __restrict__ rowAt,
                                                            RingMap ring, const S* __restrict__ x,
                                                            const S* __restrict__ c, const S* __restrict__ c2,
                                                            const int* __restrict__ slot, S* __restrict__ diag) {
  extern __shared__ __align__(16) unsigned char fac_smem[];
  S* R = reinterpret_cast<S*>(fac_smem);
  const int b = blockIdx.x, l0 = tab.blvl[b], l1 = tab.blvl[b + 1];
  if (l0 == l1) return;
  const int bstart = tab.start[l0];
  auto load = [&](FacOps<S, MODE, K>& o, int q, int l, int off) {
    o.nat = rowAt[q];
    o.x = x[q];
    o.ring = ring.at(l - l0, off, q - bstart);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t at = (int64_t)k * np + q;
      o.sl[k] = slot[at];
      o.c[k] = c[at];
      if (MODE == FAC_ILU0) o.c2[MODE == FAC_ILU0 ? k : 0] = c2[at];
    }
  };
  auto solve = [&](const FacOps<S, MODE, K>& o) {
    S d = o.x;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (o.sl[k] >= 0) {
        const S t = fac_div(o.c[k], R[o.sl[k]]);
        d = fac_sub(d, MODE == FAC_ILU0 ? fac_mul(t, o.c2[MODE == FAC_ILU0 ? k : 0]) : t);
      }
    R[o.ring] = d;
    diag[o.nat] = d;
  };
  const int t = threadIdx.x;
  FacOps<S, MODE, K> cur, nxt;
  int s = tab.start[l0], e = tab.end[l0];
  bool on = s + t < e;
  if (on) load(cur, s + t, l0, t);
  for (int l = l0; l < l1; ++l) {
    int sn = 0, en = 0;
    if (l + 1 < l1) {
      sn = tab.start[l + 1];
      en = tab.end[l + 1];
    }
    const bool onn = sn + t < en;
    if (onn) load(nxt, sn + t, l + 1, t);
    if (on) solve(cur);
    for (int p = t + blockDim.x; s + p < e; p += blockDim.x) {   // levels wider than the CTA
      FacOps<S, MODE, K> o;
      load(o, s + p, l, p);
      solve(o);
    }
    __syncthreads();
    cur = nxt;
    on = onn;
    s = sn;
    e = en;
  }
}

// L_ik = a_ik / U_kk, U_ii, and the rest as it is (lu is a copy of the values).
__global__ void k_ilu0_finish(int n, int nb, const int* __restrict__ blo, const int* __restrict__ rp,
                              const int* __restrict__ ci, int rbase, int cbase, const double* __restrict__ diag,
                              double* __restrict__ lu) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int a = 0, z = nb - 1;
    while (a < z) {
      const int mid = (a + z + 1) >> 1;
      if (blo[mid] <= i) a = mid; else z = mid - 1;
    }
    const int lo = blo[a];
    for (int j = rp[i] - rbase; j < rp[i + 1] - rbase; ++j) {
      const int c = ci[j] - cbase;
      if (c == i) lu[j] = diag[i];
      else if (c >= lo && c < i) lu[j] = __ddiv_rn(lu[j], diag[c]);
    }
  }
}

__global__ void k_dilu_inv(int n, const double* __restrict__ D, double* __restrict__ Dinv) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    Dinv[i] = __ddiv_rn(1.0, D[i]);
}

// Runs the recurrence into diag; false when the matrix or the plan needs the general kernels.
template <class S, int MODE>
static bool fac_run(const IluPlan& P, int kmax, const DevMat<double>& A, const double* vlo, const LevelTab& tab,
                    const int* blo, const int* bhi, const int* d_pos, const int* d_rowAt, const int* d_lev, S* diag) {
  if (kmax > kFacMaxK) return false;
  int max_span = 0;
  for (int b = 0; b < P.nb; ++b)
    if (P.blk_lvl[b + 1] > P.blk_lvl[b])
      max_span = std::max(max_span, align4(P.lvl_end[P.blk_lvl[b + 1] - 1]) - P.lvl_start[P.blk_lvl[b]]);
  const int maxWp = std::max(4, P.maxWp);
  const int64_t by_level = (int64_t)P.W * maxWp;
  const RingMap ring = by_level <= max_span ? RingMap{P.W, maxWp} : RingMap{0, 0};
  const int64_t smem = std::min<int64_t>(by_level, max_span) * (int64_t)sizeof(S);
  if (smem > 200 * 1024) return false;
  cudaStream_t st = stream();
  const int np = P.np, K = kmax <= 3 ? 3 : kFacMaxK;
  const size_t nk = (size_t)K * np;
  DBuf x, c, c2, slot, other(sizeof(int));
  x.alloc(sizeof(S) * (size_t)np, false);
  c.alloc(sizeof(S) * nk, false);
  if (MODE == FAC_ILU0) c2.alloc(sizeof(S) * nk, false);
  slot.alloc(sizeof(int) * nk, false);
  const int grid = std::max(1, std::min((np + 255) / 256, 8 * num_sms()));
  k_fac_operands<S, MODE><<<grid, 256, 0, st>>>(np, P.nb, K, d_rowAt, d_pos, d_lev, blo, bhi, tab.blvl, tab.start,
                                                A.rowptr, A.col, A.rbase, A.cbase, A.val, vlo, ring, dp<S>(x),
                                                dp<S>(c), dp<S>(c2), dp<int>(slot), dp<int>(other));
  PB_CUDA(cudaGetLastError());
  int no = 0;
  d2h(&no, other.p, sizeof(int));
  if (no) return false;
  const int threads = std::min(kFacThreads, std::max(32, (P.maxWp + 31) & ~31));
  auto go = [&](auto kern) {
    PB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    kern<<<P.nb, threads, (size_t)smem, st>>>(np, tab, d_rowAt, ring, dp<S>(x), dp<S>(c), dp<S>(c2), dp<int>(slot),
                                              diag);
    PB_CUDA(cudaGetLastError());
  };
  if (K == 3) go(k_fac_sweep<S, MODE, 3>); else go(k_fac_sweep<S, MODE, kFacMaxK>);
  return true;
}

bool ilu_dd_diag(const IluPlan& P, const DevMat<double>& A, const double* al, const int* blo, const int* bhi,
                 const int* d_pos, const int* d_rowAt, const int* d_lev, dd* diag) {
  if (P.kmax > kFacMaxK) return false;
  const size_t nl = std::max<size_t>(P.lvl_start.size(), 1);
  DBuf blvl(sizeof(int) * (P.nb + 1)), lst(sizeof(int) * nl), lend(sizeof(int) * nl);
  h2d(blvl.p, P.blk_lvl.data(), sizeof(int) * (P.nb + 1));
  h2d(lst.p, P.lvl_start.data(), sizeof(int) * P.lvl_start.size());
  h2d(lend.p, P.lvl_end.data(), sizeof(int) * P.lvl_end.size());
  return fac_run<dd, FAC_DILU>(P, P.kmax, A, al, LevelTab{dp<int>(blvl), dp<int>(lst), dp<int>(lend)}, blo, bhi, d_pos,
                               d_rowAt, d_lev, diag);
}

// L and U values (ILU(0): lu; D-ILU: the matrix's) and D^-1 of every block, one CTA each.
struct Factor {
  DBuf lu, Dd, Di;
  const double *vL = nullptr, *vU = nullptr, *dinv = nullptr;
  // The recurrence in level order where it applies (plan, kmax couplings a row), then the rest
  // in parallel; otherwise the general kernels.
  void run_plan(const IluPlan& P, int kmax, const DevMat<double>& A, int ilu_method, const LevelTab& tab,
                const int* blo, const int* bhi, const int* d_pos, const int* d_rowAt, const int* d_lev,
                cudaStream_t st) {
    const int n = P.n, grid = std::max(1, std::min((n + 255) / 256, 8 * num_sms()));
    if (ilu_method != 2) {
      Dd.alloc(sizeof(double) * n);
      const bool done = ilu_method == 0
                            ? fac_run<double, FAC_ILU0>(P, kmax, A, nullptr, tab, blo, bhi, d_pos, d_rowAt, d_lev, dp<double>(Dd))
                            : fac_run<double, FAC_DILU>(P, kmax, A, nullptr, tab, blo, bhi, d_pos, d_rowAt, d_lev, dp<double>(Dd));
      if (done && ilu_method == 0) {
        lu.alloc(sizeof(double) * std::max<int64_t>(A.nnz, 1), false);
        d2d(lu.p, A.val, sizeof(double) * A.nnz);
        k_ilu0_finish<<<grid, 256, 0, st>>>(n, P.nb, blo, A.rowptr, A.col, A.rbase, A.cbase, dp<double>(Dd),
                                            dp<double>(lu));
        PB_CUDA(cudaGetLastError());
        vL = vU = dp<double>(lu);
        return;
      }
      if (done) {
        Di.alloc(sizeof(double) * n, false);
        k_dilu_inv<<<grid, 256, 0, st>>>(n, dp<double>(Dd), dp<double>(Di));
        PB_CUDA(cudaGetLastError());
        vL = vU = A.val;
        dinv = dp<double>(Di);
        return;
      }
    }
    run(A, n, P.nb, P.maxWp, ilu_method, tab, blo, bhi, d_rowAt, st);
  }

  void run(const DevMat<double>& A, int n, int nb, int maxw, int ilu_method, const LevelTab& tab, const int* blo,
           const int* bhi, const int* d_rowAt, cudaStream_t st) {
    vL = vU = A.val;
    if (ilu_method == 0) {
      lu.alloc(sizeof(double) * std::max<int64_t>(A.nnz, 1));
      d2d(lu.p, A.val, sizeof(double) * A.nnz);
      k_ilu0_factor<<<nb, ilu_factor_threads(maxw), 0, st>>>(tab, blo, bhi, d_rowAt, A.rowptr, A.col, A.rbase,
                                                             A.cbase, dp<double>(lu));
      vL = vU = dp<double>(lu);
    } else {
      Dd.alloc(sizeof(double) * n);
      Di.alloc(sizeof(double) * n);
      k_dilu_diag<<<nb, ilu_factor_threads(maxw), 0, st>>>(tab, blo, bhi, d_rowAt, A.rowptr, A.col, A.val, A.rbase,
                                                           A.cbase, ilu_method == 2 ? 1 : 0, dp<double>(Dd),
                                                           dp<double>(Di));
      dinv = dp<double>(Di);
    }
    PB_CUDA(cudaGetLastError());
  }
};

template <class T>
int ilu_setup_device(const IluPlan& P, const DevMat<double>& A, int ilu_method,
                     const int* d_pos, const int* d_rowAt, const int* d_lev, IluDev<T>& D) {
  cudaStream_t st = stream();
  D.nb = P.nb; D.np = P.np; D.n = P.n;
  D.dilu = ilu_method != 0;
  D.W = P.W;
  D.maxWp = std::max(4, P.maxWp);
  // every chunk carries the same number of coupled entries per row (the matrix-wide
  // maximum, rounded up to a supported count)
  const int kuni = record_couplings(P.kmax);
  std::vector<int> blk_chunk;
  std::vector<IluChunk> ch = plan_chunks(P, grp_rows((int)sizeof(T), kuni), kuni, blk_chunk);
  D.K = kuni;
  RingMap ring;
  D.grp = grp_layout<T>(P, ch, blk_chunk, kuni, D, ring);
  if (!D.grp) {
    // the general sweep: its ring holds the last W levels when they fit
    const int budget = sweep_smem_budget();
    const int64_t ring_bytes = general_ring_bytes(P, (int)sizeof(T));
    D.ring = ring_bytes <= kGeneralRing;
    const int64_t ring_alloc = D.ring ? ((ring_bytes + 127) & ~int64_t(127)) : 0;
    // per-chunk records for the general sweep
    int64_t oF = 0, oB = 0;
    int64_t max_stage = 0;
    for (auto& c : ch) {
      c.offF = oF; c.offB = oB;
      int64_t bf = chunk_bytes<T>(c.wpad, c.KL), bb = chunk_bytes<T>(c.wpad, c.KU);
      oF += align16(bf); oB += align16(bb);
      max_stage = std::max(max_stage, std::max(bf, bb) + (int64_t)c.wpad * (int64_t)sizeof(T));
    }
    D.packF_bytes = std::max<int64_t>(oF, 16);
    D.packB_bytes = std::max<int64_t>(oB, 16);
    D.stage_bytes = (int)((max_stage + 127) & ~int64_t(127));
    int nst = 16;
    auto need = [&](int k) { return (int64_t)((16 * k + 16 + 127) & ~127) + ring_alloc + (int64_t)k * D.stage_bytes; };
    while (nst > 2 && need(nst) > budget) --nst;
    PB_CHECK(need(nst) <= budget, PARCEL_B_E_UNSUPPORTED,
             "block-Jacobi level too wide for shared memory (stage %d bytes)", D.stage_bytes);
    D.nstages = nst;
    D.smem_bytes = (int)need(nst);
    std::vector<ProdDesc> tf(ch.size()), tb(ch.size());
    for (size_t i = 0; i < ch.size(); ++i) {
      const IluChunk& c = ch[i];
      PB_CHECK(c.offF / 16 < INT32_MAX && c.offB / 16 < INT32_MAX, PARCEL_B_E_UNSUPPORTED,
               "packed preconditioner larger than 32 GiB");
      tf[i] = ProdDesc{(int)(c.offF / 16), c.start, (int)chunk_bytes<T>(c.wpad, c.KL),
                       (int)(c.wpad * sizeof(T))};
      tb[i] = ProdDesc{(int)(c.offB / 16), c.start, (int)chunk_bytes<T>(c.wpad, c.KU),
                       (int)(c.wpad * sizeof(T))};
    }
    D.tabF.alloc(sizeof(ProdDesc) * std::max<size_t>(ch.size(), 1));
    D.tabB.alloc(sizeof(ProdDesc) * std::max<size_t>(ch.size(), 1));
    h2d(D.tabF.p, tf.data(), sizeof(ProdDesc) * ch.size());
    h2d(D.tabB.p, tb.data(), sizeof(ProdDesc) * ch.size());
  }
  D.chunks.alloc(sizeof(IluChunk) * std::max<size_t>(ch.size(), 1));
  h2d(D.chunks.p, ch.data(), sizeof(IluChunk) * ch.size());
  D.blk_chunk.alloc(sizeof(int) * (P.nb + 1));
  h2d(D.blk_chunk.p, blk_chunk.data(), sizeof(int) * (P.nb + 1));
  DBuf blo(sizeof(int) * P.nb), bhi(sizeof(int) * P.nb);
  h2d(blo.p, P.blk_lo.data(), sizeof(int) * P.nb);
  h2d(bhi.p, P.blk_hi.data(), sizeof(int) * P.nb);
  const size_t nl = std::max<size_t>(P.lvl_start.size(), 1);
  DBuf blvl(sizeof(int) * (P.nb + 1)), lst(sizeof(int) * nl), lend(sizeof(int) * nl);
  h2d(blvl.p, P.blk_lvl.data(), sizeof(int) * (P.nb + 1));
  h2d(lst.p, P.lvl_start.data(), sizeof(int) * P.lvl_start.size());
  h2d(lend.p, P.lvl_end.data(), sizeof(int) * P.lvl_end.size());

  trace_mark("ilu: tables to device");
  // factorisation in natural CSR order
  Factor F;
  F.run_plan(P, P.kmax, A, ilu_method, LevelTab{dp<int>(blvl), dp<int>(lst), dp<int>(lend)}, dp<int>(blo), dp<int>(bhi),
             d_pos, d_rowAt, d_lev, st);
  trace_mark("ilu: factor");
  // every byte of them that is read is packed below
  D.packF.alloc(D.packF_bytes, false);
  D.packB.alloc(D.packB_bytes, false);
  if (D.grp) {
    const FpSrc<T> src{F.vL, F.vU, F.dinv};
    k_ilu_pack_grp<T, FpSrc<T>><<<std::max(1, std::min(D.ngroups, 65535)), 256, 0, st>>>(
        dp<int4>(D.ginfo), dp<int64_t>(D.goff), D.ngroups, dp<IluChunk>(D.chunks), dp<int>(blo), dp<int>(bhi),
        dp<int>(blvl), dp<int>(lst), d_rowAt, d_pos, d_lev, A.rowptr, A.col, A.rbase, A.cbase, src,
        D.dilu ? 1 : 0, ring, (D.ring_elems - 1) * (int)sizeof(T), D.K,
        dp<unsigned char>(D.packF),
        dp<unsigned char>(D.packB));
  } else {
    k_ilu_pack<T><<<std::min<int>((int)ch.size(), 65535) > 0 ? std::min<int>((int)ch.size(), 65535) : 1,
                    128, 0, st>>>(
        dp<IluChunk>(D.chunks), (int)ch.size(), dp<int>(blo), dp<int>(bhi), dp<int>(blvl),
        dp<int>(lst), d_rowAt, d_pos, d_lev, A.rowptr, A.col, A.rbase, A.cbase, F.vL, F.vU,
        F.dinv, D.dilu ? 1 : 0, D.ring ? 1 : 0, D.W, D.maxWp,
        dp<unsigned char>(D.packF), dp<unsigned char>(D.packB));
  }
  PB_CUDA(cudaGetLastError());
  D.ytmp.alloc(sizeof(T) * (P.np + 4));
  PB_CUDA(cudaMemsetAsync(D.ytmp.p, 0, sizeof(T) * (P.np + 4), st));
  D.err.alloc(sizeof(int));
  PB_CUDA(cudaMemsetAsync(D.err.p, 0, sizeof(int), st));
  // temporaries (the factors, blo, ...) are freed when this function returns: make sure
  // the kernels that read them have finished.
  sync();
  return 0;
}

// ------------------------------------------------------------------ many small blocks, set-up
// The wavefront plan of tens of thousands of small blocks, one thread per block walking its
// rows in order; no per-chunk tables go out (64,000 boxes of 4^3: 28 ms with the plan and the
// tables made on the host, 0.8 ms so).  A thread's dependent loads (row pointer, column, level)
// take 1 to 2 us a row, so blocks of more than kSmallWalk rows get a CTA each (k_plan_levels):
// 1,200 blocks of 1,000 rows 1.7 ms on the host, 4.9 ms walked by threads, 0.25 ms so.
constexpr int kSmallWalk = 128;

struct SmallStat {
  int maxw, max_levels, span;
};

__global__ void k_small_levels(int nb, const int* __restrict__ starts, const int* __restrict__ rp,
                               const int* __restrict__ ci, int rbase, int cbase, int* lev, int* low, int* wid,
                               int* __restrict__ nlev, PlanStat* stat) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  const int lo = starts[b], hi = starts[b + 1];
  int maxlev = 0, kmax = 0;
  bool missing = false;
  for (int i = lo; i < hi; ++i) {   // low (zeroed): the level forced by upper entries of earlier rows
    const int a = rp[i] - rbase, z = rp[i + 1] - rbase;
    int L = low[i], nl = 0, nu = 0;
    bool diag = false, fixed = false, unsorted = false;
    for (int j = a; j < z; ++j) {
      const int c = ci[j] - cbase;
      if (c < lo || c >= hi) continue;
      if (c < i) {
        unsorted |= fixed;
        L = max(L, lev[c] + 1);
        ++nl;
      } else if (c == i) {
        diag = true;
      } else {
        fixed = true;
        low[c] = max(low[c], L + 1);
        ++nu;
      }
    }
    if (unsorted)   // a lower entry after an upper one: redo the upper entries with the final level
      for (int j = a; j < z; ++j) {
        const int c = ci[j] - cbase;
        if (c > i && c < hi) low[c] = max(low[c], L + 1);
      }
    missing |= !diag;
    lev[i] = L;
    wid[lo + L] += 1;   // zeroed; a block has no more levels than rows
    maxlev = max(maxlev, L);
    kmax = max(kmax, max(nl, nu));
  }
  nlev[b] = maxlev + 1;
  atomicMax(&stat->kmax, kmax);
  if (missing) atomicMin(&stat->missing, b);
}

// Every block's stretch of the layout, and the largest values.
__global__ void k_small_spans(int nb, const int* __restrict__ starts, const int* __restrict__ wid,
                              const int* __restrict__ nlev, int* __restrict__ span, SmallStat* stat) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  const int lo = starts[b], nl = nlev[b];
  int sp = 0, maxw = 0;
  for (int l = 0; l < nl; ++l) {
    const int w = wid[lo + l];
    sp += (w + 3) & ~3;
    maxw = max(maxw, w);
  }
  span[b] = sp;
  atomicMax(&stat->maxw, maxw);
  atomicMax(&stat->max_levels, nl);
  atomicMax(&stat->span, sp);
}

// Level ranges, block by block.
__global__ void k_small_layout(int nb, const int* __restrict__ starts, const int* __restrict__ blvl,
                               const int* __restrict__ first, const int* __restrict__ span,
                               const int* __restrict__ wid, int* __restrict__ lst, int* __restrict__ lend,
                               int2* __restrict__ box) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  const int lo = starts[b], l0 = blvl[b], nl = blvl[b + 1] - l0;
  int cur = first[b];
  for (int l = 0; l < nl; ++l) {
    const int w = wid[lo + l];
    lst[l0 + l] = cur;
    lend[l0 + l] = cur + w;
    cur = (cur + w + 3) & ~3;
  }
  box[b] = make_int2(first[b], span[b]);
}

// One segment per block for k_plan_pos.
__global__ void k_small_segs(int nb, const int* __restrict__ starts, const int* __restrict__ blvl,
                             PlanSeg* __restrict__ seg) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < nb) seg[b] = PlanSeg{starts[b], starts[b + 1], blvl[b]};
}

bool ilu_small_blocks(const BlockSplit& bs, int n) {
  if (bs.nb < 8 * num_sms() || 4 * (int64_t)n > INT_MAX) return false;
  for (int b = 0; b < bs.nb; ++b) {
    int lo, hi;
    bs.rows(b, n, &lo, &hi);
    if (hi - lo > kSmallMaxRows) return false;
  }
  return true;
}

bool ilu_small_plan(const BlockSplit& bs, const DevMat<double>& A, SmallPlan& P) {
  cudaStream_t st = stream();
  const int nb = bs.nb, n = A.n;
  P.nb = nb;
  P.n = n;
  std::vector<int> starts(nb + 1, n);
  for (int b = 0; b < nb; ++b) {
    int hi;
    bs.rows(b, n, &starts[b], &hi);
  }
  P.starts.alloc(sizeof(int) * (nb + 1));
  h2d(P.starts.p, starts.data(), sizeof(int) * (nb + 1));
  DBuf lev(sizeof(int) * n), low(sizeof(int) * n), wid(sizeof(int) * n), stat(sizeof(SmallStat)), pstat(sizeof(PlanStat)),
      nlev(sizeof(int) * (nb + 1)), span(sizeof(int) * (nb + 1)), first(sizeof(int) * (nb + 1));   // zero-filled
  PlanStat ph{0, INT_MAX};
  h2d(pstat.p, &ph, sizeof(ph));
  const int grid = (nb + 127) / 128;
  int max_rows = 0;
  for (int b = 0; b < nb; ++b) max_rows = std::max(max_rows, starts[b + 1] - starts[b]);
  if (max_rows <= kSmallWalk) {
    k_small_levels<<<grid, 128, 0, st>>>(nb, dp<int>(P.starts), A.rowptr, A.col, A.rbase, A.cbase, dp<int>(lev),
                                         dp<int>(low), dp<int>(wid), dp<int>(nlev), dp<PlanStat>(pstat));
    PB_CUDA(cudaGetLastError());
  } else {
    plan_levels<false>(A, nb, max_rows, dp<int>(P.starts), dp<int>(lev), dp<int>(low), dp<int>(wid), nullptr, nullptr,
                       nullptr, dp<int>(nlev), dp<PlanStat>(pstat));
  }
  k_small_spans<<<grid, 128, 0, st>>>(nb, dp<int>(P.starts), dp<int>(wid), dp<int>(nlev), dp<int>(span),
                                      dp<SmallStat>(stat));
  PB_CUDA(cudaGetLastError());
  P.blvl.alloc(sizeof(int) * (nb + 1));
  size_t tmp_bytes = 0;
  PB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, dp<int>(nlev), dp<int>(P.blvl), nb + 1, st));
  DBuf tmp(std::max<size_t>(tmp_bytes, 16));
  PB_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tmp_bytes, dp<int>(nlev), dp<int>(P.blvl), nb + 1, st));
  PB_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tmp_bytes, dp<int>(span), dp<int>(first), nb + 1, st));
  int totals[2];
  SmallStat h;
  PB_CUDA(cudaMemcpyAsync(&h, stat.p, sizeof(h), cudaMemcpyDeviceToHost, st));
  PB_CUDA(cudaMemcpyAsync(&ph, pstat.p, sizeof(ph), cudaMemcpyDeviceToHost, st));
  PB_CUDA(cudaMemcpyAsync(&totals[0], dp<int>(P.blvl) + nb, sizeof(int), cudaMemcpyDeviceToHost, st));
  PB_CUDA(cudaMemcpyAsync(&totals[1], dp<int>(first) + nb, sizeof(int), cudaMemcpyDeviceToHost, st));
  sync();
  PB_CHECK(ph.missing == INT_MAX, PARCEL_B_E_ZERO_PIVOT,
           "block-Jacobi block %d has a row without an in-block diagonal entry", ph.missing);
  if (ph.kmax > 8) return false;   // more couplings than the records hold
  P.totlev = totals[0];
  P.np = totals[1];
  P.maxw = h.maxw;
  P.max_levels = h.max_levels;
  P.kmax = ph.kmax;
  P.span = h.span;
  P.lo.alloc(sizeof(int) * P.totlev);
  P.hi.alloc(sizeof(int) * P.totlev);
  P.pos.alloc(sizeof(int) * n);
  P.rowAt.alloc(sizeof(int) * P.np);
  PB_CUDA(cudaMemsetAsync(P.rowAt.p, 0xFF, sizeof(int) * P.np, st));   // padding: -1
  P.box.alloc(sizeof(int2) * nb);
  k_small_layout<<<grid, 128, 0, st>>>(nb, dp<int>(P.starts), dp<int>(P.blvl), dp<int>(first), dp<int>(span),
                                       dp<int>(wid), dp<int>(P.lo), dp<int>(P.hi), dp<int2>(P.box));
  PB_CUDA(cudaGetLastError());
  DBuf seg, next;
  seg.alloc(sizeof(PlanSeg) * nb, false);
  next.alloc(sizeof(int) * P.totlev, false);
  d2d(next.p, P.lo.p, sizeof(int) * P.totlev);
  k_small_segs<<<grid, 128, 0, st>>>(nb, dp<int>(P.starts), dp<int>(P.blvl), dp<PlanSeg>(seg));
  PB_CUDA(cudaGetLastError());
  k_plan_pos<<<(nb + 7) / 8, 256, 0, st>>>(nb, dp<PlanSeg>(seg), dp<int>(lev), dp<int>(next), dp<int>(P.pos),
                                          dp<int>(P.rowAt));
  PB_CUDA(cudaGetLastError());
  sync();   // the temporaries above are released on return
  return true;
}

template <class T>
void ilu_small_setup(SmallPlan& P, const DevMat<double>& A, int ilu_method, const int* d_pos, const int* d_rowAt,
                     IluDev<T>& D) {
  cudaStream_t st = stream();
  D.nb = P.nb; D.np = P.np; D.n = P.n;
  D.dilu = ilu_method != 0;
  D.small = true;
  D.ring = D.grp = false;
  D.K = 8;
  for (int c : {6, 4, 3, 2, 1})
    if (P.kmax <= c) D.K = c;
  const int* blo = dp<int>(P.starts);
  Factor F;
  F.run(A, P.n, P.nb, P.maxw, ilu_method, LevelTab{dp<int>(P.blvl), dp<int>(P.lo), dp<int>(P.hi)}, blo, blo + 1,
        d_rowAt, st);
  // lanes per block: the widest level, rounded up to 8, 16 or 32 (wider levels take several
  // rows per lane)
  D.s_lpb = P.maxw <= 8 ? 8 : (P.maxw <= 16 ? 16 : 32);
  // the staged variant when a block's area lets a warp's blocks (at most 4) fit the default
  // 48 KB of a CTA
  const int KC = small_kc(D.K);
  const int levcap = align4(std::max(P.max_levels, 1));
  const int64_t tb = (int64_t)P.span * (2 + D.K + (D.dilu ? 0 : 1)) * (int64_t)sizeof(T) +
                     (int64_t)P.span * KC * 2 + 2LL * levcap * 4;
  D.s_box_bytes = 0;
  if (tb <= kStageBoxBytes) {
    D.s_span = P.span;
    D.s_levcap = levcap;
    D.s_box_bytes = (int)tb;
  }
  const bool staged = D.s_box_bytes > 0;
  const size_t rk = (size_t)P.np * D.K, ck = staged ? 2 * (size_t)P.np * KC : sizeof(int) * rk;
  D.s_cF.alloc(ck); D.s_vF.alloc(sizeof(T) * rk); D.s_dF.alloc(sizeof(T) * P.np);
  D.s_cB.alloc(ck); D.s_vB.alloc(sizeof(T) * rk); D.s_dB.alloc(sizeof(T) * P.np);
  const int g = (int)std::min<int64_t>(((int64_t)P.n + 255) / 256, 8LL * num_sms());
  k_ilu_small_pack<T><<<std::max(g, 1), 256, 0, st>>>(
      P.n, P.nb, blo, blo + 1, d_pos, A.rowptr, A.col, A.rbase, A.cbase, F.vL, F.vU, F.dinv, D.dilu ? 1 : 0, D.K,
      dp<int>(D.s_cF), dp<T>(D.s_vF), dp<T>(D.s_dF), dp<int>(D.s_cB), dp<T>(D.s_vB), dp<T>(D.s_dB), dp<int2>(P.box),
      KC, staged ? dp<unsigned short>(D.s_cF) : nullptr, staged ? dp<unsigned short>(D.s_cB) : nullptr);
  PB_CUDA(cudaGetLastError());
  D.s_blvl = std::move(P.blvl);
  D.s_lo = std::move(P.lo);
  D.s_hi = std::move(P.hi);
  D.s_box = std::move(P.box);
  D.ytmp.alloc(sizeof(T) * (P.np + 4));
  D.err.alloc(sizeof(int));
  sync();   // the factors are released on return
}
template void ilu_small_setup<double>(SmallPlan&, const DevMat<double>&, int, const int*, const int*, IluDev<double>&);
template void ilu_small_setup<float>(SmallPlan&, const DevMat<double>&, int, const int*, const int*, IluDev<float>&);

template <class T, bool DILU, bool RING>
static void launch_ilu(const IluDev<T>& D, const IluSolveArgs<T>& a, cudaStream_t st) {
  auto kern = k_ilu_solve<T, DILU, RING>;
  static int configured = 0;
  if (configured < D.smem_bytes) {
    PB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured = 227 * 1024;
  }
  kern<<<D.nb, kIluThreads, D.smem_bytes, st>>>(a);
}

template <class T, bool DILU, int KM, int MAXC>
static void launch_grp(const IluDev<T>& D, const GrpArgs<T>& a, cudaStream_t st) {
  auto kern = k_ilu_sweep_grp<T, DILU, KM, MAXC>;
  static bool configured = false;
  if (!configured) {
    PB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured = true;
  }
  kern<<<D.nb, D.nc + 32, D.smem_bytes, st>>>(a);
}

template <class T, bool DILU, int K, int LPB>
static void launch_small_lpb(const IluDev<T>& D, const T* r, T* s, const int* gate, cudaStream_t st) {
  const int64_t warps = ((int64_t)D.nb + 32 / LPB - 1) / (32 / LPB);
  const int grid = (int)std::min<int64_t>((warps * 32 + kSmallThreads - 1) / kSmallThreads, 16LL * num_sms());
  k_ilu_small<T, DILU, K, LPB><<<grid, kSmallThreads, 0, st>>>(
      D.nb, dp<int>(D.s_blvl), dp<int>(D.s_lo), dp<int>(D.s_hi), dp<int>(D.s_cF), dp<T>(D.s_vF), dp<T>(D.s_dF),
      dp<int>(D.s_cB), dp<T>(D.s_vB), dp<T>(D.s_dB), r, dp<T>(D.ytmp), s, gate);
}

// Shared memory of a CTA besides its blocks' areas (the fused reduction's).
constexpr int kStageStatic = 1024;

template <class T, bool DILU, int K, int LPB, bool CG>
static void launch_staged(const IluDev<T>& D, const T* r, T* s, const int* gate, cudaStream_t st,
                          const SmallCg<T>& cg = {}) {
  constexpr int BPW = 32 / LPB;
  const int warp_bytes = BPW * D.s_box_bytes;
  const int wpc = std::max(1, std::min(kStageWarps, (48 * 1024 - (CG ? kStageStatic : 0)) / warp_bytes));
  const int64_t groups = ((int64_t)D.nb + BPW - 1) / BPW;
  const int grid = (int)std::min<int64_t>((groups + wpc - 1) / wpc, 32LL * num_sms());
  k_ilu_small_staged<T, DILU, K, LPB, CG><<<grid, wpc * 32, (size_t)wpc * warp_bytes, st>>>(
      D.nb, dp<int2>(D.s_box), dp<int>(D.s_blvl), dp<int>(D.s_lo), dp<int>(D.s_hi), dp<unsigned short>(D.s_cF),
      dp<T>(D.s_vF), dp<T>(D.s_dF), dp<unsigned short>(D.s_cB), dp<T>(D.s_vB), dp<T>(D.s_dB), r, s, gate, D.s_span,
      D.s_levcap, D.s_box_bytes, cg);
}

template <class T, bool DILU, int K>
static void launch_small(const IluDev<T>& D, const T* r, T* s, const int* gate, cudaStream_t st) {
  if (D.s_box_bytes > 0) {
    PB_CHECK((reinterpret_cast<uintptr_t>(r) & 15) == 0, PARCEL_B_E_ARG, "right-hand side not 16-byte aligned");
    if (D.s_lpb == 8) launch_staged<T, DILU, K, 8, false>(D, r, s, gate, st);
    else if (D.s_lpb == 16) launch_staged<T, DILU, K, 16, false>(D, r, s, gate, st);
    else launch_staged<T, DILU, K, 32, false>(D, r, s, gate, st);
    return;
  }
  if (D.s_lpb == 8) launch_small_lpb<T, DILU, K, 8>(D, r, s, gate, st);
  else if (D.s_lpb == 16) launch_small_lpb<T, DILU, K, 16>(D, r, s, gate, st);
  else launch_small_lpb<T, DILU, K, 32>(D, r, s, gate, st);
}

bool ilu_setup_dd(const IluPlan& P, const DevMat<double>& A, const double* al, const double* dih, const double* dil,
                  int precision, const int* d_pos, const int* d_rowAt, const int* d_lev, IluDev<dd>& D) {
  cudaStream_t st = stream();
  D.nb = P.nb; D.np = P.np; D.n = P.n;
  D.dilu = true;
  D.W = P.W;
  D.maxWp = std::max(4, P.maxWp);
  int kuni = 0;
  for (int c : {6, 4, 3, 2, 1})
    if (P.kmax <= c) kuni = c;
  // a stage ring takes most of an SM: with eight blocks per SM and more the unstaged sweep,
  // several CTAs to an SM, is the better one
  if (kuni == 0 || P.nb >= 8 * num_sms()) return false;
  std::vector<int> blk_chunk;
  const std::vector<IluChunk> ch = plan_chunks(P, grp_rows((int)sizeof(dd), kuni), kuni, blk_chunk);
  D.K = kuni;
  RingMap ring;
  if (!grp_layout<dd>(P, ch, blk_chunk, kuni, D, ring)) return false;
  D.grp = true;
  DBuf chunks(sizeof(IluChunk) * std::max<size_t>(ch.size(), 1)), blo(sizeof(int) * P.nb), bhi(sizeof(int) * P.nb),
      blvl(sizeof(int) * (P.nb + 1)), lst(sizeof(int) * std::max<size_t>(P.lvl_start.size(), 1));
  h2d(chunks.p, ch.data(), sizeof(IluChunk) * ch.size());
  h2d(blo.p, P.blk_lo.data(), sizeof(int) * P.nb);
  h2d(bhi.p, P.blk_hi.data(), sizeof(int) * P.nb);
  h2d(blvl.p, P.blk_lvl.data(), sizeof(int) * (P.nb + 1));
  h2d(lst.p, P.lvl_start.data(), sizeof(int) * P.lvl_start.size());
  D.packF.alloc(D.packF_bytes, false);
  D.packB.alloc(D.packB_bytes, false);
  const DdSrc src{A.val, precision == 2 ? al : nullptr, dih, precision == 2 ? dil : nullptr};
  k_ilu_pack_grp<dd, DdSrc><<<std::max(1, std::min(D.ngroups, 65535)), 256, 0, st>>>(
      dp<int4>(D.ginfo), dp<int64_t>(D.goff), D.ngroups, dp<IluChunk>(chunks), dp<int>(blo), dp<int>(bhi),
      dp<int>(blvl), dp<int>(lst), d_rowAt, d_pos, d_lev, A.rowptr, A.col, A.rbase, A.cbase, src, 1, ring,
      (D.ring_elems - 1) * (int)sizeof(dd), D.K, dp<unsigned char>(D.packF), dp<unsigned char>(D.packB));
  PB_CUDA(cudaGetLastError());
  D.ytmp.alloc(sizeof(dd) * (P.np + 4));
  D.err.alloc(sizeof(int));
  sync();   // the temporaries above are released on return
  return true;
}

template <class T>
static GrpArgs<T> grp_args(const IluDev<T>& D, const T* r, T* s, const int* gate) {
  GrpArgs<T> g;
  g.tabF = dp<GrpDesc>(D.tabF);
  g.tabB = dp<GrpDesc>(D.tabB);
  g.blk_grp = dp<int>(D.blk_grp);
  g.packF = dp<unsigned char>(D.packF);
  g.packB = dp<unsigned char>(D.packB);
  g.r = r;
  g.y = dp<T>(D.ytmp);
  g.s = s;
  g.stage_bytes = D.stage_bytes;
  g.nstages = D.nstages;
  g.ring_elems = D.ring_elems;
  g.gate = gate;
  g.err = dp<int>(D.err);
  return g;
}

void ilu_apply_dd(const IluDev<dd>& D, const dd* r, dd* s, cudaStream_t st) {
  const GrpArgs<dd> g = grp_args<dd>(D, r, s, nullptr);
#define GRP_DD(KM_)                                                                                \
  case KM_:                                                                                        \
    if (D.nc <= 256) launch_grp<dd, true, KM_, 256>(D, g, st);                                     \
    else launch_grp<dd, true, KM_, grp_rows(sizeof(dd), KM_)>(D, g, st);                           \
    break;
  switch (D.K) {
    GRP_DD(1) GRP_DD(2) GRP_DD(3) GRP_DD(4) GRP_DD(6)
    default: PB_CHECK(false, PARCEL_B_E_ARG, "unsupported coupling count %d", D.K);
  }
#undef GRP_DD
  PB_CUDA(cudaGetLastError());
}

template <class T>
bool ilu_apply_cg(const IluDev<T>& D, T* r, const T* q, const double* c, T* s, const Red& red, const int* gate,
                  cudaStream_t st) {
  // the staged sweep alone, with room for the reduction, 16-byte aligned vectors and block
  // stretches that cover the whole layout
  if (!D.small || D.s_box_bytes == 0) return false;
  if ((32 / D.s_lpb) * D.s_box_bytes > 48 * 1024 - kStageStatic) return false;
  if (((reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(s)) & 15) != 0)
    return false;
  SmallCg<T> cg;
  cg.q = q; cg.r = r; cg.c = c; cg.red = red;
#define SMALL_CG(K_)                                                                                            \
  case K_:                                                                                                      \
    if (D.s_lpb == 8) {                                                                                         \
      if (D.dilu) launch_staged<T, true, K_, 8, true>(D, r, s, gate, st, cg);                                   \
      else launch_staged<T, false, K_, 8, true>(D, r, s, gate, st, cg);                                         \
    } else if (D.s_lpb == 16) {                                                                                 \
      if (D.dilu) launch_staged<T, true, K_, 16, true>(D, r, s, gate, st, cg);                                  \
      else launch_staged<T, false, K_, 16, true>(D, r, s, gate, st, cg);                                        \
    } else {                                                                                                    \
      if (D.dilu) launch_staged<T, true, K_, 32, true>(D, r, s, gate, st, cg);                                  \
      else launch_staged<T, false, K_, 32, true>(D, r, s, gate, st, cg);                                        \
    }                                                                                                           \
    break;
  switch (D.K) {
    SMALL_CG(1) SMALL_CG(2) SMALL_CG(3) SMALL_CG(4) SMALL_CG(6) SMALL_CG(8)
    default: return false;
  }
#undef SMALL_CG
  PB_CUDA(cudaGetLastError());
  return true;
}
template bool ilu_apply_cg<double>(const IluDev<double>&, double*, const double*, const double*, double*, const Red&,
                                   const int*, cudaStream_t);
template bool ilu_apply_cg<float>(const IluDev<float>&, float*, const float*, const double*, float*, const Red&,
                                  const int*, cudaStream_t);

// Iteration layout <-> sweep order (D.perm), where the two differ.
template <class T>
__global__ void k_to_sweep(int np, const int* __restrict__ perm, const T* __restrict__ r, T* __restrict__ q,
                           const int* gate) {
  if (gated(gate)) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
    const int p = perm[i];
    q[i] = p >= 0 ? r[p] : T(0);
  }
}
template <class T>
__global__ void k_from_sweep(int np, const int* __restrict__ perm, const T* __restrict__ q, T* __restrict__ s,
                             const int* gate) {
  if (gated(gate)) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
    const int p = perm[i];
    if (p >= 0) s[p] = q[i];
  }
}

__global__ void k_sweep_perm(int np, const int* __restrict__ rowAt, const int* __restrict__ pos,
                             int* __restrict__ perm) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
    const int k = rowAt[i];
    perm[i] = k >= 0 ? pos[k] : -1;
  }
}

template <class T>
void ilu_reorder(IluDev<T>& D, const int* sweep_rowAt, const int* layout_pos) {
  D.perm.alloc(sizeof(int) * (size_t)D.np, false);
  D.rq.alloc(sizeof(T) * (size_t)(D.np + 4));
  D.sq.alloc(sizeof(T) * (size_t)(D.np + 4));
  const int grid = std::max(1, std::min((D.np + 255) / 256, 8 * num_sms()));
  k_sweep_perm<<<grid, 256, 0, stream()>>>(D.np, sweep_rowAt, layout_pos, dp<int>(D.perm));
  PB_CUDA(cudaGetLastError());
}
template void ilu_reorder<double>(IluDev<double>&, const int*, const int*);
template void ilu_reorder<float>(IluDev<float>&, const int*, const int*);

template <class T>
void ilu_clear_error(const IluDev<T>& D, bool fail) {
  if (D.err.p) PB_CUDA(cudaMemsetAsync(D.err.p, fail ? 1 : 0, sizeof(int), stream()));
}
void ilu_raise_error(int flag) {
  PB_CHECK(flag == 0, PARCEL_B_E_CUDA, "block-Jacobi sweep gave up waiting (code %d)", flag);
}
template <class T>
void ilu_check_error(const IluDev<T>& D) {
  int flag = 0;
  if (D.err.p) d2h(&flag, D.err.p, sizeof(int));
  if (flag) ilu_clear_error<T>(D);   // reported once: a kept operator's next call starts clean
  ilu_raise_error(flag);
}
template void ilu_clear_error<double>(const IluDev<double>&, bool);
template void ilu_clear_error<float>(const IluDev<float>&, bool);
template void ilu_clear_error<dd>(const IluDev<dd>&, bool);
template void ilu_check_error<double>(const IluDev<double>&);
template void ilu_check_error<float>(const IluDev<float>&);
template void ilu_check_error<dd>(const IluDev<dd>&);

template <class T>
static void ilu_sweep(const IluDev<T>& D, const T* r, T* s, const int* gate, cudaStream_t st);

template <class T>
void ilu_apply(const IluDev<T>& D, const T* r, T* s, const int* gate, cudaStream_t st) {
  if (!D.perm.p) {
    ilu_sweep<T>(D, r, s, gate, st);
    return;
  }
  const int grid = std::max(1, std::min((D.np + 255) / 256, 8 * num_sms()));
  k_to_sweep<T><<<grid, 256, 0, st>>>(D.np, dp<int>(D.perm), r, dp<T>(D.rq), gate);
  ilu_sweep<T>(D, dp<T>(D.rq), dp<T>(D.sq), gate, st);
  k_from_sweep<T><<<grid, 256, 0, st>>>(D.np, dp<int>(D.perm), dp<T>(D.sq), s, gate);
  PB_CUDA(cudaGetLastError());
}

template <class T>
static void ilu_sweep(const IluDev<T>& D, const T* r, T* s, const int* gate, cudaStream_t st) {
  if (D.small) {
#define SMALL(K_)                                                                                  \
  case K_:                                                                                         \
    if (D.dilu) launch_small<T, true, K_>(D, r, s, gate, st); else launch_small<T, false, K_>(D, r, s, gate, st); \
    break;
    switch (D.K) {
      SMALL(1) SMALL(2) SMALL(3) SMALL(4) SMALL(6) SMALL(8)
      default: PB_CHECK(false, PARCEL_B_E_ARG, "unsupported coupling count %d", D.K);
    }
#undef SMALL
    PB_CUDA(cudaGetLastError());
    return;
  }
  if (D.grp) {
    const GrpArgs<T> g = grp_args<T>(D, r, s, gate);
    // 256 consumers leave each thread twice the registers of 512 (grp_rows)
#define GRP_C(KM_, MAXC_)                                                                          \
  if (D.dilu) launch_grp<T, true, KM_, MAXC_>(D, g, st); else launch_grp<T, false, KM_, MAXC_>(D, g, st);
#define GRP(KM_)                                                                                   \
  case KM_:                                                                                        \
    if (D.nc <= 256) { GRP_C(KM_, 256) } else { GRP_C(KM_, grp_rows(sizeof(T), KM_)) }             \
    break;
    switch (D.K) {
      GRP(1) GRP(2) GRP(3) GRP(4) GRP(6) GRP(8)
      default: PB_CHECK(false, PARCEL_B_E_ARG, "unsupported coupling count %d", D.K);
    }
#undef GRP
#undef GRP_C
    PB_CUDA(cudaGetLastError());
    return;
  }
  IluSolveArgs<T> a;
  a.tabF = dp<ProdDesc>(D.tabF);
  a.tabB = dp<ProdDesc>(D.tabB);
  a.blk_chunk = dp<int>(D.blk_chunk);
  a.packF = dp<unsigned char>(D.packF);
  a.packB = dp<unsigned char>(D.packB);
  a.r = r;
  a.y = dp<T>(D.ytmp);
  a.s = s;
  a.W = D.W;
  a.maxWp = D.maxWp;
  a.stage_bytes = D.stage_bytes;
  a.nstages = D.nstages;
  a.ring_elems = D.ring ? D.W * D.maxWp + 1 : 0;
  a.gate = gate;
  a.err = dp<int>(D.err);
  if (D.dilu) {
    if (D.ring) launch_ilu<T, true, true>(D, a, st); else launch_ilu<T, true, false>(D, a, st);
  } else {
    if (D.ring) launch_ilu<T, false, true>(D, a, st); else launch_ilu<T, false, false>(D, a, st);
  }
  PB_CUDA(cudaGetLastError());
}

template int ilu_setup_device<double>(const IluPlan&, const DevMat<double>&, int, const int*,
                                      const int*, const int*, IluDev<double>&);
template int ilu_setup_device<float>(const IluPlan&, const DevMat<double>&, int, const int*,
                                     const int*, const int*, IluDev<float>&);
template void ilu_apply<double>(const IluDev<double>&, const double*, double*, const int*, cudaStream_t);
template void ilu_apply<float>(const IluDev<float>&, const float*, float*, const int*, cudaStream_t);

}  // namespace pb
