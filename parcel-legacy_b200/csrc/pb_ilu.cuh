// pb_ilu.cuh -- block-Jacobi ILU(0) / D-ILU preconditioner on the level-major layout.
#pragma once

#include <vector>

#include "pb_common.cuh"

namespace pb {

// Device matrix view.  Row pointers and columns may be 1-based (the reference's arrays,
// rbase = 1, cbase = istart) or 0-based (internal copies, rbase = cbase = 0).
template <class VT>
struct DevMat {
  int n = 0;
  int64_t nnz = 0;
  const int* rowptr = nullptr;
  const int* col = nullptr;
  const VT* val = nullptr;
  int rbase = 0;
  int cbase = 0;
  // Sliced ELLPACK copy (32-row slices, column-major within a slice) used by the SpMV
  // when present: entry k of row r lives at s_off[r/32] + 32 k + r%32.
  int nslices = 0;
  const int* s_off = nullptr;
  const int* s_w = nullptr;
  const int* s_col = nullptr;
  const VT* s_val = nullptr;
  // Diagonal (DIA) copy used by the SpMV when present (natural layout of a matrix whose
  // entries lie on at most kDiaMaxDiag diagonals): entry of row r on diagonal k (column
  // r + d_off[k], offsets ascending) at d_val[(r - r % 32) nd + 32 k + r % 32] (32-row
  // slices, as the ELLPACK copy), zero where the row has no entry.
  int ndiag = 0;
  const int* d_off = nullptr;
  const VT* d_val = nullptr;
};

template <class VT>
struct SellBuf {
  DBuf off, w, col, val;
  DBuf doff, dval;   // diagonal copy (build_dia)
};

constexpr int kDiaMaxDiag = 16;

// Builds the sliced-ELLPACK copy of the natural CRS matrix A in the row order
// rowAt (device: permuted position -> natural row, -1 = empty row; null = identity) with
// columns mapped through pos (device: natural -> permuted; null = identity).  Slice widths
// and offsets are computed on the device.  Fills M's SELL fields.
template <class VT>
void build_sell(const DevMat<double>& A, int np, const int* rowAt_d, const int* pos_d, SellBuf<VT>& buf,
                DevMat<VT>& M);
// Builds the diagonal copy of the natural CRS matrix A when every entry lies on one of at
// most kDiaMaxDiag diagonals and the copy holds at most 1.5 nnz values; fills M's DIA fields
// and returns the number of diagonals (0: not built).
template <class VT>
int build_dia(const DevMat<double>& A, SellBuf<VT>& buf, DevMat<VT>& M);

// One chunk = up to kIluChunk rows of one wavefront level of one block.  Wider levels are
// split into several chunks (their rows are independent; each chunk is one sweep step).
struct IluChunk {
  int start;         // permuted position of the first row (multiple of 4)
  int w;             // rows
  int wpad;          // rows rounded up to 4
  int KL, KU;        // max strictly-lower / strictly-upper in-block entries of its rows
  int lvl;           // level index within the block
  int off_in_level;  // position of the chunk's first row within its level
  int blk;           // block-Jacobi block
  int64_t offF, offB;   // byte offsets of the packed forward / backward data
  // left uninitialised: the plan writes every field, and a plan of tens of thousands of
  // small blocks holds hundreds of thousands of chunks
  __host__ __device__ IluChunk() {}
};
constexpr int kIluChunk = 512;      // rows per chunk (multiple of 4)
// largest shared-memory ring of the double-double sweep without staged records
constexpr int kDdRingBytes = 160 * 1024;
constexpr int kIluHeader = 32;      // bytes of the per-chunk header in the packed data

// Wavefront levels of every block and the permuted, padded layout: what the host keeps of it.
struct IluPlan {
  int n = 0;            // natural rows
  int np = 0;           // permuted length incl. padding
  int nb = 0;           // blocks
  int W = 1;            // ring depth in levels
  int maxWp = 0;        // widest level (padded)
  int max_levels = 0;
  int kmax = 0;         // strictly-lower or strictly-upper in-block entries of a row, the larger
  std::vector<int> blk_lo, blk_hi;   // natural row ranges [lo, hi)
  std::vector<int> lvl_start;   // per block-level (global index) permuted start
  std::vector<int> lvl_end;     // per block-level permuted end (start + width)
  std::vector<int> blk_lvl;     // nb + 1 index into lvl_start
};

// Device-resident preconditioner.
template <class T>
struct IluDev {
  int nb = 0, np = 0, n = 0;
  int W = 1, maxWp = 0;
  bool ring = true;  // general sweep: its ring of W levels fits
  bool dilu = false;
  bool grp = false;  // grouped sweep (its ring and two stages fit, K <= 8); else the general one
  int nc = 256;      // consumer threads of the grouped sweep
  int ring_elems = 0;   // entries of the grouped sweep's ring, the zero slot included
  int K = 0;         // coupled entries per row in every record
  int ngroups = 0;
  int stage_bytes = 0, nstages = 0, smem_bytes = 0;
  DBuf chunks;      // IluChunk[]
  DBuf tabF, tabB;  // producer descriptors: per group (grouped sweep) or per chunk
  DBuf blk_grp;     // int[nb+1]: first group of each block
  DBuf ginfo, goff; // per group {first chunk, end chunk, sstart, sspan} and record offsets
  DBuf blk_chunk;   // int[nb+1]
  DBuf packF, packB;
  int64_t packF_bytes = 0, packB_bytes = 0;
  DBuf ytmp;        // forward result, np + 1 entries
  DBuf err;         // int error flag
  // set by ilu_reorder when the sweep order is not the iteration layout: sweep position ->
  // layout position (-1: padding), and the sweep's input and output
  DBuf perm, rq, sq;
  // Many small blocks (k_ilu_small): one warp per block, per-row records in the iteration
  // layout: K coupled entries (permuted column or -1, value) and a diagonal factor for each
  // sweep, forward (F) and backward (B).
  bool small = false;
  int s_lpb = 32;                           // lanes per block (8, 16 or 32)
  DBuf s_blvl, s_lo, s_hi;                  // block -> first level (nb + 1); level -> [lo, hi)
  DBuf s_cF, s_vF, s_dF, s_cB, s_vB, s_dB;
  // staged variant (k_ilu_small_staged): per block its first iteration-layout position and
  // its stretch rounded up to 4 positions; the largest stretch and level count; the shared
  // memory of one block (0: the stretches are too long, the unstaged sweep runs)
  DBuf s_box;
  int s_span = 0, s_levcap = 0, s_box_bytes = 0;
};

// Natural rows [lo, hi) of block-Jacobi block b of nb (0-based).
void ilu_block_rows(int b, int nb, int n, int* lo, int* hi);

// Row ranges of the block-Jacobi blocks: divide_region's equal split of the n rows into nb
// parts (common.f90:125-182), or explicit 0-based row starts, starts[nb] = n (the boxes of a
// stencil-format matrix, laid out one after another).
struct BlockSplit {
  int nb = 1;
  std::vector<int> starts;
  void rows(int b, int n, int* lo, int* hi) const {
    if (starts.empty()) { ilu_block_rows(b, nb, n, lo, hi); return; }
    *lo = starts[b];
    *hi = starts[b + 1];
  }
};
// Threads of the one-CTA-per-block factorisation kernels: the widest level rounded up to a
// warp, at most 256 (a CTA walks its block's levels with a stride of its size, so any size
// gives the same result; small blocks with narrow levels then fit many more CTAs per SM).
inline int ilu_factor_threads(int maxWp) { return std::min(256, std::max(32, (maxWp + 31) & ~31)); }

// Whether levels may be moved later than the early ones: not at all, where that shortens the ring of
// the sweep, or only where the sweep gets a better form by it.
enum class Tighten { no, shorter, better_form };

// Wavefront plan of the block-Jacobi blocks of the natural matrix A (device arrays), for a sweep on
// values of tsize bytes.  pos and lev (n entries) receive every row's permuted position and its
// level within its block, rowAt (np entries) the row at every position, -1 for padding.  Returns
// whether levels were moved (Tighten::no: whether a block's early levels make its ring too long).
bool ilu_build_plan(const DevMat<double>& A, const BlockSplit& blocks, Tighten tighten, int tsize, IluPlan& P,
                    DBuf& pos, DBuf& rowAt, DBuf& lev);

// Factorises (ILU(0)) or computes the D-ILU diagonal on the device and packs the sweep
// data.  ilu_method: 0 ILU(0), 1 ILUD, 2 MLUD (define.f90:40-42).  Returns a status.
template <class T>
int ilu_setup_device(const IluPlan& P, const DevMat<double>& A, int ilu_method,
                     const int* d_pos, const int* d_rowAt, const int* d_lev, IluDev<T>& D);

// Many small blocks (at least eight per SM, none above 1,024 rows): the wavefront plan built
// on the device.  ilu_small_plan is false when a row has more couplings than the warp sweep's
// records hold; the general plan takes such a matrix.
struct SmallPlan {
  int n = 0, nb = 0, np = 0, totlev = 0, maxw = 0, max_levels = 0, kmax = 0, span = 0;
  DBuf starts;            // nb + 1 first rows
  DBuf blvl, lo, hi;      // block -> first level; level -> [lo, hi) in the iteration layout
  DBuf box;               // block -> {first position, stretch}
  DBuf pos, rowAt;        // row -> position; position -> row or -1
};
bool ilu_small_blocks(const BlockSplit& bs, int n);
bool ilu_small_plan(const BlockSplit& bs, const DevMat<double>& A, SmallPlan& P);
template <class T>
void ilu_small_setup(SmallPlan& P, const DevMat<double>& A, int ilu_method, const int* d_pos, const int* d_rowAt,
                     IluDev<T>& D);

// The double-double D-ILU sweep on the grouped records: lays out the sweep data of the natural
// matrix (ah, al: value parts, al may be null) and the diagonal dih + dil (precision 1 drops
// the low parts of both).  False when the sweep does not take this plan (more than six
// couplings per row and sweep, levels too wide or too far apart for shared memory, or so many
// blocks that one CTA per SM leaves the chip idle).
struct dd;
bool ilu_setup_dd(const IluPlan& P, const DevMat<double>& A, const double* al, const double* dih, const double* dil,
                  int precision, const int* d_pos, const int* d_rowAt, const int* d_lev, IluDev<dd>& D);
// The double-double D-ILU (ILUD) diagonal by natural row, recurrence in level order; false when
// the general kernel has to compute it.
bool ilu_dd_diag(const IluPlan& P, const DevMat<double>& A, const double* al, const int* blo, const int* bhi,
                 const int* d_pos, const int* d_rowAt, const int* d_lev, dd* diag);
// s = M^-1 r on level-ordered vectors of np entries.
void ilu_apply_dd(const IluDev<dd>& D, const dd* r, dd* s, cudaStream_t st);

// CG's r += c q, s = M^-1 r and the sums <s, r>, <r, r> (red's epilogue) in one launch; false
// when this preconditioner has no such sweep (the caller then takes the separate kernels).
struct Red;
template <class T>
bool ilu_apply_cg(const IluDev<T>& D, T* r, const T* q, const double* c, T* s, const Red& red, const int* gate,
                  cudaStream_t st);

// The sweeps' error flag: a sweep whose bounded wait runs out sets it and leaves its output
// incomplete.  A solve clears it first (fail: sets it instead, as if one had given up; tests only),
// and every call that runs sweeps raises an error if it is set at the end.
template <class T>
void ilu_clear_error(const IluDev<T>& D, bool fail = false);
void ilu_raise_error(int flag);
template <class T>
void ilu_check_error(const IluDev<T>& D);   // waits for the stream

// Makes ilu_apply take and give vectors in another layout than the sweep's own order.
template <class T>
void ilu_reorder(IluDev<T>& D, const int* sweep_rowAt, const int* layout_pos);

// s = M^-1 r on permuted vectors (np entries each).
template <class T>
void ilu_apply(const IluDev<T>& D, const T* r, T* s, const int* gate, cudaStream_t st);

}  // namespace pb
