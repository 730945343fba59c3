// pb_solvers.cu -- PCG, BiCGStab and GMRES(m) drivers on B200.
//
// Reference loops (restated): KSP_pCG (src/pcg.f90:224-892), KSP_pBiCG
// (src/pbicg.f90:280-698), KSP_pGMRES (src/pgmres.f90:62-525) with GivensRotations and
// update_xVec (src/pcagmres.f90:190-242, 1136-1236).
//
// The reference's GPU path synchronises the device and moves a scalar across PCIe for
// every dot product and axpy (src/CUDA/src/cu_common.cu:412-446,
// src/parcel_vec.f90:466-470).  Here every scalar stays on the device (KState) and the
// solver logic runs in the epilogue of the reduction that produces it, so an iteration
// is a fixed sequence of kernel launches.  Each kernel first reads a device flag and
// returns at once after the reference loop has exited, which lets a whole restart cycle
// (GMRES) or a chunk of iterations (CG, BiCGStab) be captured once into a CUDA graph and
// replayed; the host looks at the flag once per replay.
#include <algorithm>
#include <chrono>
#include <type_traits>

#include "pb_cg_small.cuh"
#include "pb_mgs.cuh"

#include <functional>
#include "pb_solvers.cuh"

namespace pb {

double now_s() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// ------------------------------------------------------------------ options
namespace {
thread_local const std::vector<int>* t_block_starts = nullptr;
}  // namespace

ScopedBlockStarts::ScopedBlockStarts(const std::vector<int>* starts) { t_block_starts = starts; }
ScopedBlockStarts::~ScopedBlockStarts() { t_block_starts = nullptr; }

BlockSplit block_split(const Options& o, int n) {
  BlockSplit bs;
  if (o.block_starts.empty()) {
    bs.nb = std::max(1, std::min(o.nblocks, n));
    return bs;
  }
  const auto& s = o.block_starts;
  PB_CHECK(s.size() >= 2 && s.front() == 0 && s.back() == n, PARCEL_B_E_ARG,
           "explicit blocks must start at row 0 and end at n = %d", n);
  for (size_t b = 0; b + 1 < s.size(); ++b)
    PB_CHECK(s[b + 1] > s[b], PARCEL_B_E_ARG, "explicit block %d is empty", (int)b);
  bs.nb = (int)s.size() - 1;
  bs.starts = s;
  return bs;
}

Options resolve_options(const parcel_b_input* p) {
  Options o;
  if (t_block_starts) o.block_starts = *t_block_starts;
  if (!p) return o;
  if (p->solver > 0) o.solver = p->solver;
  if (p->ipreflag >= 0) o.precon = p->ipreflag;
  if (o.precon == PARCEL_B_PRECON_ADDITIVESCHWARZ) o.precon = PARCEL_B_PRECON_BLOCKJACOBI;
  if (p->ILU_method >= 0) o.ilu_method = p->ILU_method;
  if (p->precon_thblock > 0) o.nblocks = p->precon_thblock;
  if (p->GMRES_m > 0) o.m = p->GMRES_m;
  if (p->GMRES_GSflag > 0) o.gs = p->GMRES_GSflag;
  if (p->itrmax > 0) o.itrmax = p->itrmax;
  if (p->rtolmax != -1.0) o.rtol = p->rtolmax;
  if (p->abstolmax > 0.0) o.abstol = p->abstolmax;
  if (p->CAGMRES_sstep > 0) o.sstep = p->CAGMRES_sstep;
  if (p->CAGMRES_tstep > 0) o.tstep = p->CAGMRES_tstep;
  if (p->CAGMRES_basis >= 0) o.basis = p->CAGMRES_basis;
  if (p->CAGMRES_QRflag > 0) o.qrflag = p->CAGMRES_QRflag;
  if (p->inner_precision > 0) o.inner = p->inner_precision;
  if (p->residual_dd > 0) o.residual_dd = 1;
  if (p->inner_rtol > 0.0) o.inner_rtol = p->inner_rtol;
  if (p->max_refine > 0) o.max_refine = p->max_refine;
  if (p->independ_nvec > 0) o.independ_nvec = p->independ_nvec;
  if (p->reserved[0] == 1) o.use_graphs = false;
  if (p->reserved[1] == 1) o.fused_mgs = false;
  if (p->reserved[2] == 1) o.fail_sweep = true;
  return o;
}

// ------------------------------------------------------------------ workspace
void Workspace::init() {
  part.alloc(sizeof(double) * (size_t)red_blocks() * kMaxRed);
  ticket.alloc(sizeof(unsigned) * 4);
  state.alloc(sizeof(KState));
  PB_CUDA(cudaMemsetAsync(ticket.p, 0, sizeof(unsigned) * 4, stream()));
  PB_CUDA(cudaMemsetAsync(state.p, 0, sizeof(KState), stream()));
}

Red Workspace::red(int epi) const {
  Red r;
  r.part = dp<double>(part);
  r.ticket = dp<unsigned>(ticket);
  r.epi = epi;
  r.ea.st = st();
  return r;
}

// ------------------------------------------------------------------ preconditioner
template <class T>
__global__ void k_pj_dinv(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                          const double* __restrict__ va, int rbase, int cbase, T* __restrict__ dinv) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double d = 0.0;
    for (int j = rp[i] - rbase; j < rp[i + 1] - rbase; ++j)
      if (ci[j] - cbase == i) d = va[j];
    if (d == 0.0) d = 1.0e-300;   // get_DInv_crs (matrix.f90:3104-3144)
    dinv[i] = (T)(1.0 / d);
  }
}

template <class T>
void Precon<T>::apply(int64_t np, const T* r, T* s, const int* gate, cudaStream_t st) const {
  switch (kind) {
    case PARCEL_B_PRECON_NONE:
      lincomb<T>(np, s, r, cimm(1.0), nullptr, cimm(0.0), nullptr, cimm(0.0), gate, st);
      break;
    case PARCEL_B_PRECON_POINTJACOBI:
      scale<T>(np, s, dp<T>(dinv), r, gate, st);
      break;
    case PARCEL_B_PRECON_BLOCKJACOBI:
      // the sweeps may read r over the whole padded iteration layout
      PB_CHECK(ilu.perm.p || np >= ilu.np, PARCEL_B_E_ARG, "vector of %lld entries, the iteration layout has %d", (long long)np,
               ilu.np);
      ilu_apply<T>(ilu, r, s, gate, st);
      break;
  }
}

// ------------------------------------------------------------------ system setup
template <class T>
void build_system(const Options& o, const parcel_b_crs& A, bool dev, System<T>& S) {
  cudaStream_t st = stream();
  trace_mark(nullptr);
  S.n = A.n;
  S.nnz = A.nnz;
  const int* rp = A.rowptr;
  const int* ci = A.col;
  const double* va = A.val;
  if (!dev) {
    S.up_rowptr.alloc(sizeof(int) * (A.n + 1), false);
    S.up_col.alloc(sizeof(int) * std::max<int64_t>(A.nnz, 1), false);
    S.up_val.alloc(sizeof(double) * std::max<int64_t>(A.nnz, 1), false);
    h2d(S.up_rowptr.p, A.rowptr, sizeof(int) * (A.n + 1));
    h2d(S.up_col.p, A.col, sizeof(int) * A.nnz);
    h2d(S.up_val.p, A.val, sizeof(double) * A.nnz);
    rp = dp<int>(S.up_rowptr);
    ci = dp<int>(S.up_col);
    va = dp<double>(S.up_val);
  }
  S.Anat.n = A.n;
  S.Anat.nnz = A.nnz;
  S.Anat.rowptr = rp;
  S.Anat.col = ci;
  S.Anat.val = va;
  S.Anat.rbase = 1;
  S.Anat.cbase = A.istart;
  S.M.kind = o.precon;

  if (o.precon == PARCEL_B_PRECON_BLOCKJACOBI) {
    const BlockSplit bs = block_split(o, A.n);
    SmallPlan sp;
    if (ilu_small_blocks(bs, A.n) && ilu_small_plan(bs, S.Anat, sp)) {
      trace_mark("setup: wavefront plan");
      S.np = sp.np;
      S.permuted = true;
      S.ilu_levels_max = sp.max_levels;
      S.ilu_nblocks = sp.nb;
      S.pos = std::move(sp.pos);
      S.rowAt = std::move(sp.rowAt);
      S.A = DevMat<T>{};
      S.A.nnz = A.nnz;
      build_sell<T>(S.Anat, S.np, dp<int>(S.rowAt), dp<int>(S.pos), S.Asell, S.A);
      trace_mark("setup: sliced ELLPACK");
      ilu_small_setup<T>(sp, S.Anat, o.ilu_method, dp<int>(S.pos), dp<int>(S.rowAt), S.M.ilu);
      trace_mark("setup: ILU factor + pack");
      return;
    }
    IluPlan P;
    // BiCGStab's recurrences amplify the order of a sum to 1e-3 of its residual history, so its
    // vectors keep the early levels' order whatever order the sweep takes.  A sweep in another
    // order costs two copies per application (6 of 60 us on 97 x 89 x 83 in 48 blocks), so it is
    // taken only where levels were moved and the sweep got a better form by it.
    const bool keep_order = o.solver == PARCEL_B_SOLVER_BICG;
    const bool loose = ilu_build_plan(S.Anat, bs, keep_order ? Tighten::no : Tighten::shorter, sizeof(T), P, S.pos,
                                      S.rowAt, S.lev);
    IluPlan Q;
    DBuf qpos, qrowAt, qlev;
    const bool reorder = keep_order && loose &&
                         ilu_build_plan(S.Anat, bs, Tighten::better_form, sizeof(T), Q, qpos, qrowAt, qlev);
    trace_mark("setup: wavefront plan");
    S.np = P.np;
    S.permuted = true;
    S.ilu_levels_max = P.max_levels;
    S.ilu_nblocks = P.nb;
    S.A = DevMat<T>{};
    S.A.nnz = A.nnz;
    build_sell<T>(S.Anat, P.np, dp<int>(S.rowAt), dp<int>(S.pos), S.Asell, S.A);
    trace_mark("setup: sliced ELLPACK");
    if (reorder) {
      ilu_setup_device<T>(Q, S.Anat, o.ilu_method, dp<int>(qpos), dp<int>(qrowAt), dp<int>(qlev), S.M.ilu);
      ilu_reorder<T>(S.M.ilu, dp<int>(qrowAt), dp<int>(S.pos));
    } else {
      ilu_setup_device<T>(P, S.Anat, o.ilu_method, dp<int>(S.pos), dp<int>(S.rowAt), dp<int>(S.lev), S.M.ilu);
    }
    trace_mark("setup: ILU factor + pack");
  } else {
    S.np = A.n;
    S.permuted = false;
    if constexpr (std::is_same<T, double>::value) {
      S.A = S.Anat;
    } else {
      S.Aval_T.alloc(sizeof(T) * std::max<int64_t>(A.nnz, 1));
      convert<T, double>(A.nnz, dp<T>(S.Aval_T), va, st);
      S.A.n = A.n; S.A.nnz = A.nnz; S.A.rowptr = rp; S.A.col = ci;
      S.A.val = dp<T>(S.Aval_T); S.A.rbase = 1; S.A.cbase = A.istart;
    }
    {
      DevMat<T> M = S.A;
      build_sell<T>(S.Anat, A.n, nullptr, nullptr, S.Asell, M);
      S.spmv_diagonals = build_dia<T>(S.Anat, S.Asell, M);
      S.A = M;
    }
    if (o.precon == PARCEL_B_PRECON_POINTJACOBI) {
      S.M.dinv.alloc(sizeof(T) * A.n);
      k_pj_dinv<T><<<8 * num_sms(), 256, 0, st>>>(A.n, rp, ci, va, 1, A.istart, dp<T>(S.M.dinv));
      PB_CUDA(cudaGetLastError());
    }
  }
}

// ------------------------------------------------------------------ graph replay
static int read_done(const KState* st, cudaStream_t s) {
  static int* pinned = nullptr;
  if (!pinned) PB_CUDA(cudaMallocHost(&pinned, sizeof(int)));
  PB_CUDA(cudaMemcpyAsync(pinned, &st->done, sizeof(int), cudaMemcpyDeviceToHost, s));
  PB_CUDA(cudaStreamSynchronize(s));
  return *pinned;
}

// The state at the end of a solve; an error if a preconditioner sweep gave up.
template <class T>
static KState read_state(KState* st, const System<T>& S) {
  KState h;
  if (S.M.ilu.err.p) d2d(&st->sweep_err, S.M.ilu.err.p, sizeof(int));
  d2h(&h, st, sizeof(KState));
  ilu_raise_error(h.sweep_err);
  return h;
}

static void init_state(Workspace& W, int itr0, int itrmax) {
  KState h;
  memset(&h, 0, sizeof(h));
  h.itr = itr0;
  h.last_inner = 1;
  h.itrmax = itrmax;
  h2d(W.state.p, &h, sizeof(KState));
}

// ------------------------------------------------------------------ PCG
template <class T>
static SolveOut run_pcg(const Options& o, const System<T>& S, const T* b, T* x, double* hist,
                        KrylovWork& kw) {
  cudaStream_t st = stream();
  Workspace& W = kw.W;
  const int64_t np = S.np;
  const size_t vb = sizeof(T) * np;
  const int small_grid = S.permuted ? 0 : cg_small_grid<T>(np, S.A.nnz);
  const bool none = S.M.kind == PARCEL_B_PRECON_NONE;
  T *R = kw.buf<T>(vb), *P = kw.buf<T>(vb), *Q = kw.buf<T>(vb);
  T* Sv = none && !small_grid ? R : kw.buf<T>(vb);   // s = M^-1 r
  KState* K = W.st();
  init_state(W, 1, o.itrmax);
  const int* gdone = &K->done;
  auto red = [&](int epi) {
    Red rr = W.red(epi);
    rr.ea.hist = hist; rr.ea.rtol = o.rtol; rr.ea.abstol = o.abstol;
    return rr;
  };
  int launches = 0;
  // r = b - A x; s = M^-1 r; bnorm, rnorm, rho0 = <s, r>   (pcg.f90:442-478)
  spmv<T, T>(S.A, x, R, SPMV_RES, b, nullptr, st);
  if (Sv != R) S.M.apply(np, R, Sv, nullptr, st);
  PB_CUDA(cudaMemsetAsync(P, 0, sizeof(T) * np, st));
  DotSel sel;
  sel.a[0] = 1; sel.b[0] = 1;   // <b, b>
  sel.a[1] = 2; sel.b[1] = 2;   // <r, r>
  sel.a[2] = 3; sel.b[2] = 2;   // <s, r>
  lincomb_dot<T>(np, nullptr, b, cimm(0), R, cimm(0), Sv, cimm(0), nullptr, nullptr, sel, 3,
                 red(EPI_CG_INIT), nullptr, st);
  launches += 3;
  auto finish = [&]() -> SolveOut {
    // x = alpha p + x   (pcg.f90:733)
    lincomb<T>(np, x, P, cdev(&K->alpha), x, cimm(1.0), nullptr, cimm(0), nullptr, st);
    KState h = read_state(K, S);
    SolveOut out;
    out.niter = h.niter;
    out.iret = h.iret;
    out.breakdown = h.breakdown;
    out.launches = launches + 1;
    return out;
  };
  // short vectors in the natural layout: all iterations in cooperative launches
  if (const int grid = small_grid) {
    CgSmallArgs<T> ca;
    ca.A = S.A;
    ca.dinv = S.M.kind == PARCEL_B_PRECON_POINTJACOBI ? dp<T>(S.M.dinv) : nullptr;
    ca.x = x; ca.r = R; ca.s = Sv; ca.p = P; ca.p2 = Q;
    ca.st = K; ca.hist = hist; ca.rtol = o.rtol;
    const size_t words = sizeof(unsigned long long) * cg_small_slots(grid);
    ca.slots = kw.buf<unsigned long long>(words);
    ca.err = kw.buf<int>(sizeof(int));
    PB_CUDA(cudaMemsetAsync(ca.slots, 0, words, st));
    PB_CUDA(cudaMemsetAsync(ca.err, 0, sizeof(int), st));
    // a launch ends after 4,096 iterations (about 20 ms), so that one does not run for long
    ca.maxit = 4096;
    int err = 0;
    for (int64_t it = 0; it <= o.itrmax && !err && !read_done(K, st); it += ca.maxit) {
      ca.tag0 = (unsigned)it;
      cg_small<T>(ca, st);
      launches += 1;
      d2h(&err, ca.err, sizeof(int));
    }
    PB_CHECK(err == 0, PARCEL_B_E_CUDA, "CG grid sum timed out");
    return finish();
  }
  const int chunk = 16;
  int& per_chunk = kw.per_cycle;   // counted when the chunk is captured
  auto iterations = [&] {
    per_chunk = 0;
    for (int it = 0; it < chunk; ++it) {
      cg_axpy2<T>(np, x, P, Sv, K, gdone, st);                            // x += alpha p; p = s + beta p
      int sa[2] = {1, 0}, sb[2] = {0, 0};
      spmv_dot<T, T>(S.A, P, Q, SPMV_Y, nullptr, nullptr, 1, sa, sb, red(EPI_CG_GAMMA), gdone, st);
      if (S.M.kind == PARCEL_B_PRECON_BLOCKJACOBI &&
          ilu_apply_cg<T>(S.M.ilu, R, Q, &K->tmp[0], Sv, red(EPI_CG_DOT2), gdone, st)) {
        per_chunk += 3;
        continue;
      }
      if (none || S.M.kind == PARCEL_B_PRECON_POINTJACOBI) {
        cg_step<T>(np, R, Q, none ? nullptr : dp<T>(S.M.dinv), none ? nullptr : Sv, &K->tmp[0], red(EPI_CG_DOT2),
                   gdone, st);
        per_chunk += 3;
        continue;
      }
      per_chunk += 5;
      lincomb<T>(np, R, Q, cdev(&K->tmp[0]), R, cimm(1.0), nullptr, cimm(0), gdone, st);  // r = -alpha q + r
      S.M.apply(np, R, Sv, gdone, st);                                    // s = M^-1 r
      cg_dots<T>(np, Sv, R, red(EPI_CG_DOT2), gdone, st);                  // <s, r>, <r, r>
    }
  };
  GraphRunner& G = kw.G;
  const int max_chunks = o.itrmax / chunk + 2;
  for (int c = 0; c < max_chunks; ++c) {
    if (read_done(K, st)) break;
    G.launch(iterations, o.use_graphs, st);
    launches += per_chunk;
  }
  return finish();
}

// ------------------------------------------------------------------ BiCGStab
template <class T>
static SolveOut run_bicg(const Options& o, const System<T>& S, const T* b, T* x, double* hist,
                         KrylovWork& kw) {
  cudaStream_t st = stream();
  Workspace& W = kw.W;
  const int64_t np = S.np;
  const size_t vb = sizeof(T) * np;
  T *R = kw.buf<T>(vb), *R0 = kw.buf<T>(vb), *P = kw.buf<T>(vb), *Q = kw.buf<T>(vb), *PP = kw.buf<T>(vb),
    *E = kw.buf<T>(vb), *PE = kw.buf<T>(vb), *V = kw.buf<T>(vb);
  KState* K = W.st();
  init_state(W, 1, o.itrmax);
  const int* gdone = &K->done;
  auto red = [&](int epi) {
    Red rr = W.red(epi);
    rr.ea.hist = hist; rr.ea.rtol = o.rtol;
    return rr;
  };
  int launches = 0;
  spmv<T, T>(S.A, x, R, SPMV_RES, b, nullptr, st);
  DotSel sel;
  sel.a[0] = 1; sel.b[0] = 1;   // <b, b>
  sel.a[1] = 2; sel.b[1] = 2;   // <r, r>
  lincomb_dot<T>(np, nullptr, b, cimm(0), R, cimm(0), nullptr, cimm(0), nullptr, nullptr, sel, 2,
                 red(EPI_BICG_INIT), nullptr, st);
  d2d(R0, R, vb);
  d2d(P, R, vb);
  launches += 2;
  const int chunk = 8;
  auto iterations = [&] {
    for (int it = 0; it < chunk; ++it) {
      S.M.apply(np, P, PP, gdone, st);                                        // pp = M^-1 p
      int sa[2] = {2, 0}, sb[2] = {0, 0};
      spmv_dot<T, T>(S.A, PP, Q, SPMV_Y, nullptr, R0, 1, sa, sb, red(EPI_BICG_C2), gdone, st);  // q, c2
      lincomb<T>(np, E, R, cimm(1.0), Q, cdev(&K->tmp[0]), nullptr, cimm(0), gdone, st);      // e = r - alpha q
      S.M.apply(np, E, PE, gdone, st);                                        // pe = M^-1 e
      int sa2[2] = {2, 0}, sb2[2] = {0, 0};
      spmv_dot<T, T>(S.A, PE, V, SPMV_Y, nullptr, E, 2, sa2, sb2, red(EPI_BICG_C3), gdone, st);  // v, <e,v>, <v,v>
      lincomb<T>(np, x, PP, cdev(&K->alpha), PE, cdev(&K->c3), x, cimm(1.0), gdone, st);   // x += alpha pp + c3 pe
      DotSel d3;
      d3.a[0] = 0; d3.b[0] = 4;   // <r, r0>
      d3.a[1] = 0; d3.b[1] = 0;   // <r, r>
      lincomb_dot<T>(np, R, E, cimm(1.0), V, cdev(&K->tmp[1]), nullptr, cimm(0), R0, nullptr, d3, 2,
                     red(EPI_BICG_END), gdone, st);                           // r = e - c3 v
      lincomb<T>(np, P, R, cimm(1.0), Q, cdev(&K->tmp[2]), P, cdev(&K->beta), gdone, st);  // p = r - beta c3 q + beta p
    }
  };
  GraphRunner& G = kw.G;
  const int max_chunks = o.itrmax / chunk + 2;
  for (int c = 0; c < max_chunks; ++c) {
    if (read_done(K, st)) break;
    G.launch(iterations, o.use_graphs, st);
    launches += 8 * chunk;
  }
  KState h = read_state(K, S);
  SolveOut out;
  out.niter = h.niter;
  out.iret = h.iret;
  out.breakdown = h.breakdown;
  out.launches = launches;
  return out;
}

// ------------------------------------------------------------------ GMRES(m)
template <class T>
static SolveOut run_gmres(const Options& o, const System<T>& S, const T* b, T* x, double* hist,
                          KrylovWork& kw) {
  cudaStream_t st = stream();
  Workspace& W = kw.W;
  const int64_t np = S.np;
  const int m = o.m;
  PB_CHECK(m >= 1 && m < kMaxRed, PARCEL_B_E_ARG, "GMRES restart length %d outside [1, %d)", m, kMaxRed);
  const int64_t ldv = (np + 31) & ~int64_t(31);
  const size_t vb = sizeof(T) * np;
  T *R = kw.buf<T>(vb), *V = kw.buf<T>(sizeof(T) * ldv * (m + 1)), *PV = kw.buf<T>(vb), *Wv = kw.buf<T>(vb),
    *V0 = kw.buf<T>(vb), *X0 = kw.buf<T>(vb);   // zero-filled: the tails past np stay zero
  // Flexible GMRES keeps z_j = M_j^-1 v_j (the preconditioner may change between
  // columns) and updates x with Z y instead of M^-1 V y.
  const bool flex = o.flexible || S.extra != nullptr;
  T* Z = flex ? kw.buf<T>(sizeof(T) * ldv * m) : nullptr;
  // precon(in, out, az): out = M^-1 in (+ the extra stage); with the extra stage and az
  // given, az = A out comes from the stage and the caller's SpMV is skipped.
  auto precon = [&](const T* in, T* out, T* az, const int* gate) {
    if (S.extra) S.extra->begin(S, in, gate, st);
    S.M.apply(np, in, out, gate, st);
    if (S.extra) S.extra->apply(S, in, out, az, gate, st);
  };
  const int precon_launches = 1 + (S.extra ? S.extra->launches() : 0);
  const size_t mb = sizeof(double) * (m + 1);
  double *hb = kw.buf<double>(mb * m), *eb = kw.buf<double>(mb), *csb = kw.buf<double>(mb), *snb = kw.buf<double>(mb),
         *yb = kw.buf<double>(mb);
  KState* K = W.st();
  init_state(W, 1, o.itrmax);
  const int* gdone = &K->done;
  const int* gskip = &K->skip_inner;
  auto red = [&](int epi, int k = 0, int j = 0) {
    Red rr = W.red(epi);
    rr.ea.hist = hist; rr.ea.rtol = o.rtol; rr.ea.abstol = o.abstol;
    rr.ea.h = hb; rr.ea.e = eb; rr.ea.cs = csb;
    rr.ea.sn = snb; rr.ea.m = m; rr.ea.k = k; rr.ea.j = j;
    return rr;
  };
  int launches = 0;
  {  // bnorm = ||b||
    Red rr = red(EPI_NORM2);
    rr.ea.out = &K->bnorm;
    DotSel sel;
    sel.a[0] = 1; sel.b[0] = 1;
    lincomb_dot<T>(np, nullptr, b, cimm(0), nullptr, cimm(0), nullptr, cimm(0), nullptr, nullptr, sel, 1,
                   rr, nullptr, st);
    launches += 1;
  }
  // Fused one-launch MGS (pb_mgs.cu) when the vector fits its register tiling.
  const bool fused_mgs = o.gs != PARCEL_B_GS_CGS && o.fused_mgs && mgs_supported<T>(np);
  // The staged variant reduces through per-(column, pass, CTA) slots that start every
  // cycle as all-ones bytes; the others through per-(column, pass) counters that start at 0.
  const bool staged_mgs = fused_mgs && mgs_staged<T>(np);
  const size_t nslots = (size_t)m * (m + 2) * (size_t)(num_sms() + 1);   // partials, then totals
  double* mparts = kw.buf<double>(sizeof(double) * 2 * (size_t)std::max(1, mgs_grid<T>()));
  unsigned* mctr = kw.buf<unsigned>(sizeof(unsigned) * (size_t)m * (m + 2));
  int* merr = kw.buf<int>(sizeof(int));
  double* mslots = staged_mgs ? kw.buf<double>(sizeof(double) * nslots) : nullptr;
  PB_CUDA(cudaMemsetAsync(merr, 0, sizeof(int), st));
  int& per_cycle = kw.per_cycle;   // counted when the cycle is captured
  auto cycle = [&] {
    per_cycle = 0;
    if (staged_mgs) {
      PB_CUDA(cudaMemsetAsync(mslots, 0xFF, sizeof(double) * nslots, st));
      ++per_cycle;
    } else if (fused_mgs) {
      PB_CUDA(cudaMemsetAsync(mctr, 0, sizeof(unsigned) * (size_t)m * (m + 2), st));
      ++per_cycle;
    }
    int sa[2] = {0, 0}, sb[2] = {0, 0};
    spmv_dot<T, T>(S.A, x, R, SPMV_RES, b, nullptr, 1, sa, sb, red(EPI_GM_RESTART), gdone, st);
    ++per_cycle;
    for (int j = 1; j <= m; ++j) {
      T* Vj = V + (size_t)(j - 1) * ldv;
      if (j == 1) {
        lincomb<T>(np, Vj, R, cdev(&K->tmp[0]), nullptr, cimm(0), nullptr, cimm(0), gskip, st);
        ++per_cycle;
      }
      T* Pj = flex ? Z + (size_t)(j - 1) * ldv : PV;
      const bool az_from_stage = S.extra && S.extra->provides_az() && fused_mgs && o.gs != PARCEL_B_GS_CGS;
      precon(Vj, Pj, az_from_stage ? Wv : nullptr, gskip);
      per_cycle += precon_launches;
      if (o.gs == PARCEL_B_GS_CGS) {
        spmv<T, T>(S.A, Pj, Wv, SPMV_Y, nullptr, gskip, st);
        multidot<T>(np, j, Wv, V, ldv, red(EPI_GM_HCGS, 0, j), gskip, st);
        cgs_update<T>(np, j, Wv, V, ldv, hb + (size_t)(j - 1) * (m + 1), red(EPI_GM_NORM, 0, j),
                      gskip, st);
        per_cycle += 3;
      } else if (fused_mgs) {
        if (!az_from_stage) spmv<T, T>(S.A, Pj, Wv, SPMV_Y, nullptr, gskip, st);
        MgsArgs<T> ma;
        ma.np = np; ma.j = j; ma.w = Wv; ma.V = V; ma.ldv = ldv;
        ma.vnext = (j < m) ? V + (size_t)j * ldv : nullptr;
        ma.parts = mparts;
        ma.ctr = mctr + (size_t)(j - 1) * (m + 2);
        if (staged_mgs) {
          ma.slots = mslots + (size_t)(j - 1) * (m + 2) * num_sms();
          ma.totals = mslots + (size_t)m * (m + 2) * num_sms() + (size_t)(j - 1) * (m + 2);
        }
        ma.err = merr;
        ma.gate = gskip;
        ma.red = red(EPI_GM_NORM, 0, j);
        mgs_column<T>(ma, st);
        per_cycle += az_from_stage ? 1 : 2;
      } else {
        int sa1[2] = {0, 0}, sb1[2] = {2, 0};   // <w, v_1>
        spmv_dot<T, T>(S.A, Pj, Wv, SPMV_Y, nullptr, V, 1, sa1, sb1, red(EPI_GM_H, 1, j), gskip, st);
        ++per_cycle;
        for (int k = 1; k <= j; ++k) {
          const T* Vk = V + (size_t)(k - 1) * ldv;
          DotSel d;
          if (k < j) { d.a[0] = 0; d.b[0] = 4; }   // <w, v_{k+1}>
          else { d.a[0] = 0; d.b[0] = 0; }         // <w, w>
          const T* Vnext = (k < j) ? V + (size_t)k * ldv : nullptr;
          lincomb_dot<T>(np, Wv, Vk, cdev(&K->tmp[1]), Wv, cimm(1.0), nullptr, cimm(0), Vnext, nullptr, d, 1,
                         (k < j) ? red(EPI_GM_H, k + 1, j) : red(EPI_GM_NORM, 0, j), gskip, st);
          ++per_cycle;
        }
      }
      if (j < m && !(fused_mgs && o.gs != PARCEL_B_GS_CGS)) {
        lincomb<T>(np, V + (size_t)j * ldv, Wv, cdev(&K->tmp[2]), nullptr, cimm(0), nullptr, cimm(0), gskip, st);
        ++per_cycle;
      }
    }
    // update_xVec: y = H^-1 e; v0 = V y; x0 = M^-1 v0; x = x0 + x
    gm_backsolve(hb, eb, yb, m, K, gdone, st);
    if (flex) {
      sum_vec<T>(np, X0, Z, ldv, yb, K, gdone, st);
    } else {
      sum_vec<T>(np, V0, V, ldv, yb, K, gdone, st);
      S.M.apply(np, V0, X0, gdone, st);
      ++per_cycle;
    }
    lincomb<T>(np, x, X0, cimm(1.0), x, cimm(1.0), nullptr, cimm(0), gdone, st);
    gm_post(K, m, st);
    per_cycle += 4;
  };
  GraphRunner& G = kw.G;
  const int max_cycles = o.itrmax / m + 2;
  for (int c = 0; c < max_cycles; ++c) {
    if (read_done(K, st)) break;
    G.launch(cycle, o.use_graphs, st);
    launches += per_cycle;
    if (o.on_cycle) (*o.on_cycle)(c);
  }
  KState h = read_state(K, S);
  int merr_h = 0;
  d2h(&merr_h, merr, sizeof(int));
  PB_CHECK(merr_h == 0, PARCEL_B_E_CUDA, "MGS grid barrier timed out");
  SolveOut out;
  out.niter = h.niter;
  out.iret = h.iret;
  out.breakdown = h.breakdown;
  out.launches = launches;
  return out;
}

template <class T>
SolveOut run_krylov(const Options& o, const System<T>& S, const T* b, T* x, double* hist_dev, KrylovWork* keep) {
  KrylovWork own;
  KrylovWork& kw = keep ? *keep : own;
  kw.begin(o, &S, S.extra, b, x, hist_dev);
  ilu_clear_error<T>(S.M.ilu, o.fail_sweep);
  switch (o.solver) {
    case PARCEL_B_SOLVER_CG: return run_pcg<T>(o, S, b, x, hist_dev, kw);
    case PARCEL_B_SOLVER_BICG: return run_bicg<T>(o, S, b, x, hist_dev, kw);
    case PARCEL_B_SOLVER_GMRES: return run_gmres<T>(o, S, b, x, hist_dev, kw);
    default:
      PB_CHECK(false, PARCEL_B_E_UNSUPPORTED, "solver %d is not provided by this build", o.solver);
  }
  return SolveOut{};
}

template void build_system<double>(const Options&, const parcel_b_crs&, bool, System<double>&);
template void build_system<float>(const Options&, const parcel_b_crs&, bool, System<float>&);
template SolveOut run_krylov<double>(const Options&, const System<double>&, const double*, double*,
                                     double*, KrylovWork*);
template SolveOut run_krylov<float>(const Options&, const System<float>&, const float*, float*,
                                    double*, KrylovWork*);

}  // namespace pb
