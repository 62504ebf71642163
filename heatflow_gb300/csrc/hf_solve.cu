// Linear solve of one implicit step, H x = S (linbcg, mod_Sparse.f90:372-434, replaced).
//
// Method.  H is symmetric negative definite, so the reference's Jacobi-preconditioned BiCG is,
// in exact arithmetic, Jacobi-PCG (rr == r, pp == p).  The GPU runs the same iteration as plain CG
// on the symmetrically scaled operator  Ah = S^-1 (-H) S^-1,  S = diag(sqrt|H_II|), whose diagonal
// is 1: identical iterates, no divisions and one coefficient array fewer per pass.
//
// Each step is a refinement loop:
//   x = x0                                                 (RHS kernel)
//   repeat:  r = S - H x (FP64, true residual), test ||r||/||S||        k_residual
//            g = -S^-1 r / sigma ; solve Ah y = g by CG   (FP64, or FP32 in mixed mode)
//            x += sigma S^-1 y                                           k_xupdate
// The reference adds TINY to every x0 when any x0 - T < TINY (mod_evolve.f90:141).  Here the
// first residual is that of x0 + TINY, formed as r(x0) - TINY * (H 1) from a stored row-sum
// vector, and the TINY itself joins x with the first update: the same iterate, without seven
// extra FP64 additions per cell.
//
// GB300 issues FP64 at ~1 TFLOP/s, so the FP64 kernels (residual, x update, FP64 CG) are bound by
// FP64 instructions: they spend them only on the arithmetic itself (no FP64 compares, no FP64
// accumulation of FP32 quantities), and where a condition is the same for a whole launch it selects a
// loop: an FP64 instruction that is predicated off takes the pipe all the same.  The FP32 kernels
// accumulate in FP32 within a block.
//
// The inner solve of one grid is one persistent kernel, of three (choose_solve): k_solve_cluster,
// k_solve_res, k_solve_one.  Batches: k_solve_batch.  Residuals and x update are kernels of their own
// but in small batches (split_solve).  launch_inner_iteration runs the same passes as plain launches.
//
// All solver state is per instance in device memory; tiles of instances that are not in the
// phase a kernel serves return at once (per-instance convergence masks).
#include <algorithm>
#include <climits>
#include <cstddef>
#include <type_traits>

#include "hf_ctx.cuh"

#define HF_FILE_ID 3   // index-check sites of the checked build: 100000 * file + line

namespace hf {

template <typename T> struct Vec;
template <> struct Vec<double> {
  __device__ static double* y(const DevArrays& A) { return A.y; }
  __device__ static double* r(const DevArrays& A) { return A.r; }
  __device__ static double* p(const DevArrays& A) { return A.p; }
  __device__ static double* pb(const DevArrays& A, int64_t k) { return (k & 1) ? A.p2 : A.p; }
  __device__ static double* q(const DevArrays& A) { return A.q; }
  __device__ static const double* ax(const DevArrays& A) { return A.a64x; }
  __device__ static const double* ay(const DevArrays& A) { return A.a64y; }
  __device__ static const double* az(const DevArrays& A) { return A.a64z; }
};
template <> struct Vec<float> {
  __device__ static float* y(const DevArrays& A) { return A.y32; }
  __device__ static float* r(const DevArrays& A) { return A.r32; }
  __device__ static float* p(const DevArrays& A) { return A.p32; }
  __device__ static float* pb(const DevArrays& A, int64_t k) { return (k & 1) ? A.p232 : A.p32; }
  __device__ static float* q(const DevArrays& A) { return A.q32; }
  __device__ static const float* ax(const DevArrays& A) { return A.a32x; }
  __device__ static const float* ay(const DevArrays& A) { return A.a32y; }
  __device__ static const float* az(const DevArrays& A) { return A.a32z; }
};

// ---- step bookkeeping ------------------------------------------------------------------------
__device__ __forceinline__ void begin_step(InstScal& s, int64_t itime) {
  s.itime = itime;
  s.outer_active = (s.status == 0) ? 1 : 0;
  s.inner_active = 0;
  s.refine = 0;
  s.iter = 0;
  s.step_iters = 0;
  s.x0flag = 0;
  s.tiny_pending = 0;
  s.err = 0.0;
  s.hx_fresh = 0;
  s.xw = 0;
  s.phase = s.outer_active ? PH_RES_INIT : PH_IDLE;   // the persistent solve's first round
}

// Finished steps rotate the temperature roles: T^(n-1) <- T^n, T^n <- x (mod_evolve.f90:169-170).
// The stored H x of the final x becomes H T^n, the previous H T^n becomes H T^(n-1); a step that
// ended without a sweep of its final x (accepted at its first residual) leaves no valid product.
__device__ __forceinline__ void end_step(InstScal& s) {
  if (s.status != 0) {
    s.hx_ok = 0;
    return;
  }
  const int r0 = s.role[0], r1 = s.role[1], r2 = s.role[2], r3 = s.role[3];
  s.role[0] = r2;  // x
  s.role[1] = r0;  // old T^n
  s.role[2] = r1;  // free
  s.role[3] = r3;  // free
  if (s.hx_fresh) {
    s.hx_role ^= 1;
    s.hx_ok = s.hx_ok < 2 ? s.hx_ok + 1 : 2;
  } else {
    s.hx_ok = 0;
  }
  s.hx_fresh = 0;
}

__global__ void k_step_begin(DevArrays A, int64_t itime) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kStamps) A.stamps[i] = i == kStampBegin ? gtimer() : 0ull;
  if (i < A.ninst) begin_step(A.scal[i], itime);
}

__global__ void k_step_end(DevArrays A) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) A.stamps[kStampEnd] = gtimer();
  if (i < A.ninst) end_step(A.scal[i]);
}

// The reference adds TINY to every x0 when any x0 - T < TINY (mod_evolve.f90:140-141) so that its
// BiCG never starts from a zero residual.  The TINY moves only the starting point: the system and
// its solution are unchanged.  Under the reference's own stopping rule (HF_STOP_RECURSIVE) the
// iterates follow linbcg's, so the TINY is applied (in the first residual as -TINY * H1, in x with
// the first update).  Under HF_STOP_TRUE every step is accepted on the true residual of its final
// x, whatever the start, and this CG treats a zero residual itself, so the TINY is skipped: one
// FP64 instruction per cell less in the first residual and in the x update (GB300's FP64 pipe
// bounds both).
// (The mixed solve has the true-residual criterion only.)
template <typename T>
__device__ __forceinline__ bool tiny_applies(const DevArrays& A, const InstScal& s) {
  return sizeof(T) == 8 && s.x0flag != 0 && A.opts.criterion == HF_STOP_RECURSIVE;
}
// f(true_type or false_type): a loop instantiated for either value of a uniform condition, because FP64
// instructions that are predicated off take the FP64 pipe all the same.
template <class F>
__device__ __forceinline__ void for_flag(bool flag, F f) {
  if (flag) f(std::true_type{});
  else f(std::false_type{});
}

// ---- neighbour access for the columns of a task ------------------------------------------------
// x neighbours come from the lanes of the same warp (shuffles); lanes at a task edge, periodic
// wraps and the y neighbours are loaded; the z neighbours roll through registers as the block
// marches along z.  Inactive lanes hold zeros, so every lane can take part in the shuffles.
constexpr unsigned kFull = 0xffffffffu;

// Value and z-face of plane z0-1 of chunk j (zeros at a non-periodic bottom face).
template <typename T, typename C, class V>
__device__ __forceinline__ void plane_below(const DevArrays& A, const TCell& c, int j, V v,
                                            const C* __restrict__ cz, T& vm, C& czm) {
  vm = T(0);
  czm = C(0);
  if (!c.act(j) || c.nz < 2) return;
  int l;
  if (c.z0 > 0) l = c.base(j) + (c.z0 - 1) * c.nxy;
  else if (c.pz) l = c.base(j) + (c.nz - 1) * c.nxy;
  else return;
  vm = v(l);
  czm = cz[HF_IX(A, l, c.n())];
}

template <typename T, class V>
__device__ __forceinline__ T plane_above(const TCell& c, int j, V v, int z) {
  if (!c.act(j) || c.nz < 2) return T(0);
  if (z + 1 < c.nz) return v(c.base(j) + (z + 1) * c.nxy);
  if (c.pz) return v(c.base(j));
  return T(0);
}

// FP32 block sum of one value into *dst, a partial sum of a task (one conversion per block).
__device__ __forceinline__ void task_store_f(double* dst, float v) {
  __shared__ float red[kBlock / 32];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = lane < kBlock / 32 ? red[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    if (lane == 0) *dst = (double)v;
  }
}

// ---- task bodies ---------------------------------------------------------------------------------
// Each body does one kernel's work for one task; the kernels of the split solve and the persistent
// solve kernels call the same bodies, so every path computes the same bits.  Vectors that some phase of the persistent kernel writes
// (temperature buffers, CG vectors) are read through plain pointers: within one launch they change
// between rounds, so they must not be taken for read-only data.  The operator, S and the scalings
// do not change during a solve and are read through const __restrict__ pointers.
//
// Loads are issued ahead of their use by hand (next plane of a stencil, four planes of an
// element-wise pass), because the compiler may not move a load above a store to a vector it cannot
// prove distinct.

// x-neighbour loads of a column (offsets from the cell, or kNoNbr): lane 0 loads its west
// neighbour, lane 31 its east neighbour, and the first and last columns of a periodic axis their wraps;
// all other x neighbours come from the adjacent lanes by shuffles.
constexpr int kNoNbr = -2147483647 - 1;
struct XEdge { int w, e; };
__device__ __forceinline__ XEdge x_edges(const TCell& c) {
  XEdge r{kNoNbr, kNoNbr};
  if (!c.act(0)) return r;
  const int x = c.x(0), nx = c.nx;
  if (x == 0) {
    if (c.px && nx > 1) r.w = nx - 1;
  } else if (c.lane == 0) {
    r.w = -1;
  }
  if (x + 1 < nx) {
    if (c.lane == 31) r.e = 1;
  } else if (c.px && nx > 1) {
    r.e = -(nx - 1);
  }
  return r;
}
// y-neighbour offsets (north = +y, south = -y) of an active column, or kNoNbr.
__device__ __forceinline__ int y_north(const TCell& c) {
  if (!c.act(0) || c.ny < 2) return kNoNbr;
  if (c.y + 1 < c.ny) return c.nx;
  return c.py ? -(c.ny - 1) * c.nx : kNoNbr;
}
__device__ __forceinline__ int y_south(const TCell& c) {
  if (!c.act(0) || c.ny < 2) return kNoNbr;
  if (c.y > 0) return -c.nx;
  return c.py ? (c.ny - 1) * c.nx : kNoNbr;
}

__device__ __forceinline__ float2 pair_of(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 pair_of(double a, double b) { return make_double2(a, b); }

// First residual of a step from the products the last two steps stored: x0 = T^n + (T^n - T^(n-1))
// (mod_evolve.f90:141), so S - H x0 = S - 2 H T^n + H T^(n-1) up to the rounding of x0 (~1e-16 of
// the terms).  Pointwise: 40 B and 4 FP64 instructions per cell (mixed) instead of the stencil
// sweep's 64 B and 9.  The step's acceptance test stays the FP64 residual of the final x.  Bound by
// HBM and the FP64 pipe alike; the loads of U pairs are issued together (256^3 slab 144 -> 120 us, 64
// uneven grids 242 -> 121, against passes over column tiles).
template <typename TR>
__device__ __forceinline__ void res_hx_task(const DevArrays& A, double* part, int64_t task,
                                            const InstScal& s) {
  constexpr bool F32 = sizeof(TR) == 4;
  constexpr int U = F32 ? 4 : 2;
  const Chunk c = task_chunk(A, task);
  const InstDesc& d = *c.d;
  const double* __restrict__ b = A.b + d.off;
  const double* __restrict__ yc = A.hx[s.hx_role] + d.off;
  const double* __restrict__ yp = A.hx[1 - s.hx_role] + d.off;
  const double* __restrict__ rsum = A.rsum + d.off;
  const TR* __restrict__ sinv;
  if constexpr (F32) sinv = A.sinv32 + d.off;
  else sinv = A.sinv + d.off;
  TR* R = Vec<TR>::r(A) + d.off4;             // the inner solve's layout
  [[maybe_unused]] const int n = d.n, n4 = d.sx * d.ny * d.nz;
  const float isig = (float)(1.0 / s.sigma);
  const bool tiny = tiny_applies<TR>(A, s);       // the residual of x0 + TINY: r(x0) - TINY * H1
  double rr = 0.0, gg64 = 0.0;
  float gg = 0.f;
  SqSum rq;                                    // mixed: ||r||^2 off the FP64 pipe
  auto cell = [&](auto with_tiny, double bv, double cv, double pv, TR si, int l) -> TR {
    double a = fma(-2.0, cv, bv);
    a = a + pv;
    if constexpr (decltype(with_tiny)::value) a = fma(-kTiny, rsum[l], a);
    if constexpr (F32) {
      rq.add(a);
      const float g = -si * f64_to_f32_trunc(a) * isig;
      gg = fmaf(g, g, gg);
      return g;
    } else {
      rr = fma(a, a, rr);
      const double g = -si * a;
      gg64 = fma(g, g, gg64);
      return g;
    }
  };
  auto cells = [&](auto with_tiny) {
    for (unsigned l0 = c.first(); l0 < c.end; l0 += c.step * U) {
      double2 bv[U], cv[U], pv[U];
      decltype(ld_pair(sinv, 0, true)) sv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned l = l0 + c.step * u;
        if (l >= c.end) continue;
        const bool two = l + 1 < c.end;
        const int lc = HF_IXP(A, l, n, two);
        bv[u] = ld_pair(b, lc, two);
        cv[u] = ld_pair(yc, lc, two);
        pv[u] = ld_pair(yp, lc, two);
        sv[u] = ld_pair(sinv, lc, two);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned l = l0 + c.step * u;
        if (l >= c.end) continue;
        const bool two = l + 1 < c.end;
        const TR g0 = cell(with_tiny, bv[u].x, cv[u].x, pv[u].x, sv[u].x, l);
        TR g1 = TR(0);
        if (two) g1 = cell(with_tiny, bv[u].y, cv[u].y, pv[u].y, sv[u].y, l + 1);
        if (c.rows4) {
          st_pair(R, HF_IXP(A, l, n4, two), two, pair_of(g0, g1));
        } else {
          R[HF_IX(A, c.inner(l), n4)] = g0;
          if (two) R[HF_IX(A, c.inner(l + 1), n4)] = g1;
        }
      }
    }
  };
  if constexpr (F32) cells(std::false_type{});
  else for_flag(tiny, cells);
  if constexpr (F32) {
    rr = rq.value();
    task_store_f(part + A.pcap + task, gg);
    const double v[1] = {rr};
    tile_store<1>(part + task, A.pcap, v);
  } else {
    const double v[2] = {rr, gg64};
    tile_store<2>(part + task, A.pcap, v);
  }
}

// FP64 true residual of one task: r = S - H x with x in the x-read buffer (INIT: x0 from the RHS
// kernel) or, after an update, in the x-write buffer (the epilogue then swaps the roles).  Writes
// g = -S^-1 r / sigma into the inner residual (type TR).  FP64 work per cell: 7 FMA for S - Hx,
// 1 FMA for ||r||^2 on the FP64 path (the mixed path sums it in FP32, SqSum); after an update
// also H x = S - r into hx[1 - hx_role] (1 subtraction).
template <bool INIT, typename TR, bool XOUT = false>
__device__ __forceinline__ void res_task(const DevArrays& A, double* part, int64_t task,
                                          const InstScal& s) {
  if (INIT && s.hx_ok >= 2) {
    res_hx_task<TR>(A, part, task, s);
    return;
  }
  const TCell c = task_cell(A, task);
  const int64_t off = c.off;
  const double* X = A.tbuf[INIT ? s.role[2] : s.role[3]] + off;
  const double* __restrict__ diag = A.diag + off;
  const double* __restrict__ b = A.b + off;
  const double* __restrict__ cx = A.cx + off;
  const double* __restrict__ cy = A.cy + off;
  const double* __restrict__ cz = A.cz + off;
  const double* __restrict__ rsum = A.rsum + off;
  const float* __restrict__ sinv32 = A.sinv32 + off;
  const double* __restrict__ sinv = A.sinv + off;
  TR* R = Vec<TR>::r(A) + c.off4;             // the inner solve's layout
  const int rxy = c.nxy4, rbase = c.base4(0);
  double* HX = A.hx[1 - s.hx_role] + off;
  // host-buffer steps (the persistent solve of their graphs): x into the result buffer too
  double* XO = (XOUT && !INIT) ? A.xout + A.inst[c.inst].hoff : nullptr;
  const float isig = (float)(1.0 / s.sigma);
  // mixed: ||r||^2 summed in FP32 over per-thread scaled r (one FP64 instruction less per cell on
  // this FP64-bound sweep)
  SqSum rq;
  // INIT: the residual of x0 + TINY (mod_evolve.f90:141) is r(x0) - TINY * H1
  const bool tiny = INIT && tiny_applies<TR>(A, s);
  const bool act = c.act(0);
  const int nz = c.nz, nxy = c.nxy, base = c.base(0);
  const XEdge xe = x_edges(c);
  const int yn = y_north(c), ys = y_south(c);
  const int n = c.n();
  auto xval = [&](int m) -> double { return X[HF_IX(A, m, n)]; };
  // the operands of a plane; those of the next are loaded while one is computed
  struct Plane {
    double up, diag, b, cx, cy, cz, cys, xn, xs, xw, cxw, xe, rs, si;
    float si32;
  };
  auto load = [&](int z, Plane& o) {
    o.up = plane_above<double>(c, 0, xval, z);
    o.xw = o.cxw = o.xe = o.xn = o.xs = o.cys = o.rs = o.si = 0.0;
    o.cx = o.diag = o.b = o.cy = o.cz = 0.0;
    o.si32 = 0.f;
    if (!act) return;
    const int l = base + z * nxy, lc = HF_IX(A, l, n);
    o.diag = diag[lc];
    o.b = b[lc];
    o.cx = cx[lc];
    o.cy = cy[lc];
    o.cz = cz[lc];
    if (tiny) o.rs = rsum[lc];
    if (xe.w != kNoNbr) { o.xw = xval(l + xe.w); o.cxw = cx[HF_IX(A, l + xe.w, n)]; }
    if (xe.e != kNoNbr) o.xe = xval(l + xe.e);
    if (yn != kNoNbr) o.xn = xval(l + yn);
    if (ys != kNoNbr) { o.cys = cy[HF_IX(A, l + ys, n)]; o.xs = xval(l + ys); }
    if (sizeof(TR) == 4) o.si32 = sinv32[lc];
    else o.si = sinv[lc];
  };
  double xm, czm;
  plane_below<double>(A, c, 0, xval, cz, xm, czm);
  double xc = act ? xval(base + c.z0 * nxy) : 0.0;
  double rr = 0.0, gg64 = 0.0;
  float gg = 0.f;
  Plane cur, nxt;
  load(c.z0, cur);
  for (int z = c.z0; z < c.z1; ++z) {
    if (z + 1 < c.z1) load(z + 1, nxt);
    const double up = __shfl_up_sync(kFull, xc, 1), cup = __shfl_up_sync(kFull, cur.cx, 1);
    const double dn = __shfl_down_sync(kFull, xc, 1);
    if (act) {
      const bool west = c.lane > 0 && c.x(0) > 0;
      const double xw = west ? up : cur.xw, cxw = west ? cup : cur.cxw;
      const double xeast = (c.x(0) + 1 < c.nx && c.lane < 31) ? dn : cur.xe;
      double a = fma(-cur.diag, xc, cur.b);
      if (tiny) a = fma(-kTiny, cur.rs, a);
      a = fma(-cur.cx, xeast, a);
      a = fma(-cxw, xw, a);
      if (yn != kNoNbr) a = fma(-cur.cy, cur.xn, a);
      if (ys != kNoNbr) a = fma(-cur.cys, cur.xs, a);
      if (nz > 1) {
        a = fma(-cur.cz, cur.up, a);
        a = fma(-czm, xm, a);
      }
      if (sizeof(TR) == 8) rr = fma(a, a, rr);
      else rq.add(a);
      const int lc = HF_IX(A, base + z * nxy, n);
      if (!INIT) HX[lc] = cur.b - a;
      if (XOUT && !INIT) XO[lc] = xc;
      if (sizeof(TR) == 4) {             // mixed: g in FP32, scaled by 1/sigma
        const float g = -cur.si32 * f64_to_f32_trunc(a) * isig;
        R[HF_IX(A, rbase + z * rxy, c.n4())] = (TR)g;
        gg = fmaf(g, g, gg);
      } else {                           // FP64 path: sigma = 1
        const double g = -cur.si * a;
        R[HF_IX(A, rbase + z * rxy, c.n4())] = (TR)g;
        gg64 = fma(g, g, gg64);
      }
    }
    czm = cur.cz;
    xm = xc;
    xc = cur.up;
    cur = nxt;
  }
  if (sizeof(TR) == 4) rr = rq.value();
  if (sizeof(TR) == 4) {
    task_store_f(part + A.pcap + task, gg);
    const double v[1] = {rr};
    tile_store<1>(part + task, A.pcap, v);
  } else {
    const double v[2] = {rr, gg64};
    tile_store<2>(part + task, A.pcap, v);
  }
}

// The inner solution y at the end of an inner solve.  A direction p_k enters y one pass late, in
// the pass that forms p_(k+1) and reads p_k anyway (pq_task): the last one is still missing where
// the solve ended on a CG update (InstScal::ypend).  old, last: which of y and p are read.
template <typename T>
struct YEnd {
  T alpha;
  bool old, last;
  __device__ __forceinline__ explicit YEnd(const InstScal& s)
      : alpha((T)s.alpha), old(s.ypend == 0 || s.iter > 1), last(s.ypend != 0) {}
  __device__ __forceinline__ T operator()(T y, T p) const {
    return last ? fma(alpha, p, old ? y : T(0)) : y;
  }
};

// Solution update of some cells: x_new = x + sigma S^-1 y (+ TINY once).  Bound by HBM (256^3 slab 94 ->
// 78 us, 5.9 TB/s).
template <typename TY>
__device__ __forceinline__ void xupd_cells(const DevArrays& A, const Chunk& c, const InstScal& s) {
  constexpr bool F32 = sizeof(TY) == 4;
  const InstDesc& d = *c.d;
  const double* XR = A.tbuf[s.role[2]] + d.off;
  double* XW = A.tbuf[s.role[3]] + d.off;
  const TY* Y = Vec<TY>::y(A) + d.off4;       // the inner solve's layout
  const TY* P = Vec<TY>::pb(A, s.iter - 1) + d.off4;
  const YEnd<TY> ye(s);
  const TY* __restrict__ sinv;
  if constexpr (F32) sinv = A.sinv32 + d.off;
  else sinv = A.sinv + d.off;
  [[maybe_unused]] const int n = d.n, n4 = d.sx * d.ny * d.nz;
  const bool use_y = s.iter > 0;
  const bool tiny = !F32 && s.tiny_pending != 0;
  const float sig = (float)s.sigma_prev;
  auto inner = [&](const TY* v, int l, bool two) {
    if (c.rows4) return ld_pair(v, HF_IXP(A, l, n4, two), two);
    return pair_of(v[HF_IX(A, c.inner(l), n4)], two ? v[HF_IX(A, c.inner(l + 1), n4)] : TY(0));
  };
  auto cell = [&](auto with_tiny, double x, TY y, TY si) -> double {
    if constexpr (decltype(with_tiny)::value) x = x + kTiny;
    if (use_y) {
      if constexpr (F32) x = x + f32_to_f64(sig * si * y);
      else x = fma(si, y, x);                 // sigma = 1 on the FP64 path
    }
    return x;
  };
  auto cells = [&](auto with_tiny) {
    for (unsigned l = c.first(); l < c.end; l += c.step) {
      const bool two = l + 1 < c.end;
      decltype(ld_pair(sinv, 0, true)) y{}, p{}, si{};
      const double2 x = ld_pair(XR, HF_IXP(A, l, n, two), two);
      if (use_y) {
        if (ye.old) y = inner(Y, l, two);
        if (ye.last) p = inner(P, l, two);
        si = ld_pair(sinv, HF_IXP(A, l, n, two), two);
      }
      st_pair(XW, HF_IXP(A, l, n, two), two,
              make_double2(cell(with_tiny, x.x, ye(y.x, p.x), si.x), cell(with_tiny, x.y, ye(y.y, p.y), si.y)));
    }
  };
  if constexpr (F32) cells(std::false_type{});
  else for_flag(tiny, cells);
}

// ---- the inner solve's passes ------------------------------------------------------------------
// An inner CG iteration is two passes over the vectors of type T, each ended by the sum it forms:
//   pq:   y += alpha p_(k-1), p_k = r + beta p_(k-1), q = Ah p_k, p.q     (9 T per cell)
//   upd:  r -= alpha q, r.r                                               (3 T per cell)
// y takes a direction one pass late, where p_(k-1) is read anyway (YEnd adds the last one), and p
// is formed by the pass that applies Ah to it: 12 T per cell and iteration against 14 with a
// direction update of its own and y in the second pass, and two grid-wide sums instead of three
// rounds.  Iteration 0 has p_0 = r and no y.
//
// Tasks (InstDesc::cgn of them): a block's thread owns one 16-byte vector (4 FP32 or 2 FP64 cells)
// of a tile of cgw vectors x cgr rows and marches the task's planes along z.  The operands
// come through shared memory (cp.async), two planes ahead of the one that is computed: loads to
// registers left the distance to the compiler, whose schedule of the same loop took 110 to 157 us at
// 256^3 depending on the code around it.  p is formed once per cell, from r and p_(k-1), and shared:
// three planes of the tile with the cells around it, whose p is formed from their r and p_(k-1) as well
// (the value that their own tile stores) by threads that take one such vector or cell each.  One
// block barrier per plane.
// The shared memory starts on 128 bytes: 48 bytes off, the passes at 256^3 took 124 and 36 us instead of
// 108 and 30 (32 bytes off: 111 and 30).
// The rows of the inner solve's layout are padded to 4 cells: in a row's last vector the cells past
// nx have zero coefficients, and q and r are kept zero there.  A face that does not exist has a
// zero coefficient or a zero neighbour.
// Bound by HBM in FP32 and by the FP64 pipe in FP64 (9 instructions per cell).  Measured on the
// layered slab: 256^3 FP32, pq 108 us (5.6 TB/s) and upd 30 us (6.7 TB/s), where the direction
// update, the SpMV and the update took 38 + 68 + 75 us; 190 x 192 x 192 FP64, 134 + 30 us against
// 34 + 111 + 68 us.
template <typename T>
struct alignas(16) Vec16 {
  static constexpr int N = 16 / (int)sizeof(T);
  T v[N];
};
template <typename T>
__device__ __forceinline__ Vec16<T> ld16(const T* p) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  return *reinterpret_cast<const Vec16<T>*>(&u);
}
template <typename T>
__device__ __forceinline__ Vec16<T> ld16cg(const T* p) {   // from L2
  const uint4 u = __ldcg(reinterpret_cast<const uint4*>(p));
  return *reinterpret_cast<const Vec16<T>*>(&u);
}
template <typename T>
__device__ __forceinline__ void st16(T* p, const Vec16<T>& v) {
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(&v);
}

// p of three planes: rows -1..rows of a tile, each of nq vectors with one more at either end (the
// cell beside the row's first is the last of its vector, the cell beside its last the first of its
// vector).  A stage holds what one plane's step needs, by thread: r, p_(k-1) and y of the plane above
// and the plane's own faces; and of the vectors and cells beyond the tile r and p_(k-1) of the plane
// above and the plane's y or x faces.
constexpr int kPqStages = 3;
template <typename T>
struct PqShared {
  struct Stage {
    Vec16<T> r[kBlock], po[kBlock], y[kBlock], ax[kBlock], ay[kBlock], az[kBlock];
    Vec16<T> hr[kTileHalo], hpo[kTileHalo], hf[kTileHalo];
  } st[kPqStages];
  Vec16<T> p[3][kTilePlane];
};
template <typename T>
constexpr int kPqSmem = (int)sizeof(PqShared<T>);   // 99 KB: two blocks per SM
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
template <typename T>
__device__ __forceinline__ void cp16(Vec16<T>* dst, const T* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
template <typename T>
__device__ __forceinline__ void cp1(T* dst, const T* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src), "n"((int)sizeof(T))
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// This thread's groups of copies have arrived, but for the newest N.
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Place of a thread in task `local` of the inner solve's passes.
struct CgPos {
  int x, y, z0, z1, vx, ry, x0, y0;
  bool act;
};
template <typename T>
__device__ __forceinline__ CgPos cg_pos(const InstDesc& d, int local) {
  const int bx = local % d.cgnx, rest = local / d.cgnx, by = rest % d.cgny, bz = rest / d.cgny;
  CgPos c;
  c.ry = (int)(threadIdx.x / (unsigned)d.cgw);
  c.vx = (int)threadIdx.x - c.ry * d.cgw;
  c.x0 = bx * d.cgw * Vec16<T>::N;
  c.y0 = by * d.cgr;
  c.x = c.x0 + c.vx * Vec16<T>::N;
  c.y = c.y0 + c.ry;
  c.z0 = (int)((int64_t)bz * d.nz / d.cgnz);
  c.z1 = (int)((int64_t)(bz + 1) * d.nz / d.cgnz);
  c.act = c.x < d.nx && c.y < d.ny && c.ry < d.cgr;
  return c;
}

// The vector or cell beyond a tile that a thread also forms: threads 0..nq-1 the row above the tile's
// last one, nq..2nq-1 the row below its first (with that row's y faces), then the cells beside the first
// column (with their x faces) and beside the last.  hl: its cell in a plane, or -1; hp: its place in the
// tile's plane of p; hvec: a vector; hc: with a face (ay, or ax for a cell).
struct Beyond { int hl, hp; bool hvec, hc; };
template <typename T>
__device__ __forceinline__ Beyond beyond_of(const InstDesc& d, const CgPos& c) {
  constexpr int V = Vec16<T>::N;
  const int tid = threadIdx.x, nq = d.cgw, rows = d.cgr, prow = nq + 2;
  const int nx = d.nx, ny = d.ny, sx = d.sx;
  const int nv = min(nq, (nx - c.x0 + V - 1) / V), nr = min(rows, ny - c.y0);   // vectors, rows in use
  Beyond b{-1, 0, true, false};
  if (tid < 2 * nq) {
    const int v = tid < nq ? tid : tid - nq, xv = c.x0 + v * V;
    if (v < nv && ny > 1) {
      if (tid < nq) {
        if (c.y0 + nr < ny) b.hl = (c.y0 + nr) * sx + xv;
        else if (d.py) b.hl = xv;
        b.hp = (nr + 1) * prow + v + 1;
      } else {
        if (c.y0 > 0) b.hl = (c.y0 - 1) * sx + xv;
        else if (d.py) b.hl = (ny - 1) * sx + xv;
        b.hp = v + 1;
        b.hc = true;
      }
    }
  } else if (tid < 2 * nq + 2 * rows) {
    const bool west = tid < 2 * nq + rows;
    const int row = tid - 2 * nq - (west ? 0 : rows);
    b.hvec = false;
    if (row < nr) {
      const int lr = (c.y0 + row) * sx, xe = c.x0 + nv * V;
      if (west) {
        if (c.x0 > 0) b.hl = lr + c.x0 - 1;
        else if (d.px && nx > 1) b.hl = lr + nx - 1;
        b.hp = (row + 1) * prow;
        b.hc = true;
      } else {
        if (xe < nx) b.hl = lr + xe;
        else if (d.px && nx > 1) b.hl = lr;
        b.hp = (row + 1) * prow + nv + 1;
      }
    }
  }
  return b;
}

// The sum of a pass over a task.  FP32 sums cover at most 8192 cells, 8 planes of the 4 cells of each
// thread: a task of no more planes is added up in FP32, of a deeper one every 8 planes a warp's, and
// these in FP64 (ms a step against sums in FP32 to the end: 64 uneven grids 2.56 -> 2.58, 256^3 1.402 -> 1.405).
template <typename T>
struct TaskSum {
  static constexpr int kPlanes = 8;
  T part = T(0);                              // of the present group of planes
  double whole = 0.0;                         // of those before it: the warp's
  __device__ __forceinline__ T warp_part() const {
    T v = part;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
  }
  // a group of kPlanes ends, and not the task with it (all threads)
  __device__ __forceinline__ void group() {
    if constexpr (sizeof(T) == 4) {
      whole += f32_to_f64(warp_part());
      part = T(0);
    }
  }
  __device__ __forceinline__ void store(double* slot, int planes) {
    if constexpr (sizeof(T) == 4) {
      if (planes <= kPlanes) {
        task_store_f(slot, part);
        return;
      }
      // a round waits for this: the FP64 adds by one warp, the last group's among them
      __shared__ double red[kBlock / 32];
      __shared__ float last[kBlock / 32];
      const float v = warp_part();
      __syncthreads();
      if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = whole;
        last[threadIdx.x >> 5] = v;
      }
      __syncthreads();
      if (threadIdx.x < 32) {
        const int w = threadIdx.x & (kBlock / 32 - 1);
        double t = red[w] + f32_to_f64(last[w]);
#pragma unroll
        for (int o = kBlock / 64; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
        if (threadIdx.x == 0) *slot = t;
      }
    } else {
      const double v[1] = {part};
      tile_store<1>(slot, 0, v);
    }
  }
};

// off: the instance's first cell (d.off4; a constant 0 where there is one instance keeps the base
// pointers out of the registers).  pslot: the place of the task's sum; dyn: kPqSmem<T> bytes of
// shared memory.
template <typename T, bool FIRST>
__device__ __forceinline__ void pq_form(const DevArrays& A, const InstDesc& d, int64_t off, int local,
                                        const InstScal& s, double* pslot, char* dyn) {
  constexpr int V = Vec16<T>::N;
  typedef Vec16<T> VT;
  PqShared<T>& sm = *reinterpret_cast<PqShared<T>*>(dyn);
  const CgPos c = cg_pos<T>(d, local);
  const int tid = threadIdx.x, nq = d.cgw, rows = d.cgr, prow = nq + 2;
  const int nx = d.nx, ny = d.ny, nz = d.nz, sx = d.sx, nxy = sx * ny;
  [[maybe_unused]] const int n4 = nxy * nz;
  const int z0 = c.z0, z1 = c.z1;
  const bool act = c.act;
  const int last = min(V - 1, nx - 1 - c.x);   // the vector's last grid cell; cells past it are padding
  const int64_t k = s.iter;
  const T beta = (T)s.beta, alpha = (T)s.alpha;      // alpha: of the previous iteration
  const T* R = Vec<T>::r(A) + off;
  const T* Po = Vec<T>::pb(A, k + 1) + off;
  T* Pn = Vec<T>::pb(A, k) + off;
  T* Q = Vec<T>::q(A) + off;
  T* Y = Vec<T>::y(A) + off;
  const T* __restrict__ ax = Vec<T>::ax(A) + off;
  const T* __restrict__ ay = Vec<T>::ay(A) + off;
  const T* __restrict__ az = Vec<T>::az(A) + off;
  const int lxy = c.y * sx + c.x;
  const int own = (c.ry + 1) * prow + c.vx + 1;
  const Beyond by = beyond_of<T>(d, c);
  const int hl = by.hl, hp = by.hp;
  const bool hvec = by.hvec, hc = by.hc;
  // where the faces below this thread's row and beside its first cell come from
  const bool hsouth = ny > 1 && (c.y > 0 || d.py), hwest = nx > 1 && (c.x > 0 || d.px);
  const VT zero{};
  auto form = [&](const VT& r, const VT& po) -> VT {
    VT p;
#pragma unroll
    for (int i = 0; i < V; ++i) p.v[i] = FIRST ? r.v[i] : fma(beta, po.v[i], r.v[i]);
    return p;
  };
  auto above = [&](int z) { return z < nz || (d.pz && nz > 1); };   // plane z, or the wrap of z = nz
  const bool rdy = act && k > 1;
  // the copies of plane z's step
  auto issue = [&](int z, typename PqShared<T>::Stage& st) {
    if (z < z1) {
      const int za = z + 1 < nz ? z + 1 : 0;   // the plane above (or its wrap)
      if (act) {
        if (above(z + 1)) {
          const int l = HF_IXV(A, lxy + za * nxy, n4, V);
          cp16(&st.r[tid], R + l);
          if (!FIRST) cp16(&st.po[tid], Po + l);
          if (rdy && z + 1 < z1) cp16(&st.y[tid], Y + l);
        }
        const int l = HF_IXV(A, lxy + z * nxy, n4, V);
        cp16(&st.ax[tid], ax + l);
        cp16(&st.ay[tid], ay + l);
        cp16(&st.az[tid], az + l);
      }
      if (hl >= 0) {
        if (hvec) {
          if (z + 1 < z1) {
            const int l = HF_IXV(A, hl + za * nxy, n4, V);
            cp16(&st.hr[tid], R + l);
            if (!FIRST) cp16(&st.hpo[tid], Po + l);
          }
          if (hc) cp16(&st.hf[tid], ay + HF_IXV(A, hl + z * nxy, n4, V));
        } else {
          if (z + 1 < z1) {
            const int l = HF_IX(A, hl + za * nxy, n4);
            cp1(&st.hr[tid].v[0], R + l);
            if (!FIRST) cp1(&st.hpo[tid].v[0], Po + l);
          }
          if (hc) cp1(&st.hf[tid].v[0], ax + HF_IX(A, hl + z * nxy, n4));
        }
      }
    }
    cp_commit();
  };
  // p of a plane of the task: stored, and p_(k-1) goes into y
  auto keep = [&](int z, const VT& p, const VT& po, const VT& yv) {
    const int l = HF_IXV(A, lxy + z * nxy, n4, V);
    st16(Pn + l, p);
    if constexpr (!FIRST) {
      VT yn;
#pragma unroll
      for (int i = 0; i < V; ++i) yn.v[i] = fma(alpha, po.v[i], yv.v[i]);   // y is 0 before p_0
      st16(Y + l, yn);
    }
  };
  __syncthreads();                            // the block's previous task is done with shared memory
#pragma unroll
  for (int i = 0; i < kPqStages - 1; ++i) issue(z0 + i, sm.st[i]);
  // the first plane and the one below the task, on their way at the same time
  VT r = zero, po = zero, yv = zero, rb = zero, pob = zero, azm = zero, hr = zero, hpo = zero;
  if (act) {
    const int l = HF_IXV(A, lxy + z0 * nxy, n4, V);
    r = ld16(R + l);
    if (!FIRST) po = ld16(Po + l);
    if (rdy) yv = ld16(Y + l);
    int lb = -1;
    if (nz > 1 && z0 > 0) lb = lxy + (z0 - 1) * nxy;
    else if (nz > 1 && d.pz) lb = lxy + (nz - 1) * nxy;
    if (lb >= 0) {
      lb = HF_IXV(A, lb, n4, V);
      rb = ld16(R + lb);
      if (!FIRST) pob = ld16(Po + lb);
      azm = ld16(az + lb);
    }
  }
  if (hl >= 0) {
    if (hvec) {
      const int l = HF_IXV(A, hl + z0 * nxy, n4, V);
      hr = ld16(R + l);
      if (!FIRST) hpo = ld16(Po + l);
    } else {
      const int l = HF_IX(A, hl + z0 * nxy, n4);
      hr.v[0] = R[l];
      if (!FIRST) hpo.v[0] = Po[l];
    }
  }
  for (int i = tid; i < 3 * kTilePlane; i += kBlock) sm.p[0][i] = zero;
  __syncthreads();
  auto put_beyond = [&](VT* pl, const VT& hr, const VT& hpo) {
    if (hvec) pl[hp] = form(hr, hpo);
    else pl[hp].v[hc ? V - 1 : 0] = FIRST ? hr.v[0] : fma(beta, hpo.v[0], hr.v[0]);
  };
  if (act) {
    const VT p = form(r, po);
    sm.p[0][own] = p;
    sm.p[2][own] = form(rb, pob);
    keep(z0, p, po, yv);
  }
  if (hl >= 0) put_beyond(sm.p[0], hr, hpo);
  TaskSum<T> dot;
  VT *pm = sm.p[2], *pc = sm.p[0], *pu = sm.p[1];
  int si = 0;
  for (int z = z0; z < z1; ++z) {
    typename PqShared<T>::Stage& st = sm.st[si];
    cp_wait<kPqStages - 2>();                 // plane z's step has arrived
    if (act) {
      VT p = zero;
      if (above(z + 1)) {
        const VT po = FIRST ? zero : st.po[tid];
        p = form(st.r[tid], po);
        if (z + 1 < z1) keep(z + 1, p, po, rdy ? st.y[tid] : zero);
      }
      pu[own] = p;
    }
    if (hl >= 0 && z + 1 < z1) put_beyond(pu, st.hr[tid], FIRST ? zero : st.hpo[tid]);
    __syncthreads();                          // p of planes z and z + 1 and all faces of z are there
    {                                         // the stage of plane z - 1, which every thread has left
      int sn = si + kPqStages - 1;
      if (sn >= kPqStages) sn -= kPqStages;
      issue(z + kPqStages - 1, sm.st[sn]);
    }
    if (act) {
      const VT axv = st.ax[tid], azv = st.az[tid], ayv = st.ay[tid];
      const VT p = pc[own], pn = pc[own + prow], ps = pc[own - prow], pa = pu[own], pd = pm[own];
      VT ays = zero;
      if (hsouth) ays = c.ry > 0 ? st.ay[tid - nq] : st.hf[nq + c.vx];
      T axw = T(0);
      if (hwest) axw = c.vx > 0 ? st.ax[tid - 1].v[V - 1] : st.hf[2 * nq + c.ry].v[0];
      const T pw = pc[own - 1].v[V - 1], pe = pc[own + 1].v[0];
      VT qv;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const T pi = p.v[i];
        T acc = pi;
        acc = fma(axv.v[i], i < last ? p.v[i < V - 1 ? i + 1 : i] : pe, acc);
        acc = fma(i > 0 ? axv.v[i > 0 ? i - 1 : 0] : axw, i > 0 ? p.v[i > 0 ? i - 1 : 0] : pw, acc);
        acc = fma(ayv.v[i], pn.v[i], acc);
        acc = fma(ays.v[i], ps.v[i], acc);
        acc = fma(azv.v[i], pa.v[i], acc);
        acc = fma(azm.v[i], pd.v[i], acc);
        if (i > last) acc = T(0);             // padding: q stays 0
        dot.part = fma(pi, acc, dot.part);
        qv.v[i] = acc;
      }
      st16(Q + HF_IXV(A, lxy + z * nxy, n4, V), qv);
      azm = azv;
    }
    if (((z - z0) & 7) == 7 && z + 1 < z1) dot.group();
    VT* t = pm;
    pm = pc;
    pc = pu;
    pu = t;
    if (++si == kPqStages) si = 0;
  }
  dot.store(pslot, z1 - z0);
}
// Iteration 0 (p = r, no y) is a form of its own.
template <typename T>
__device__ __forceinline__ void pq_task(const DevArrays& A, const InstDesc& d, int64_t off, int local,
                                        const InstScal& s, double* pslot, char* dyn) {
  if (s.iter == 0) pq_form<T, true>(A, d, off, local, s, pslot, dyn);
  else pq_form<T, false>(A, d, off, local, s, pslot, dyn);
}

// r -= alpha q and r.r (and the unscaled ||r||^2 for the reference rule).  The planes are walked
// downwards: the pass before ended on the task's last ones, which are still in L2.  The iteration
// predicted to end the inner solve also forms x_new = x + sigma S^-1 y (rows of 4k cells: both
// layouts index alike).
// WEIGHTED is a form of its own: as a condition in the loop its FP64 instructions, predicated off,
// took the FP64 pipe all the same (ncu: pipe 72 % busy for 2 FMAs per cell).
// Operands arrive through shared memory (cp.async), two stages ahead of the one that is computed: the
// pq pass's shared memory leaves little L1 for loads in flight (31 us at 256^3 against 39 with loads to
// registers, the form with the x update 119 against 132).
template <typename T>
struct UpdStage { Vec16<T> q[4][kBlock], r[4][kBlock]; };     // four planes
template <typename T>
struct UpdXStage {                                            // one plane
  Vec16<T> q[kBlock], r[kBlock], p[kBlock], y[kBlock], s[kBlock];
  Vec16<double> x[Vec16<T>::N / 2][kBlock];
};
static_assert(3 * sizeof(UpdStage<float>) <= sizeof(PqShared<float>) && 3 * sizeof(UpdStage<double>) <= sizeof(PqShared<double>) &&
                  3 * sizeof(UpdXStage<float>) <= sizeof(PqShared<float>) && 3 * sizeof(UpdXStage<double>) <= sizeof(PqShared<double>),
              "the update's stages fit the pq pass's shared memory");
template <typename T, bool WEIGHTED>
__device__ __forceinline__ void upd_form(const DevArrays& A, const InstDesc& d, int local, const InstScal& s,
                                         double* pslot, int64_t stride, char* dyn) {
  constexpr int V = Vec16<T>::N;
  typedef Vec16<T> VT;
  const CgPos c = cg_pos<T>(d, local);
  const T alpha = (T)s.alpha;
  const int tid = threadIdx.x;
  const int nxy = d.sx * d.ny, lxy = c.y * d.sx + c.x;
  [[maybe_unused]] const int n4 = nxy * d.nz;
  const int last = min(V - 1, d.nx - 1 - c.x);
  T* R = Vec<T>::r(A) + d.off4;
  const T* Q = Vec<T>::q(A) + d.off4;
  TaskSum<T> rr;
  double rw = 0.0;
  if (!WEIGHTED && (s.xw & kXwThis)) {        // (never under the reference's rule)
    UpdXStage<T>* st = reinterpret_cast<UpdXStage<T>*>(dyn);
    const bool first = s.iter == 0;
    const T* P = Vec<T>::pb(A, s.iter) + d.off4;
    const T* Y = Vec<T>::y(A) + d.off4;
    const double* XR = A.tbuf[s.role[2]] + d.off;
    double* XW = A.tbuf[s.role[3]] + d.off;
    const double* sinv = A.sinv + d.off;
    const float* sinv32 = A.sinv32 + d.off;
    const float sig = (float)s.sigma_prev;
    auto issue = [&](int z, UpdXStage<T>& o) {
      if (c.act && z >= c.z0) {
        const int l = HF_IXV(A, lxy + z * nxy, n4, V);
        cp16(&o.q[tid], Q + l);
        cp16(&o.r[tid], R + l);
        cp16(&o.p[tid], P + l);
        if (!first) cp16(&o.y[tid], Y + l);
        if constexpr (sizeof(T) == 8) cp16(&o.s[tid], sinv + l);
        else cp16(&o.s[tid], sinv32 + l);
#pragma unroll
        for (int i = 0; i < V / 2; ++i) cp16(&o.x[i][tid], XR + l + 2 * i);
      }
      cp_commit();
    };
    issue(c.z1 - 1, st[0]);
    issue(c.z1 - 2, st[1]);
    int si = 0;
    for (int z = c.z1 - 1; z >= c.z0; --z) {
      const UpdXStage<T>& o = st[si];
      cp_wait<1>();
      issue(z - 2, st[si == 0 ? 2 : si - 1]);
      if (c.act) {
        const int l = HF_IXV(A, lxy + z * nxy, n4, V);
        const VT qv = o.q[tid], pv = o.p[tid], fv = o.s[tid];
        VT rv = o.r[tid], yv{};
        if (!first) yv = o.y[tid];
        Vec16<double> xv[V / 2];
#pragma unroll
        for (int i = 0; i < V / 2; ++i) xv[i] = o.x[i][tid];
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const T yo = fma(alpha, pv.v[i], yv.v[i]);
          rv.v[i] = fma(-alpha, qv.v[i], rv.v[i]);
          rr.part = fma(rv.v[i], rv.v[i], rr.part);
          double& x = xv[i / 2].v[i & 1];
          if constexpr (sizeof(T) == 8) x = fma(fv.v[i], yo, x);
          else x = x + f32_to_f64(sig * fv.v[i] * yo);
        }
        st16(R + l, rv);
#pragma unroll
        for (int i = 0; i < V / 2; ++i) st16(XW + l + 2 * i, xv[i]);
      }
      if (((c.z1 - 1 - z) & 7) == 7 && z > c.z0) rr.group();
      if (++si == 3) si = 0;
    }
  } else {
    UpdStage<T>* st = reinterpret_cast<UpdStage<T>*>(dyn);
    constexpr int U = 4;
    auto issue = [&](int zt, UpdStage<T>& o) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!c.act || zt - u < c.z0) continue;
        const int l = HF_IXV(A, lxy + (zt - u) * nxy, n4, V);
        cp16(&o.q[u][tid], Q + l);
        cp16(&o.r[u][tid], R + l);
      }
      cp_commit();
    };
    issue(c.z1 - 1, st[0]);
    issue(c.z1 - 1 - U, st[1]);
    int si = 0;
    for (int zt = c.z1 - 1; zt >= c.z0; zt -= U) {
      const UpdStage<T>& o = st[si];
      cp_wait<1>();
      issue(zt - 2 * U, st[si == 0 ? 2 : si - 1]);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int z = zt - u;
        if (!c.act || z < c.z0) continue;
        const VT qv = o.q[u][tid];
        VT rv = o.r[u][tid];
#pragma unroll
        for (int i = 0; i < V; ++i) {
          T r = fma(-alpha, qv.v[i], rv.v[i]);
          if (i > last) r = T(0);
          rv.v[i] = r;
          rr.part = fma(r, r, rr.part);
          if (WEIGHTED && i <= last) {
            const double dg = A.diag[d.off + HF_IX(A, (z * d.ny + c.y) * d.nx + c.x + i, d.nx * d.ny * d.nz)];
            rw = fma(-dg * (double)r, (double)r, rw);
          }
        }
        st16(R + HF_IXV(A, lxy + z * nxy, n4, V), rv);
      }
      if (((c.z1 - 1 - zt) & 4) && zt - U >= c.z0) rr.group();
      if (++si == 3) si = 0;
    }
  }
  if constexpr (WEIGHTED) {
    const double v[2] = {rr.part, rw};
    tile_store<2>(pslot, stride, v);
  } else {
    rr.store(pslot, c.z1 - c.z0);
  }
}
template <typename T>
__device__ __forceinline__ void upd_task(const DevArrays& A, const InstDesc& d, int local, const InstScal& s,
                                         double* pslot, char* dyn) {
  if (sizeof(T) == 8 && A.opts.criterion == HF_STOP_RECURSIVE)
    upd_form<T, sizeof(T) == 8>(A, d, local, s, pslot, A.pcap, dyn);
  else
    upd_form<T, false>(A, d, local, s, pslot, A.pcap, dyn);
}

// ---- kernels of the split solve; the inner passes on their own -----------------------------------
// A round of the split solve in its log (one thread).
__device__ __forceinline__ void log_round(SolveCtl* ctl, int32_t phase, unsigned long long now) {
  const int64_t r = ctl->rounds;
  if (r < kRoundLog) {
    ctl->phase_log[r] = phase;
    ctl->t_round[r] = now;
  }
  ctl->rounds = r + 1;
}

// log: the split solve's sweeps note their start (the first) and the end of the x update before them.
template <bool INIT, typename TR, bool XOUT = false>
__global__ void __launch_bounds__(kBlock) k_residual(DevArrays A, int log) {
  if (log && blockIdx.x == 0 && threadIdx.x == 0) {
    if (INIT) A.stamps[kStampSolve] = A.sctl->t_start = gtimer();
    else if (A.scal[0].outer_active && !A.scal[0].inner_active && !(A.scal[0].xw & kXwDone))
      log_round(A.sctl, HF_PHASE_XUPD, gtimer());
  }
  const InstScal& s = A.scal[A.tasks[blockIdx.x].x];
  if (!s.outer_active || s.inner_active) return;
  if (INIT != (s.refine == 0)) return;
  res_task<INIT, TR, XOUT>(A, A.partials, blockIdx.x, s);
}

template <typename TY>
__global__ void __launch_bounds__(kBlock) k_xupdate(DevArrays A) {
  const int64_t task = blockIdx.x / kFine;
  const InstScal& s = A.scal[task_inst(A, task)];
  if (!s.outer_active || s.inner_active || s.refine == 0 || (s.xw & kXwDone)) return;
  xupd_cells<TY>(A, task_chunk<kFine>(A, task, (int)(blockIdx.x % kFine)), s);
}

template <typename T>
__global__ void __launch_bounds__(kBlock) k_cg_pq(DevArrays A) {
  extern __shared__ __align__(128) char dyn[];
  const int inst = A.cg_inst[blockIdx.x];
  const InstScal& s = A.scal[inst];
  if (!s.inner_active) return;
  const InstDesc& d = A.inst[inst];
  pq_task<T>(A, d, d.off4, (int)(blockIdx.x - d.cg0), s, A.partials + blockIdx.x, dyn);
}

template <typename T>
__global__ void __launch_bounds__(kBlock) k_cg_upd(DevArrays A) {
  extern __shared__ __align__(128) char dyn[];
  const int inst = A.cg_inst[blockIdx.x];
  const InstScal& s = A.scal[inst];
  if (!s.inner_active) return;
  const InstDesc& d = A.inst[inst];
  upd_task<T>(A, d, (int)(blockIdx.x - d.cg0), s, A.partials + blockIdx.x, dyn);
}

// ---- summation of an instance's task partials ------------------------------------------------
// One order for every path (finalize kernels, all persistent solves), for the tasks that the plan made:
// thread c adds the partials of tasks c, c + kBlock, ... in turn, the eight threads of a lane are
// added as tree8, the lanes as a shuffle tree.  The result is valid in thread 0.  Partials are read
// through L2 (written by other blocks of the same persistent launch); the loads of a pass are
// issued together, because a round of the persistent solve waits for this sum.
constexpr int kSumBatch = 4;
template <int NRV>
__device__ __forceinline__ void strided_sum(const double* part, int64_t stride, int64_t task0,
                                            int64_t ntask, int64_t first, double (&acc)[NRV]) {
  for (int64_t t0 = first; t0 < ntask; t0 += (int64_t)kSumBatch * kBlock) {
    double v[kSumBatch][NRV];
#pragma unroll
    for (int u = 0; u < kSumBatch; ++u) {
      const int64_t t = t0 + (int64_t)u * kBlock;
#pragma unroll
      for (int k = 0; k < NRV; ++k) v[u][k] = t < ntask ? __ldcg(&part[k * stride + task0 + t]) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kSumBatch; ++u) {
      if (t0 + (int64_t)u * kBlock >= ntask) break;
#pragma unroll
      for (int k = 0; k < NRV; ++k) acc[k] += v[u][k];
    }
  }
}

// Block-uniform call (all threads of the block); red: NRV * kBlock values of shared memory.
template <int NRV>
__device__ __forceinline__ void instance_sum(const double* part, int64_t stride, int64_t task0,
                                             int64_t ntask, double (&acc)[NRV], double* red) {
#pragma unroll
  for (int k = 0; k < NRV; ++k) acc[k] = 0.0;
  strided_sum<NRV>(part, stride, task0, ntask, threadIdx.x, acc);
#pragma unroll
  for (int k = 0; k < NRV; ++k) red[k * kBlock + threadIdx.x] = acc[k];
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int k = 0; k < NRV; ++k) {
      double u[8];
#pragma unroll
      for (int w = 0; w < 8; ++w) u[w] = red[k * kBlock + threadIdx.x + 32 * w];
      acc[k] = tree8(u);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int k = 0; k < NRV; ++k) acc[k] += __shfl_xor_sync(kFull, acc[k], o);
    }
  }
}

constexpr int kScalWords = (int)(sizeof(InstScal) / 8);
static_assert(sizeof(InstScal) % 8 == 0 && kScalWords < kBlock, "scalar copy");
constexpr int kDescWords = (int)(sizeof(InstDesc) / 8);
static_assert(sizeof(InstDesc) % 8 == 0 && kDescWords <= kBlock, "descriptor copy");

// ---- finalize kernels: one block per instance sums the task partials in task order ----------
// (deterministic), then runs the scalar epilogue of the producing kernel.

// The power of two nearest to a positive normal v (by its logarithm), 1 for any other: a scale, which
// needs no transcendental function.
__device__ __forceinline__ double near_pow2(double v) {
  const unsigned long long b = dbits(v), m = b & 0xfffffffffffffull;
  const int e = (int)(b >> 52);                // (the sign with it)
  if (e < 1 || e > 0x7fd) return 1.0;
  return bitsd((unsigned long long)(e + (m > 0x6a09e667f3bccull ? 1 : 0)) << 52);   // sqrt(2)
}

// Epilogue of the RHS kernel (mod_evolve.f90:70-127 checks, initial scale of the FP32 rhs).
__device__ void epi_rhs(InstScal& s, const InstDesc& d, const DevOpts& o, const double* tot) {
  s.bb = tot[0];
  s.x0flag = tot[1] > 0.0 ? 1 : 0;
  if (isnan(tot[0])) {              // some S is NaN: which vector failed is diagnosed later
    s.status |= kStatusRhsNan;
    s.outer_active = 0;
    s.failed_step = s.itime;
    s.phase = PH_IDLE;
    return;
  }
  // scale of the first FP32 residual: a power of two near rms(S)/rms(|H_II|^(1/2)) * 1e-6
  const double rms = sqrt(tot[0] / (double)d.n) * d.mean_sinv * 1e-6;
  s.sigma = o.precision == HF_PREC_MIXED ? near_pow2(rms) : 1.0;
}

// Epilogue of the diagnosis pass: the first failing vector in the reference's order.
__device__ void epi_rhs_diag(InstScal& s, const double* tot) {
  int st = 0;
  if (tot[1] > 0) st = 1 << (HF_ENAN_Q - HF_ENAN_B);
  else if (tot[2] > 0) st = 1 << (HF_ENAN_QDENS - HF_ENAN_B);
  else if (tot[3] > 0) st = 1 << (HF_ENAN_SCAT - HF_ENAN_B);
  else if (tot[4] > 0) st = 1 << (HF_ENAN_S - HF_ENAN_B);
  s.status = st ? st : (1 << (HF_ENAN_S - HF_ENAN_B));
}

// Epilogue of a residual sweep: convergence test and set-up of the next inner solve.
// rel, rms: the square roots of ||r||^2 over ||S||^2 and over the number of cells.
template <bool INIT>
__device__ void epi_residual_s(InstScal& s, const InstDesc& G, const DevOpts& o, const double* tot, double rel,
                               double rms_r) {
  s.xw = 0;                              // this sweep consumed any x formed by a CG update
  if (!INIT) {
    const int t = s.role[2]; s.role[2] = s.role[3]; s.role[3] = t;
    s.tiny_pending = 0;
  } else {
    s.tiny_pending = (o.criterion == HF_STOP_RECURSIVE) ? s.x0flag : 0;   // tiny_applies
  }
  s.rr_true = tot[0];
  s.relres = s.bb > 0.0 ? rel : (tot[0] > 0.0 ? INFINITY : 0.0);
  s.refine += 1;
  s.tot_refine += 1;
  if (isnan(tot[0])) {                   // x holds a NaN (mod_evolve.f90:153-158)
    s.status |= 1 << (HF_ENAN_X - HF_ENAN_B);
    s.failed_step = s.itime;
    s.outer_active = 0;
    return;
  }
  bool done, converged;
  if (o.criterion == HF_STOP_RECURSIVE) {
    done = (s.refine >= 2);              // the reference solves once; this sweep only forms x
    converged = true;
  } else {
    converged = (s.relres <= o.tol);
    done = (converged && !s.tiny_pending) || (s.refine > o.max_refine) ||
           (tot[0] == 0.0 && !s.tiny_pending);
  }
  if (done) {
    s.outer_active = 0;
    s.hx_fresh = INIT ? 0 : 1;           // a sweep after an update stored H x of the final x
    if (!converged) s.unconverged += 1;
    s.last_relres = s.relres;
    s.last_err = (o.criterion == HF_STOP_RECURSIVE) ? s.err : s.relres;
    s.last_iter = s.step_iters;
    return;
  }
  s.iter = 0;
  s.ypend = 0;
  if (o.criterion != HF_STOP_RECURSIVE && converged) {   // only the +TINY is left to apply
    s.inner_active = 0;
    return;
  }
  s.inner_active = 1;
  s.gg0 = tot[1];
  s.rho = tot[1];
  s.beta = 0.0;
  s.sigma_prev = s.sigma;
  if (o.precision == HF_PREC_MIXED) {
    s.eta = fmax(o.inner_tol, 0.1 * o.tol / fmax(s.relres, 1e-300));
    s.sigma = near_pow2(rms_r * G.mean_sinv);
  } else {
    s.eta = fmax(0.1 * o.tol / fmax(s.relres, 1e-300), 1e-15);
    s.sigma = 1.0;
  }
  if (!(tot[1] > 0.0)) s.inner_active = 0;  // exact already: go straight to the update
  if (s.inner_active && o.criterion == HF_STOP_TRUE && (G.nx & 3) == 0) {
    const int64_t cap = (o.precision == HF_PREC_MIXED) ? (int64_t)o.inner_itmax : o.itmax;
    s.xw = kXwAllowed | (cap <= 1 ? kXwThis : 0);
  }
}


__device__ void epi_spmv_s(InstScal& s, const double* tot) {
  s.pq = tot[0];
  s.ypend = 0;                           // the pass took the previous direction into y
  if (tot[0] > 0.0 && isfinite(tot[0])) {
    s.alpha = s.rho / tot[0];
  } else {            // breakdown (p = 0 or non-finite): stop this inner solve
    s.alpha = 0.0;
    s.inner_active = 0;
  }
}


// What the epilogue of a CG update divides and roots: r.r over that of the iteration before, over
// the inner solve's first, and the stopping criterion (the reference's on the unscaled recursive
// residual r = -S rh sigma, mod_Sparse.f90:420).
struct UpdRatios { double shrink, first; };
__device__ __forceinline__ double upd_err(const InstScal& s, bool weighted, double rr_w, double first) {
  if (weighted) return s.bb > 0.0 ? sqrt(rr_w) * s.sigma_prev / sqrt(s.bb) : 0.0;
  return s.gg0 > 0.0 ? sqrt(first) : 0.0;
}

// stop: the criterion is met.  The caller sets s.err.
template <typename T>
__device__ __forceinline__ void epi_upd_s(InstScal& s, const DevOpts& o, const double* tot, const UpdRatios& q,
                                          bool stop) {
  const bool weighted = (o.criterion == HF_STOP_RECURSIVE);
  const double rho_new = tot[0];
  s.beta = q.shrink;
  s.rho = rho_new;
  s.iter += 1;
  s.ypend = 1;
  s.step_iters += 1;
  if (sizeof(T) == 8) s.tot_iters += 1; else s.tot_inner += 1;
  if (weighted) s.rr_w = tot[1];
  const int64_t cap = (sizeof(T) == 8) ? o.itmax : (int64_t)o.inner_itmax;
  if (!stop && s.iter >= cap) {
    stop = true;
    if (weighted) s.unconverged += 1;
  }
  if (!(rho_new > 0.0)) stop = true;
  if (stop) s.inner_active = 0;
  // Fused x update: whether the update that just ran formed x, and whether the next one should.
  // The next iteration is predicted to end the solve when it reaches the iteration cap, or when
  // the criterion shrinks once more by this iteration's factor: err_k^2 (rho_k / rho_(k-1)) <= eta^2.
  const int32_t wrote = (s.xw & kXwThis) ? kXwDone : 0;
  s.xw = (s.xw & kXwAllowed) | wrote;
  if (!stop && (s.xw & kXwAllowed)) {
    const double next = q.first * q.shrink;
    if (s.iter + 1 >= cap || next <= s.eta * s.eta) s.xw |= kXwThis;
  }
}


template <typename T>
__device__ __forceinline__ void epi_upd(InstScal& s, const DevOpts& o, const double* tot) {
  const bool weighted = o.criterion == HF_STOP_RECURSIVE;
  const UpdRatios q{tot[0] / s.rho, tot[0] / s.gg0};
  s.err = upd_err(s, weighted, tot[1], q.first);
  epi_upd_s<T>(s, o, tot, q, s.err <= (weighted ? o.tol : s.eta));
}

// Whether instance s took part in the producing kernel (the producers' own entry tests).
template <int KIND>
__device__ __forceinline__ bool took_part(const InstScal& s) {
  switch (KIND) {
    case FIN_RHS: return s.outer_active != 0;
    case FIN_RHS_DIAG: return (s.status & kStatusRhsNan) != 0;
    case FIN_RES_INIT: return s.outer_active && !s.inner_active && s.refine == 0;
    case FIN_PQ:
    case FIN_UPD: return s.inner_active != 0;
    default: return s.outer_active && !s.inner_active && s.refine != 0;      // FIN_RES
  }
}

// One block; a few microseconds of latency that nothing hides (four of them in a step), so all loads are
// issued at once (one grid's sums need no descriptor), the scalars are worked on in shared memory, and
// the two divisions and roots run side by side in two lanes: at 64^3 6.4 -> 4.6 us (a step 4 %
// less), at 128^3 8.3 -> 6.7.
template <int KIND>
__global__ void __launch_bounds__(kBlock) k_finalize(DevArrays A, CtrlState* ctrl,
                                                  cudaGraphConditionalHandle hw, int graph) {
  constexpr int NR = KIND == FIN_RHS_DIAG ? 5 : 2;
  constexpr bool RES = KIND == FIN_RES_INIT || KIND == FIN_RES;
  const int inst = blockIdx.x, tid = threadIdx.x;
  __shared__ InstScal sh;
  __shared__ InstDesc sd;
  __shared__ double red[kBlock * NR];
  const unsigned long long start = gtimer();
  if (RES && A.ninst == 1 && tid == 0) A.sctl->arrived = 0ull;   // of the inner solve that may follow
  if (KIND == FIN_RHS && inst == 0 && tid == 0) A.stamps[kStampFin] = start;
  const bool loop = graph && RES, one = A.ninst == 1;
  int32_t gave_up = 0;
  if (loop && tid == 0) gave_up = A.sctl->err | A.sctl->guard_hit;
  if (tid < kScalWords)
    reinterpret_cast<unsigned long long*>(&sh)[tid] = reinterpret_cast<const unsigned long long*>(A.scal + inst)[tid];
  if (tid < kDescWords)
    reinterpret_cast<unsigned long long*>(&sd)[tid] = reinterpret_cast<const unsigned long long*>(A.inst + inst)[tid];
  if (!one) __syncthreads();
  double acc[NR];
  if (KIND == FIN_PQ || KIND == FIN_UPD)
    instance_sum<NR>(A.partials, A.pcap, one ? 0 : sd.cg0, one ? A.ncg : (int64_t)sd.cgn, acc, red);
  else
    instance_sum<NR>(A.partials, A.pcap, one ? 0 : sd.task0, one ? A.ntasks : (int64_t)sd.ntask, acc, red);
  const bool part = took_part<KIND>(sh);       // (instance_sum holds a block barrier)
  __syncthreads();                             // every thread has looked before the epilogue changes sh
  if (part && tid < 32) {
    double rel = 0.0, rms = 0.0;
    if (RES) {
      const double rr = __shfl_sync(kFull, acc[0], 0), root = sqrt(rr / (tid == 1 ? (double)sd.n : sh.bb));
      rel = root;
      rms = __shfl_sync(kFull, root, 1);
    }
    if (tid == 0) {
      if (graph && inst == 0) {
        log_round(A.sctl, KIND == FIN_RES ? (int32_t)HF_PHASE_RES
                                          : sh.hx_ok >= 2 ? (int32_t)HF_PHASE_RES_INIT_HX : (int32_t)HF_PHASE_RES_INIT,
                  start);
        A.stamps[kStampSolveEnd] = start;
      }
      switch (KIND) {
        case FIN_RHS: epi_rhs(sh, sd, A.opts, acc); break;
        case FIN_RHS_DIAG: epi_rhs_diag(sh, acc); break;
        case FIN_RES_INIT: epi_residual_s<true>(sh, sd, A.opts, acc, rel, rms); break;
        case FIN_PQ: epi_spmv_s(sh, acc); break;
        case FIN_UPD:
          if (A.opts.precision == HF_PREC_MIXED) epi_upd<float>(sh, A.opts, acc);
          else epi_upd<double>(sh, A.opts, acc);
          break;
        default: epi_residual_s<false>(sh, sd, A.opts, acc, rel, rms); break;
      }
    }
  }
  __syncthreads();
  if (part && tid < kScalWords)
    reinterpret_cast<unsigned long long*>(A.scal + inst)[tid] = reinterpret_cast<const unsigned long long*>(&sh)[tid];
  // loop condition of the captured solve loop: set by the last instance block to finish
  if (!loop) return;
  int any_outer = sh.outer_active;
  if (!one) {
    __syncthreads();                           // the scalars are written
    if (tid != 0) return;
    __threadfence();
    if (atomicAdd(&ctrl->fin_count, 1u) != gridDim.x - 1u) return;
    __threadfence();
    any_outer = 0;
    for (int64_t i = 0; i < A.ninst; ++i) any_outer |= __ldcg(&A.scal[i].outer_active);
    ctrl->fin_count = 0u;
  }
  if (tid == 0) {
    // a kernel of the inner solves that gave up leaves its instance as it was: the loop ends there
    if (gave_up) any_outer = 0;
    ctrl->launches += KIND == FIN_RES ? 4 : 0;
    cudaGraphSetConditional(hw, any_outer ? 1u : 0u);
  }
}

// ---- captured step: control kernels of the conditional nodes -----------------------------------
__global__ void k_graph_step_begin(DevArrays A, CtrlState* ctrl, int launches_per_step) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kStamps) A.stamps[i] = i == kStampBegin ? gtimer() : 0ull;
  if (i == 0) {
    ctrl->launches += launches_per_step;   // the step's kernels outside the solve loop
  }
  if (i < A.ninst) begin_step(A.scal[i], ctrl->itime);
}

// One block: every instance rotates, then the step counter advances.  A persistent solve that
// gave up (barrier time limit or round bound) is recorded in ctrl->guard_hit, which stays set.
// In a whole-loop graph (loop != 0) it also sets the WHILE condition: another step follows while
// the step counter is below itime_end and no solve has failed, so the loop always ends.
__global__ void k_graph_step_end(DevArrays A, CtrlState* ctrl, const SolveCtl* sctl,
                                 cudaGraphConditionalHandle hloop, int loop) {
  if (threadIdx.x == 0) A.stamps[kStampEnd] = gtimer();
  for (int64_t i = threadIdx.x; i < A.ninst; i += blockDim.x) end_step(A.scal[i]);
  __syncthreads();
  if (threadIdx.x == 0) {
    ctrl->itime += 1;
    if (sctl && (sctl->err || sctl->guard_hit)) ctrl->guard_hit |= sctl->err ? 2 : 1;
    if (loop) cudaGraphSetConditional(hloop, (ctrl->itime < ctrl->itime_end && !ctrl->guard_hit) ? 1u : 0u);
  }
}

// ---- persistent solve ------------------------------------------------------------------------
// One cooperative launch runs the inner solves that are due, or in a small batch a step's whole
// refinement loop.  An instance goes through phases (PH_*); in a phase every one of its tasks does the
// phase's work, writing its partial sums to its fixed slot; then an epilogue sums the partials in the
// fixed order of instance_sum (the order the finalize kernels use, so every path obtains the same bits)
// and updates the instance's scalars (alpha, beta, convergence test, next phase).  One grid runs its
// phases in grid-wide rounds (k_solve_one); the grids of a batch each at their own pace (k_solve_batch).
//
// Termination: every wait is bounded in time (wait_ns, 4 s by default) and in polls; a block that
// gives up records SolveCtl::err and returns, and the blocks still waiting see the flag and return
// too.  The number of phases is bounded by `limit`.  Co-residency of all blocks, which the grid-wide
// barrier needs, is guaranteed by the cooperative launch (the grid never exceeds the occupancy
// bound).

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_add_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
template <typename T>
__device__ __forceinline__ int32_t phase_after(const InstScal& s) {
  if (!s.outer_active) return PH_IDLE;
  if (s.inner_active) return PH_CG_PQ;
  return (s.xw & kXwDone) ? PH_RES : PH_XUPD;   // the last CG update may have formed x already
}
__device__ __forceinline__ int phase_partials(int32_t ph) {
  return (ph == PH_RES_INIT || ph == PH_RES || ph == PH_CG_B) ? 2
         : (ph == PH_CG_PQ ? 1 : 0);
}
// The tasks of a phase: the inner solve's passes have their own (InstDesc::cgn), all others the
// cell tasks.
__device__ __forceinline__ bool cg_phase(int32_t ph) { return ph == PH_CG_PQ || ph == PH_CG_B; }
__device__ __forceinline__ unsigned phase_ntask(const InstDesc& d, int32_t ph) {
  return (unsigned)(cg_phase(ph) ? d.cgn : d.ntask);
}
__device__ __forceinline__ int64_t phase_task0(const InstDesc& d, int32_t ph) {
  return cg_phase(ph) ? d.cg0 : d.task0;
}


// Scalar epilogue of an instance after a round: its sums update the scalars and name its next phase.
// Out of line: inlined, its scalars took registers from the passes of the solve kernels.
template <typename T>
__device__ __noinline__ void phase_epilogue(InstScal& sc, const InstDesc& d, const DevOpts& o,
                                            const double (&acc)[2]) {
  switch (sc.phase) {
    case PH_RES_INIT:
      epi_residual_s<true>(sc, d, o, acc, sqrt(acc[0] / sc.bb), sqrt(acc[0] / (double)d.n));
      sc.phase = phase_after<T>(sc);
      break;
    case PH_RES:
      epi_residual_s<false>(sc, d, o, acc, sqrt(acc[0] / sc.bb), sqrt(acc[0] / (double)d.n));
      sc.phase = phase_after<T>(sc);
      break;
    case PH_CG_PQ:
      epi_spmv_s(sc, acc);
      sc.phase = sc.inner_active ? PH_CG_B : phase_after<T>(sc);
      break;
    case PH_CG_B:
      epi_upd<T>(sc, o, acc);
      sc.phase = phase_after<T>(sc);
      break;
    case PH_XUPD: sc.phase = PH_RES; break;
    default: sc.phase = PH_IDLE; break;
  }
}

// Task `local` of an instance's current phase.
template <typename T, bool XOUT, bool FULL, bool WEIGHTED>
__device__ __forceinline__ void round_task(const DevArrays& A, const InstDesc& d, double* part, int local,
                                           const InstScal& s, char* dyn) {
  if (s.phase == PH_CG_PQ) pq_task<T>(A, d, d.off4, local, s, part + d.cg0 + local, dyn);
  else if (s.phase == PH_CG_B) upd_form<T, WEIGHTED>(A, d, local, s, part + d.cg0 + local, A.pcap, dyn);
  if constexpr (FULL) {
    const int64_t task = d.task0 + local;
    switch (s.phase) {
      case PH_RES_INIT: res_task<true, T>(A, part, task, s); break;
      case PH_RES: res_task<false, T, XOUT>(A, part, task, s); break;
      case PH_XUPD: xupd_cells<T>(A, task_chunk(A, task), s); break;
      default: break;
    }
  }
}

// The phase as the round log names it.
__device__ __forceinline__ int32_t logged_phase(const InstScal& s) {
  if (s.phase == PH_RES_INIT && s.hx_ok >= 2) return HF_PHASE_RES_INIT_HX;
  if (s.phase == PH_CG_B && (s.xw & kXwThis)) return HF_PHASE_CG_BX;
  return s.phase;
}

// ---- persistent solve of several grids ---------------------------------------------------------
// Tasks come from one queue of tickets (SolveCtl::ticket).  A phase of an instance is a range of
// tickets, published in the instance's slot; the first ntasks tickets are all instances' first
// phase, in task-table order.  A block takes a ticket, finds the instance whose published range
// holds it (its threads look at all slots at once), does that task and counts it in the instance's
// done counter.  The block that finishes an instance's last task of a phase runs its epilogue and
// publishes its next phase at the end of the queue.  So no instance waits for another: with a
// grid-wide barrier after every phase, each round lasted as long as its slowest instance and the
// epilogues of all instances ran in one block while the others waited (64 grids of 16..96 cells an
// edge: 88 us a round for about 40 us of traffic; 20 steps 125 -> 88 ms).
// Tickets are handed out in order and a phase is published only after its predecessor's tickets
// were all done, so every published ticket is held by a block that is running it or will be handed
// out next: a block that waits for its ticket's range to be published never holds up the others.
// An instance's old range stays in its slot until the next replaces it; only blocks that hold one
// of its tickets match it.
// Two blocks per SM, by the passes' shared memory (99 KB each) and registers (114; the whole form, with the
// FP64 sweeps in it, has 128 and spills, in 600 to 820 B of stores).
// XOUT: the instance used by the graphs of host-buffer steps, whose residual sweeps also store x
// into A.xout (a variant of its own, so the other solves carry none of it).
constexpr int kSlotShift = 24;      // slot: first ticket << 24 | tasks << 1 | walk the tasks backwards
template <typename T, bool XOUT, bool FULL, bool WEIGHTED>
__global__ void __launch_bounds__(kBlock, 2)
    k_solve_batch(DevArrays A, SolveCtl* ctl, int64_t limit, unsigned long long wait_ns, int leaver) {
  __shared__ InstScal sh;
  __shared__ double red[kBlock * 2];
  __shared__ unsigned long long s_ticket, s_slot;
  __shared__ int s_inst, s_last, s_stop;
  extern __shared__ __align__(128) char dyn[];
  const int ninst = (int)A.ninst;
  // the first phase's tickets: all instances' cell tasks, or those of the inner solve's passes
  const unsigned long long first = (unsigned long long)(FULL ? A.ntasks : A.ncg);
  unsigned long long* slots = solve_slots(ctl);
  unsigned* done = solve_done(ctl, A.ninst);
  if (FULL && blockIdx.x == 0 && threadIdx.x == 0) A.stamps[kStampSolve] = ctl->t_start = gtimer();
  if (threadIdx.x == 0) s_ticket = atomicAdd(&ctl->ticket, 1ull);
  // failure-path check only (leaver >= 0): that block leaves with a ticket, so its instance never
  // finishes and the others' waits run out and record SolveCtl::err
  if ((int)blockIdx.x == leaver) return;
  for (;;) {
    __syncthreads();
    const unsigned long long t = s_ticket;
    int inst = -1;
    unsigned n = 0, local = 0;
    bool back = false;
    if (t < first) {
      inst = FULL ? A.tasks[t].x : A.cg_inst[t];
      local = (unsigned)(t - (unsigned long long)(FULL ? A.inst[inst].task0 : A.inst[inst].cg0));
      n = (unsigned)(FULL ? A.inst[inst].ntask : A.inst[inst].cgn);
      __syncthreads();                       // every thread has read s_ticket
    } else {
      unsigned long long t0 = 0;
      for (unsigned polls = 0;; ++polls) {
        bool hit = false;
        for (int i = threadIdx.x; i < ninst; i += kBlock) {
          const unsigned long long v = ld_relaxed_u64(slots + i);
          const unsigned long long s0 = v >> kSlotShift;
          if (t >= s0 && t - s0 < ((v >> 1) & ((1ull << (kSlotShift - 1)) - 1ull))) {
            hit = true;
            s_inst = i;
            s_slot = v;
          }
        }
        if (hit) __threadfence();            // what the epilogue before this phase wrote is visible
        if (__syncthreads_or(hit)) break;
        if (threadIdx.x == 0) {
          int stop = *(volatile unsigned*)&ctl->finished >= (unsigned)ninst || *(volatile int*)&ctl->err ||
                     *(volatile int*)&ctl->guard_hit;
          if (!stop && (polls & 63u) == 0u) {
            const unsigned long long now = gtimer();
            if (t0 == 0) t0 = now;
            if (now - t0 > wait_ns || polls > (1u << 26)) {
              atomicExch(&ctl->err, 1);
              stop = 1;
            }
          }
          s_stop = stop;
          if (!stop) __nanosleep(64);
        }
        __syncthreads();
        if (s_stop) return;
      }
      inst = s_inst;
      const unsigned long long v = s_slot;
      n = (unsigned)((v >> 1) & ((1ull << (kSlotShift - 1)) - 1ull));
      local = (unsigned)(t - (v >> kSlotShift));
      back = v & 1ull;
    }
    const InstDesc& d = A.inst[inst];
    if ((int)threadIdx.x < kScalWords)       // this instance's scalars, through L2
      reinterpret_cast<unsigned long long*>(&sh)[threadIdx.x] =
          __ldcg(reinterpret_cast<const unsigned long long*>(A.scal + inst) + threadIdx.x);
    if (threadIdx.x == kBlock - 1) s_ticket = atomicAdd(&ctl->ticket, 1ull);   // the block's next one
    __syncthreads();
    if (!FULL && t < first) {                // the inner solves that are due
      if (threadIdx.x == 0) sh.phase = sh.inner_active ? PH_CG_PQ : PH_IDLE;
      __syncthreads();
    }
    const int32_t ph = sh.phase;             // read before any thread can run the epilogue
    // the two kinds of tasks are numbered apart, and instances in phases of either kind run at once:
    // the inner solve's passes use the second table of partial sums
    double* part = A.partials + (cg_phase(ph) ? kNR * A.pcap : 0);
    round_task<T, XOUT, FULL, WEIGHTED>(A, d, part, (int)(back ? n - 1 - local : local), sh, dyn);
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      s_last = atomicAdd(done + inst, 1u) == n - 1u;
      if (s_last) __threadfence();           // every block's work of this phase is visible now
    }
    __syncthreads();
    if (!s_last) continue;
    double acc[2] = {0.0, 0.0};
    if (phase_partials(ph) > 0) instance_sum<2>(part, A.pcap, phase_task0(d, ph), n, acc, red);
    if (threadIdx.x == 0) {
      if (inst == 0 && ph != PH_IDLE) log_round(ctl, logged_phase(sh), gtimer());
      if (ph != PH_IDLE) phase_epilogue<T>(sh, d, A.opts, acc);
    }
    __syncthreads();
    if ((int)threadIdx.x < kScalWords)
      reinterpret_cast<unsigned long long*>(A.scal + inst)[threadIdx.x] =
          reinterpret_cast<const unsigned long long*>(&sh)[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) {
      done[inst] = 0u;
      __threadfence();
      if (FULL ? sh.phase == PH_IDLE : !cg_phase(sh.phase)) {
        A.stamps[kStampSolveEnd] = gtimer();
        atomicAdd(&ctl->finished, 1u);
      } else if (atomicAdd(&ctl->phases, 1ull) >= (unsigned long long)limit * (unsigned long long)ninst) {
        atomicExch(&ctl->guard_hit, 1);
      } else {
        const unsigned long long m = phase_ntask(d, sh.phase);
        const unsigned long long s0 = first + atomicAdd(&ctl->tail, m);
        st_release_u64(slots + inst, s0 << kSlotShift | m << 1 | (back ? 0ull : 1ull));
      }
    }
  }
}

// ---- persistent solve of one grid ------------------------------------------------------------
// The inner solve that is due, in grid-wide rounds (a pq or an update pass each).  Every block keeps
// the scalars itself: after each round it adds the sums of all tasks (the same adds in the same order,
// so all blocks obtain the same bits) and runs the scalar epilogue on its own copy in shared memory.
// Where the last block to arrive at a barrier does that for all, each round holds six dependent trips
// through L2, which was most of a small grid's round (64^3 slab, mixed, per iteration: 34 us in that
// form and three rounds, 14.3 in two with the epilogue in every block, 11.8 with the epilogue's
// divisions and roots side by side).  No block passes round r before all have arrived at its end, and
// the sums of round r - 1 have then been read by all: two tables, taken in turn.
// Wait until done() (one thread), in bounded time and polls; false: given up, and SolveCtl::err says so.
template <class F>
__device__ __forceinline__ int wait_for(SolveCtl* ctl, unsigned long long wait_ns, F done) {
  unsigned long long t0 = 0;
  for (unsigned polls = 0; !done(); ++polls) {
    if (polls < 64u) continue;               // a round of a small grid is a few microseconds
    if (*(volatile int*)&ctl->err) return 0;
    if ((polls & 255u) == 64u) {
      const unsigned long long now = gtimer();
      if (t0 == 0) t0 = now;
      if (now - t0 > wait_ns || polls > (1u << 27)) {
        atomicExch(&ctl->err, 1);
        return 0;
      }
    }
    __nanosleep(32);
  }
  return 1;
}

// The value up to which the criterion is met (of ||r||_w^2 under the reference's rule, of r.r over the
// solve's first r.r otherwise), or NaN where it was not found; by the first warp.  The criterion, of which
// every rounded operation is monotone, is a root, a product and a division deep, a fifth of a small grid's
// round; an iteration then only compares, with the same outcome.  The lanes try the 32 values around the
// one that exact arithmetic gives.
template <bool WEIGHTED>
__device__ __forceinline__ double stop_limit(const InstScal& s, const DevOpts& o) {
  const double bound = WEIGHTED ? o.tol : s.eta;
  const double root = WEIGHTED ? bound * sqrt(s.bb) / s.sigma_prev : bound;
  const double mid = root * root;
  const bool found = mid > 1e-290 && mid < 1e290 && (WEIGHTED ? s.bb > 0.0 : s.gg0 > 0.0);   // (bb, gg0 > 0)
  const double v = bitsd(dbits(mid) + (unsigned long long)(threadIdx.x & 31) - 16ull);
  const unsigned met = __ballot_sync(kFull, found && upd_err(s, WEIGHTED, v, v) <= bound);
  const int n = __popc(met);                   // the first n lanes, not none of them and not all
  const double lim = __shfl_sync(kFull, v, n > 0 ? n - 1 : 0);
  return n > 0 && n < 32 && met == (1u << n) - 1u ? lim : (double)NAN;
}

// The scalar epilogue of a round, by the first warp: tot[] valid in lane 0.  The two divisions side by
// side in lanes 0 and 1.  lim: stop_limit.
template <typename T, bool WEIGHTED>
__device__ __forceinline__ void round_epilogue(InstScal& sh, const DevOpts& o, int32_t ph, double (&tot)[2], double lim) {
  const int lane = threadIdx.x & 31;
  if (ph == PH_CG_PQ) {
    if (lane == 0) {
      epi_spmv_s(sh, tot);
      if (!sh.inner_active && sh.iter > 0) sh.err = upd_err(sh, WEIGHTED, sh.rr_w, sh.rho / sh.gg0);   // the last update's
      sh.phase = sh.inner_active ? PH_CG_B : phase_after<T>(sh);
    }
    return;
  }
  tot[0] = __shfl_sync(kFull, tot[0], 0);
  UpdRatios q;
  q.shrink = tot[0] / (lane == 0 ? sh.rho : sh.gg0);
  q.first = __shfl_sync(kFull, q.shrink, 1);
  if (lane == 0) {
    const double v = WEIGHTED ? tot[1] : q.first;
    const bool known = !isnan(lim);
    if (!known) sh.err = upd_err(sh, WEIGHTED, tot[1], q.first);
    epi_upd_s<T>(sh, o, tot, q, known ? v >= 0.0 && v <= lim : sh.err <= (WEIGHTED ? o.tol : sh.eta));
    if (known && !sh.inner_active) sh.err = upd_err(sh, WEIGHTED, tot[1], q.first);
    sh.phase = phase_after<T>(sh);
  }
}

// A block's arrival at the end of a round, after its last task's sums (which thread 0 wrote, behind a
// block barrier after all else that the task wrote).
__device__ __forceinline__ void round_arrive(SolveCtl* ctl) {
  if (threadIdx.x == 0) red_release_add_u64(&ctl->arrived, 1ull);
}
// The end of round r, whose sums lie at `sums` (nt first values, then nt second ones): wait for all
// blocks, add the sums, run the round's epilogue on sh.  false: the wait gave up.
template <typename T, bool WEIGHTED>
__device__ __forceinline__ bool round_finish(const DevArrays& A, SolveCtl* ctl, unsigned long long wait_ns, InstScal& sh,
                                             double* red, const double* sums, int nt, int64_t r, int64_t round0,
                                             int32_t ph, int32_t logged, double lim) {
  const int tid = threadIdx.x, G = (int)gridDim.x;
  const bool two = WEIGHTED && ph == PH_CG_B;
  int ok = 1;
  if (tid == 0)
    ok = wait_for(ctl, wait_ns, [&] {
      return ld_acquire_u64(&ctl->arrived) >= (unsigned long long)G * (unsigned long long)(r + 1);
    });
  if (!__syncthreads_and(ok)) return false;
  double a0 = 0.0, a1 = 0.0;
  for (int t = tid; t < nt; t += kBlock) {
    a0 += bitsd(ld_relaxed_u64(reinterpret_cast<const unsigned long long*>(sums + t)));
    if (two) a1 += bitsd(ld_relaxed_u64(reinterpret_cast<const unsigned long long*>(sums + nt + t)));
  }
  red[tid] = a0;
  if (WEIGHTED) red[(WEIGHTED ? 1 : 0) * kBlock + tid] = a1;
  __syncthreads();
  if (tid >= 32) {
    if (tid == 32 && blockIdx.x == 0 && round0 + r < kRoundLog) {   // the log, beside the epilogue
      ctl->phase_log[round0 + r] = logged;
      ctl->t_round[round0 + r] = gtimer();
    }
  } else {
    // the sums in every lane of the first warp: tree8 over the warps, then the lanes (those past
    // the tasks hold zeros)
    double tot[2] = {a0, a1};
    if (nt > 32) {
#pragma unroll
      for (int v = 0; v < (WEIGHTED ? 2 : 1); ++v) {
        double u[8];
#pragma unroll
        for (int w = 0; w < 8; ++w) u[w] = red[v * kBlock + tid + 32 * w];
        tot[v] = tree8(u);
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      if (o >= nt) continue;
      tot[0] += __shfl_xor_sync(kFull, tot[0], o);
      if (two) tot[1] += __shfl_xor_sync(kFull, tot[1], o);
    }
    round_epilogue<T, WEIGHTED>(sh, A.opts, ph, tot, lim);
  }
  __syncthreads();
  return true;
}

// WEIGHTED: the reference's stopping rule (upd_form).
template <typename T, bool WEIGHTED>
__global__ void __launch_bounds__(kBlock, 2)
    k_solve_one(DevArrays A, SolveCtl* ctl, int64_t limit, unsigned long long wait_ns, int leaver) {
  __shared__ InstScal sh;
  __shared__ InstDesc sd;
  __shared__ double red[(WEIGHTED ? 2 : 1) * kBlock];
  extern __shared__ __align__(128) char dyn[];
  static_assert(sizeof(InstDesc) % 8 == 0 && sizeof(InstDesc) / 8 <= kBlock, "descriptor copy");
  const int tid = threadIdx.x, G = (int)gridDim.x;
  if (tid < kScalWords)
    reinterpret_cast<unsigned long long*>(&sh)[tid] = reinterpret_cast<const unsigned long long*>(A.scal)[tid];
  if (tid < (int)(sizeof(InstDesc) / 8))
    reinterpret_cast<unsigned long long*>(&sd)[tid] = reinterpret_cast<const unsigned long long*>(A.inst)[tid];
  __syncthreads();
  if (!sh.inner_active) return;              // no inner solve is due
  const double lim = tid < 32 ? stop_limit<WEIGHTED>(sh, A.opts) : 0.0;
  __syncthreads();
  if (tid == 0) sh.phase = PH_CG_PQ;
  const int nt = sd.cgn;
  double* const sums = reinterpret_cast<double*>(solve_slots(ctl));   // two tables
  const int64_t round0 = ctl->rounds;        // of the log
  __syncthreads();
  int64_t r = 0;
  for (; cg_phase(sh.phase); ++r) {
    if (r >= limit) {
      if (blockIdx.x == 0 && tid == 0) ctl->guard_hit = 1;
      break;
    }
    const int32_t ph = sh.phase;             // read before any thread can run the epilogue
    const int32_t logged = logged_phase(sh);
    double* const mine = sums + (r & 1) * 2 * nt;
    // failure-path check only (leaver >= 0): that block leaves without posting, so the others'
    // waits run out and record SolveCtl::err
    if ((int)blockIdx.x == leaver) return;
    for (int k = blockIdx.x; k < nt; k += G) {
      if (ph == PH_CG_PQ) pq_task<T>(A, sd, 0, k, sh, mine + k, dyn);
      else upd_form<T, WEIGHTED>(A, sd, k, sh, mine + k, nt, dyn);
    }
    round_arrive(ctl);
    if (!round_finish<T, WEIGHTED>(A, ctl, wait_ns, sh, red, mine, nt, r, round0, ph, logged, lim)) return;
  }
  if (blockIdx.x != 0) return;
  if (tid < kScalWords)
    reinterpret_cast<unsigned long long*>(A.scal)[tid] = reinterpret_cast<const unsigned long long*>(&sh)[tid];
  if (tid == 0) {
    ctl->rounds = round0 + r;
    A.stamps[kStampSolveEnd] = gtimer();
  }
}

// ---- persistent solve of one grid that fits on the chip ------------------------------------------
// As k_solve_one, one task per block, with the task's vectors and faces in shared memory for the whole
// inner solve, where the tasks are no more than the blocks that run at once and their planes fit.  Of
// the cells around the task a block also keeps p and r, and updates them as their owner does, so only
// q crosses memory: a round's passes touch no memory before their sum is posted but to store q, and what
// else there is (y, the neighbours' q, the fused x update) is done while the sums travel.  q lies in
// the p buffers by the iteration's parity: a block may still read iteration k's while another stores
// that of k + 1.  A direction enters y in the update that follows it, so y is complete at the end
// (InstScal::ypend = 0).  The arithmetic and its order are those of pq_form and upd_form.
// Bound by the latency of a round (post, poll, the sums' adds and the epilogue's division).  Measured per
// CG iteration, against k_solve_one: the 64^3 slab, mixed, 8.8 us (11.8); 48^3 mixed 7.3 (9.6); 40 FP64
// tiles under the reference's rule 10.4 (13.3).
template <typename T>
struct ResLayout {                             // offsets in 16-byte vectors, for tasks of D planes
  static constexpr int kPlane = kTilePlane, kHalo = kTileHalo;
  int r, q, ax, ay, az, hr, hf, ur, azm, dg, n;
  bool has_dg;
  __host__ __device__ ResLayout(int D, bool weighted) {
    r = (D + 2) * kPlane;                      // p first: the task's planes and the two beside them
    q = r + D * kBlock;
    ax = q + D * kBlock;
    ay = ax + D * kBlock;
    az = ay + D * kBlock;
    hr = az + D * kBlock;                      // r and the faces of the cells beyond the tile (Beyond)
    hf = hr + D * kHalo;
    ur = hf + D * kHalo;                       // r of the planes above and below
    azm = ur + 2 * kBlock;                     // faces to the plane below
    dg = azm + kBlock;                         // diag (the reference's rule), if two blocks still fit
    has_dg = weighted && D <= 2;
    n = dg + (has_dg ? D * kBlock : 0);
  }
};

template <typename T, bool WEIGHTED>
__global__ void __launch_bounds__(kBlock, 2)
    k_solve_res(DevArrays A, SolveCtl* ctl, int64_t limit, unsigned long long wait_ns, int leaver, int depth) {
  constexpr int V = Vec16<T>::N, kPlane = ResLayout<T>::kPlane, kHalo = ResLayout<T>::kHalo;
  typedef Vec16<T> VT;
  __shared__ InstScal sh;
  __shared__ InstDesc sd;
  __shared__ double red[(WEIGHTED ? 2 : 1) * kBlock];
  extern __shared__ __align__(128) char dyn[];
  const int tid = threadIdx.x;
  if (tid < kScalWords)
    reinterpret_cast<unsigned long long*>(&sh)[tid] = reinterpret_cast<const unsigned long long*>(A.scal)[tid];
  if (tid < (int)(sizeof(InstDesc) / 8))
    reinterpret_cast<unsigned long long*>(&sd)[tid] = reinterpret_cast<const unsigned long long*>(A.inst)[tid];
  __syncthreads();
  if (!sh.inner_active) return;                // no inner solve is due
  const double lim = tid < 32 ? stop_limit<WEIGHTED>(sh, A.opts) : 0.0;
  __syncthreads();
  if (tid == 0) sh.phase = PH_CG_PQ;
  const int nt = sd.cgn;
  double* const sums = reinterpret_cast<double*>(solve_slots(ctl));
  const int64_t round0 = ctl->rounds;          // of the log

  const ResLayout<T> lay(depth, WEIGHTED);
  VT* const P = reinterpret_cast<VT*>(dyn);
  const CgPos c = cg_pos<T>(sd, (int)blockIdx.x);
  const Beyond by = beyond_of<T>(sd, c);
  const int nq = sd.cgw, prow = nq + 2, nx = sd.nx, ny = sd.ny, nz = sd.nz, sx = sd.sx, nxy = sx * ny;
  [[maybe_unused]] const int n4 = nxy * nz;
  const int z0 = c.z0, D = c.z1 - c.z0, lxy = c.y * sx + c.x, own = (c.ry + 1) * prow + c.vx + 1;
  const bool act = c.act;
  const int last = min(V - 1, nx - 1 - c.x);
  const bool hsouth = ny > 1 && (c.y > 0 || sd.py), hwest = nx > 1 && (c.x > 0 || sd.px);
  // the planes above and below the task (or their wraps), or -1
  const int zu = nz < 2 ? -1 : c.z1 < nz ? c.z1 : sd.pz ? 0 : -1, zd = nz < 2 ? -1 : z0 > 0 ? z0 - 1 : sd.pz ? nz - 1 : -1;
  const VT zero{};
  // this thread's vectors
  VT* const R = P + lay.r + tid;
  VT* const Qs = P + lay.q + tid;
  VT* const AX = P + lay.ax + tid;
  VT* const AY = P + lay.ay + tid;
  VT* const AZ = P + lay.az + tid;
  VT* const HR = P + lay.hr + tid;             // (threads below kHalo)
  VT* const UR = P + lay.ur + tid;
  auto at = [&](int l, int z) { return HF_IXV(A, l + z * nxy, n4, V); };
  auto diag_of = [&](int k) -> VT {
    VT g = zero;
#pragma unroll
    for (int i = 0; i < V; ++i)
      if (i <= last) g.v[i] = (T)A.diag[HF_IX(A, ((z0 + k) * ny + c.y) * nx + c.x + i, nx * ny * nz)];
    return g;
  };
  for (int i = tid; i < (D + 2) * kPlane; i += kBlock) P[i] = zero;
  for (int k = 0; k < D; ++k) {
    const int l = act ? at(lxy, z0 + k) : 0;
    R[k * kBlock] = act ? ld16(Vec<T>::r(A) + l) : zero;
    AX[k * kBlock] = act ? ld16(Vec<T>::ax(A) + l) : zero;
    AY[k * kBlock] = act ? ld16(Vec<T>::ay(A) + l) : zero;
    AZ[k * kBlock] = act ? ld16(Vec<T>::az(A) + l) : zero;
    Qs[k * kBlock] = zero;
    if (WEIGHTED && lay.has_dg) P[lay.dg + k * kBlock + tid] = act ? diag_of(k) : zero;
    if (by.hl >= 0) {
      VT h = zero, f = zero;
      if (by.hvec) {
        const int lh = at(by.hl, z0 + k);
        h = ld16(Vec<T>::r(A) + lh);
        if (by.hc) f = ld16(Vec<T>::ay(A) + lh);
      } else {
        const int lh = HF_IX(A, by.hl + (z0 + k) * nxy, n4);
        h.v[0] = Vec<T>::r(A)[lh];
        if (by.hc) f.v[0] = Vec<T>::ax(A)[lh];
      }
      HR[k * kHalo] = h;
      P[lay.hf + k * kHalo + tid] = f;
    }
  }
  UR[0] = act && zu >= 0 ? ld16(Vec<T>::r(A) + at(lxy, zu)) : zero;
  UR[kBlock] = act && zd >= 0 ? ld16(Vec<T>::r(A) + at(lxy, zd)) : zero;
  P[lay.azm + tid] = act && zd >= 0 ? ld16(Vec<T>::az(A) + at(lxy, zd)) : zero;
  __syncthreads();

  int64_t r = 0;
  for (; cg_phase(sh.phase); ++r) {
    if (r >= limit) {
      if (blockIdx.x == 0 && tid == 0) ctl->guard_hit = 1;
      break;
    }
    const int32_t ph = sh.phase;               // read before any thread can run the epilogue
    const int32_t logged = logged_phase(sh);
    double* const mine = sums + (r & 1) * 2 * nt;
    if ((int)blockIdx.x == leaver) return;     // failure-path check only (k_solve_one)
    const bool first = sh.iter == 0;
    const T alpha = (T)sh.alpha;
    T* const Q = Vec<T>::pb(A, sh.iter);
    if (ph == PH_CG_PQ) {
      const T beta = (T)sh.beta;
      auto form = [&](VT* p, const VT& rv) {   // p = r + beta p
        VT t = rv;
        if (!first) {
          const VT po = *p;
#pragma unroll
          for (int i = 0; i < V; ++i) t.v[i] = fma(beta, po.v[i], t.v[i]);
        }
        *p = t;
      };
      if (act) {
        for (int k = 0; k < D; ++k) form(P + (k + 1) * kPlane + own, R[k * kBlock]);
        if (zd >= 0) form(P + own, UR[kBlock]);
        if (zu >= 0) form(P + (D + 1) * kPlane + own, UR[0]);
      }
      if (by.hl >= 0) {
        for (int k = 0; k < D; ++k) {
          VT* const p = P + (k + 1) * kPlane + by.hp;
          if (by.hvec) {
            form(p, HR[k * kHalo]);
          } else {
            T& e = p->v[by.hc ? V - 1 : 0];
            const T h = HR[k * kHalo].v[0];
            e = first ? h : fma(beta, e, h);
          }
        }
      }
      __syncthreads();
      T dot = T(0);
      if (act) {
        VT azm = P[lay.azm + tid];
        for (int k = 0; k < D; ++k) {
          const VT *pc = P + (k + 1) * kPlane, *hf = P + lay.hf + k * kHalo;
          const VT axv = AX[k * kBlock], ayv = AY[k * kBlock], azv = AZ[k * kBlock];
          const VT p = pc[own], pn = pc[own + prow], ps = pc[own - prow], pa = pc[own + kPlane], pd = pc[own - kPlane];
          VT ays = zero;
          if (hsouth) ays = c.ry > 0 ? AY[k * kBlock - nq] : hf[nq + c.vx];
          T axw = T(0);
          if (hwest) axw = c.vx > 0 ? AX[k * kBlock - 1].v[V - 1] : hf[2 * nq + c.ry].v[0];
          const T pw = pc[own - 1].v[V - 1], pe = pc[own + 1].v[0];
          VT qv;
#pragma unroll
          for (int i = 0; i < V; ++i) {
            const T pi = p.v[i];
            T acc = pi;
            acc = fma(axv.v[i], i < last ? p.v[i < V - 1 ? i + 1 : i] : pe, acc);
            acc = fma(i > 0 ? axv.v[i > 0 ? i - 1 : 0] : axw, i > 0 ? p.v[i > 0 ? i - 1 : 0] : pw, acc);
            acc = fma(ayv.v[i], pn.v[i], acc);
            acc = fma(ays.v[i], ps.v[i], acc);
            acc = fma(azv.v[i], pa.v[i], acc);
            acc = fma(azm.v[i], pd.v[i], acc);
            if (i > last) acc = T(0);          // padding: q stays 0
            dot = fma(pi, acc, dot);
            qv.v[i] = acc;
          }
          Qs[k * kBlock] = qv;
          st16(Q + at(lxy, z0 + k), qv);
          azm = azv;
        }
      }
      if constexpr (sizeof(T) == 4) {
        task_store_f(mine + blockIdx.x, dot);
      } else {
        const double v[1] = {dot};
        tile_store<1>(mine + blockIdx.x, 0, v);
      }
      round_arrive(ctl);
    } else {
      T rr = T(0);
      double rw = 0.0;
      for (int k = D - 1; k >= 0 && act; --k) {   // (the order of upd_form)
        const VT qv = Qs[k * kBlock];
        VT rv = R[k * kBlock], dg = zero;
        if (WEIGHTED) dg = lay.has_dg ? P[lay.dg + k * kBlock + tid] : diag_of(k);
#pragma unroll
        for (int i = 0; i < V; ++i) {
          T x = fma(-alpha, qv.v[i], rv.v[i]);
          if (i > last) x = T(0);
          rv.v[i] = x;
          rr = fma(x, x, rr);
          if (WEIGHTED && i <= last) rw = fma(-(double)dg.v[i] * (double)x, (double)x, rw);
        }
        R[k * kBlock] = rv;
      }
      if constexpr (sizeof(T) == 4) {
        task_store_f(mine + blockIdx.x, rr);
      } else if constexpr (WEIGHTED) {
        const double v[2] = {rr, rw};
        tile_store<2>(mine + blockIdx.x, nt, v);
      } else {
        const double v[1] = {rr};
        tile_store<1>(mine + blockIdx.x, 0, v);
      }
      round_arrive(ctl);
      // while the sums travel
      auto upd = [&](VT* x, int l) {           // r of the cells beside the task
        const VT q = ld16cg(Q + l);
        VT t = *x;
#pragma unroll
        for (int i = 0; i < V; ++i) t.v[i] = fma(-alpha, q.v[i], t.v[i]);
        *x = t;
      };
      if (act) {
        if (zu >= 0) upd(UR, at(lxy, zu));
        if (zd >= 0) upd(UR + kBlock, at(lxy, zd));
      }
      if (by.hl >= 0) {
        for (int k = 0; k < D; ++k) {
          if (by.hvec) {
            upd(HR + k * kHalo, at(by.hl, z0 + k));
          } else {
            T& e = HR[k * kHalo].v[0];
            e = fma(-alpha, __ldcg(Q + HF_IX(A, by.hl + (z0 + k) * nxy, n4)), e);
          }
        }
      }
      const bool form_x = !WEIGHTED && (sh.xw & kXwThis);   // (never under the reference's rule)
      for (int k = 0; k < D && act; ++k) {
        const int l = at(lxy, z0 + k);
        const VT p = P[(k + 1) * kPlane + own];
        VT y = zero;
        if (!first) y = ld16(Vec<T>::y(A) + l);
#pragma unroll
        for (int i = 0; i < V; ++i) y.v[i] = fma(alpha, p.v[i], y.v[i]);
        st16(Vec<T>::y(A) + l, y);
        if (form_x) {                          // rows of 4k cells: both layouts index alike
          const double* XR = A.tbuf[sh.role[2]];
          double* XW = A.tbuf[sh.role[3]];
          const float sig = (float)sh.sigma_prev;
#pragma unroll
          for (int i = 0; i < V; ++i) {
            if constexpr (sizeof(T) == 8) XW[l + i] = fma(A.sinv[l + i], y.v[i], XR[l + i]);
            else XW[l + i] = XR[l + i] + f32_to_f64(sig * A.sinv32[l + i] * y.v[i]);
          }
        }
      }
    }
    if (!round_finish<T, WEIGHTED>(A, ctl, wait_ns, sh, red, mine, nt, r, round0, ph, logged, lim)) return;
  }
  if (blockIdx.x != 0) return;
  if (tid == 0) sh.ypend = 0;
  __syncthreads();
  if (tid < kScalWords)
    reinterpret_cast<unsigned long long*>(A.scal)[tid] = reinterpret_cast<const unsigned long long*>(&sh)[tid];
  if (tid == 0) {
    ctl->rounds = round0 + r;
    A.stamps[kStampSolveEnd] = gtimer();
  }
}

// ---- persistent solve of one small grid --------------------------------------------------------
// The inner solve of a grid of up to kClusterTasks tasks of one plane each: one thread-block cluster, whose
// blocks keep the vectors and the faces of their tasks (a run of consecutive ones) in shared memory for
// the whole solve.  A neighbour's p and faces are read from the shared memory of the block that owns
// them, each task's sums are written into every block's table, and the cluster barrier (three per
// iteration: p, p.q, r.r) takes the place of the trips through L2, which are most of a small grid's
// rounds in k_solve_one.  The same thread does the same cell's arithmetic as in pq_form and upd_form,
// and the sums are added in the same order: the same bits.  A direction enters y in the update that
// follows it, so y is complete at the end (InstScal::ypend = 0).
// Bound by the FP64 pipe of the SMs it has (1.2 us for 512 cells' products) and by latency.  25 x 25 x 1
// under the reference's rule: 6.9 us per iteration, 8.8 in k_solve_res and 11.7 in k_solve_one.
constexpr int kClusterMax = 16, kClusterSlots = 2, kClusterTasks = kClusterMax * kClusterSlots;
template <typename T, bool WEIGHTED>
struct ClusterSlot {
  Vec16<T> p[kBlock], r[kBlock], q[kBlock], y[kBlock], ax[kBlock], ay[kBlock], az[kBlock];
  Vec16<T> dg[WEIGHTED ? kBlock : 1];
  T red[sizeof(T) == 4 ? kBlock / 32 : (WEIGHTED ? 2 : 1) * kBlock];   // values of the sums (cluster_put)
};

__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of this block's shared object `p` in block `rank` of the cluster.
__device__ __forceinline__ unsigned in_block(const void* p, int rank) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ Vec16<float> ld_cluster(unsigned a, float) {
  Vec16<float> v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.v[0]), "=f"(v.v[1]), "=f"(v.v[2]), "=f"(v.v[3]) : "r"(a));
  return v;
}
__device__ __forceinline__ Vec16<double> ld_cluster(unsigned a, double) {
  Vec16<double> v;
  asm volatile("ld.shared::cluster.v2.f64 {%0,%1}, [%2];" : "=d"(v.v[0]), "=d"(v.v[1]) : "r"(a));
  return v;
}
__device__ __forceinline__ void st_cluster(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// A thread's values of the sums of a slot (FP32: its warp's sum).
template <typename T, int NRV, class S>
__device__ __forceinline__ void cluster_put(S& slot, const T (&v)[NRV]) {
  if constexpr (sizeof(T) == 4) {
    float s = v[0];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    if ((threadIdx.x & 31) == 0) slot.red[threadIdx.x >> 5] = s;
  } else {
#pragma unroll
    for (int k = 0; k < NRV; ++k) slot.red[k * kBlock + threadIdx.x] = v[k];
  }
}
// The slots' sums, in the order of task_store_f (FP32) and tile_store (FP64), into every block's table:
// value k of task t at table[k * kClusterTasks + t].
template <typename T, int NRV, class S>
__device__ __forceinline__ void cluster_post(const S* slot, int slots, int task0, int C, double* table) {
  const int lane = threadIdx.x & 31, j = threadIdx.x >> 5;
  __syncthreads();
  if (j >= slots) return;
  double t[NRV];
  if constexpr (sizeof(T) == 4) {
    float v = lane < kBlock / 32 ? slot[j].red[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    t[0] = (double)v;
  } else {
#pragma unroll
    for (int k = 0; k < NRV; ++k) {
      double u[8];
#pragma unroll
      for (int w = 0; w < 8; ++w) u[w] = slot[j].red[k * kBlock + lane + 32 * w];
      t[k] = tree8(u);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int k = 0; k < NRV; ++k) t[k] += __shfl_xor_sync(kFull, t[k], o);
    }
  }
  if (lane < C) {
#pragma unroll
    for (int k = 0; k < NRV; ++k) st_cluster(in_block(table + k * kClusterTasks + task0 + j, lane), t[k]);
  }
}

template <typename T, bool WEIGHTED>
__global__ void __launch_bounds__(kBlock, 1) k_solve_cluster(DevArrays A, SolveCtl* ctl, int64_t limit) {
  constexpr int V = Vec16<T>::N, NRV = WEIGHTED ? 2 : 1;
  typedef Vec16<T> VT;
  typedef ClusterSlot<T, WEIGHTED> Slot;
  __shared__ InstScal sh;
  __shared__ InstDesc sd;
  __shared__ double table[3 * kClusterTasks];          // p.q; r.r and the weighted r.r
  __shared__ unsigned beside[kClusterSlots][6];          // per slot: the slots e, w, n, s, up, down of it
  __shared__ int4 origin[kClusterSlots];                 // per slot: x, y, z and first cell of its tile
  extern __shared__ __align__(128) char dyn[];
  const int tid = threadIdx.x, C = (int)gridDim.x, rank = (int)blockIdx.x;
  if (tid < kScalWords)
    reinterpret_cast<unsigned long long*>(&sh)[tid] = reinterpret_cast<const unsigned long long*>(A.scal)[tid];
  if (tid < (int)(sizeof(InstDesc) / 8))
    reinterpret_cast<unsigned long long*>(&sd)[tid] = reinterpret_cast<const unsigned long long*>(A.inst)[tid];
  __syncthreads();
  if (!sh.inner_active) return;                         // no inner solve is due (in any block)
  const double lim = tid < 32 ? stop_limit<WEIGHTED>(sh, A.opts) : 0.0;
  Slot* slot = reinterpret_cast<Slot*>(dyn);
  const int nt = sd.cgn, nxy_t = sd.cgnx * sd.cgny, task0 = rank * nt / C, slots = (rank + 1) * nt / C - task0;
  const int nx = sd.nx, ny = sd.ny, nz = sd.nz, sx = sd.sx, nxy = sx * ny, nq = sd.cgw, rows = sd.cgr;
  [[maybe_unused]] const int n4 = nxy * nz;
  const int ry = tid / nq, vx = tid - ry * nq, lt = ry * sx + vx * V;
  const VT zero{};
  if (tid < slots) {
    const int t = task0 + tid, x = t % sd.cgnx * nq * V, y = t / sd.cgnx % sd.cgny * rows, z = t / nxy_t;
    origin[tid] = make_int4(x, y, z, z * nxy + y * sx + x);
  }
  if (tid >= 32 && tid - 32 < slots * 6) {
    const int j = (tid - 32) / 6, dir = (tid - 32) % 6, t = task0 + j;
    const int bx = t % sd.cgnx, by = t / sd.cgnx % sd.cgny, bz = t / nxy_t;
    int o;                                              // the task beside it (across a wrap, too)
    if (dir == 0) o = bx + 1 < sd.cgnx ? t + 1 : t - bx;
    else if (dir == 1) o = bx > 0 ? t - 1 : t + sd.cgnx - 1;
    else if (dir == 2) o = by + 1 < sd.cgny ? t + sd.cgnx : t - by * sd.cgnx;
    else if (dir == 3) o = by > 0 ? t - sd.cgnx : t + (sd.cgny - 1) * sd.cgnx;
    else if (dir == 4) o = bz + 1 < nz ? t + nxy_t : t - bz * nxy_t;
    else o = bz > 0 ? t - nxy_t : t + (nz - 1) * nxy_t;
    const int owner = ((o + 1) * C - 1) / nt;           // the block whose run of tasks holds it
    beside[j][dir] = in_block(slot + (o - owner * nt / C), owner);
  }
  for (int i = tid; i < 3 * kClusterTasks; i += kBlock) table[i] = 0.0;
  __syncthreads();
  auto active = [&](const int4& o) { return o.x + vx * V < nx && o.y + ry < ny && ry < rows; };
  for (int j = 0; j < slots; ++j) {
    const int4 o = origin[j];
    Slot& s = slot[j];
    const bool act = active(o);
    const int l = act ? HF_IXV(A, o.w + lt, n4, V) : 0;
    s.r[tid] = act ? ld16(Vec<T>::r(A) + l) : zero;
    s.ax[tid] = act ? ld16(Vec<T>::ax(A) + l) : zero;
    s.ay[tid] = act ? ld16(Vec<T>::ay(A) + l) : zero;
    s.az[tid] = act ? ld16(Vec<T>::az(A) + l) : zero;
    s.p[tid] = s.q[tid] = s.y[tid] = zero;
    if constexpr (WEIGHTED) {
      VT dg{};
      for (int i = 0; i < V; ++i)
        if (act && o.x + vx * V + i < nx)
          dg.v[i] = A.diag[HF_IX(A, (o.z * ny + o.y + ry) * nx + o.x + vx * V + i, nx * ny * nz)];
      s.dg[tid] = dg;
    }
  }
  if (tid == 0) sh.phase = PH_CG_PQ;
  const int64_t round0 = ctl->rounds;
  cluster_sync();                                       // every block's state is in place
  int64_t r = 0;
  for (; cg_phase(sh.phase); ++r) {
    if (r >= limit) {                                   // (the same in every block)
      if (rank == 0 && tid == 0) ctl->guard_hit = 1;
      break;
    }
    const int32_t ph = sh.phase, logged = logged_phase(sh);
    const T alpha = (T)sh.alpha;
    const bool first = sh.iter == 0;
    if (ph == PH_CG_PQ) {
      const T beta = (T)sh.beta;
      for (int j = 0; j < slots; ++j) {
        VT p = slot[j].r[tid];
        if (!first) {
          const VT po = slot[j].p[tid];
#pragma unroll
          for (int i = 0; i < V; ++i) p.v[i] = fma(beta, po.v[i], p.v[i]);
        }
        slot[j].p[tid] = p;
      }
      cluster_sync();                                   // p of every block is there
      for (int j = 0; j < slots; ++j) {
        Slot& s = slot[j];
        const int4 o = origin[j];
        T dot = T(0);
        if (active(o)) {
          constexpr unsigned kAx = offsetof(Slot, ax), kAy = offsetof(Slot, ay), kAz = offsetof(Slot, az);
          const int x = o.x + vx * V, y = o.y + ry, z = o.z;
          const int last = min(V - 1, nx - 1 - x);
          VT pn = zero, ps = zero, ays = zero, pa = zero, pd = zero, azm = zero;
          T pe = T(0), pw = T(0), axw = T(0);
          if (nz > 1) {
            if (z + 1 < nz || sd.pz) pa = ld_cluster(beside[j][4] + tid * 16, T(0));
            if (z > 0 || sd.pz) {
              pd = ld_cluster(beside[j][5] + tid * 16, T(0));
              azm = ld_cluster(beside[j][5] + kAz + tid * 16, T(0));
            }
          }
          if (ny > 1) {
            if (y + 1 < ny && ry < rows - 1) pn = s.p[tid + nq];
            else if (y + 1 < ny || sd.py) pn = ld_cluster(beside[j][2] + vx * 16, T(0));
            if (ry > 0) {
              ps = s.p[tid - nq];
              ays = s.ay[tid - nq];
            } else if (y > 0 || sd.py) {
              const int row = y > 0 ? rows - 1 : (ny - 1) % rows;
              const unsigned a = beside[j][3] + (row * nq + vx) * 16;
              ps = ld_cluster(a, T(0));
              ays = ld_cluster(a + kAy, T(0));
            }
          }
          if (x + V < nx && vx < nq - 1) pe = s.p[tid + 1].v[0];
          else if (x + V < nx || (sd.px && nx > 1)) pe = ld_cluster(beside[j][0] + (tid - vx) * 16, T(0)).v[0];
          if (vx > 0) {
            pw = s.p[tid - 1].v[V - 1];
            axw = s.ax[tid - 1].v[V - 1];
          } else if (x > 0 || (sd.px && nx > 1)) {      // the last cell of the tile, or of the row
            const int e = x > 0 ? nq * V - 1 : (nx - 1) % (nq * V);
            const unsigned a = beside[j][1] + (tid + e / V) * 16;
            const VT w = ld_cluster(a, T(0)), f = ld_cluster(a + kAx, T(0));
#pragma unroll
            for (int i = 0; i < V; ++i) {
              if (i == e % V) {
                pw = w.v[i];
                axw = f.v[i];
              }
            }
          }
          const VT p = s.p[tid], axv = s.ax[tid], ayv = s.ay[tid], azv = s.az[tid];
          VT qv;
#pragma unroll
          for (int i = 0; i < V; ++i) {
            const T pi = p.v[i];
            T acc = pi;
            acc = fma(axv.v[i], i < last ? p.v[i < V - 1 ? i + 1 : i] : pe, acc);
            acc = fma(i > 0 ? axv.v[i > 0 ? i - 1 : 0] : axw, i > 0 ? p.v[i > 0 ? i - 1 : 0] : pw, acc);
            acc = fma(ayv.v[i], pn.v[i], acc);
            acc = fma(ays.v[i], ps.v[i], acc);
            acc = fma(azv.v[i], pa.v[i], acc);
            acc = fma(azm.v[i], pd.v[i], acc);
            if (i > last) acc = T(0);
            dot = fma(pi, acc, dot);
            qv.v[i] = acc;
          }
          s.q[tid] = qv;
        }
        const T v[1] = {dot};
        cluster_put<T, 1>(s, v);
      }
      cluster_post<T, 1>(slot, slots, task0, C, table);
    } else {
      const bool form_x = !WEIGHTED && (sh.xw & kXwThis);
      for (int j = 0; j < slots; ++j) {
        Slot& s = slot[j];
        const int4 o = origin[j];
        T rr = T(0), rw = T(0);
        if (active(o)) {
          const int last = min(V - 1, nx - 1 - (o.x + vx * V)), l = HF_IXV(A, o.w + lt, n4, V);
          VT y = s.y[tid], rv = s.r[tid];
          const VT q = s.q[tid], p = s.p[tid];
          VT dg{};
          if constexpr (WEIGHTED) dg = s.dg[tid];
#pragma unroll
          for (int i = 0; i < V; ++i) {
            T x = fma(-alpha, q.v[i], rv.v[i]);
            if (i > last) x = T(0);
            rv.v[i] = x;
            rr = fma(x, x, rr);
            if (WEIGHTED && i <= last) rw = fma(-dg.v[i] * x, x, rw);
            y.v[i] = fma(alpha, p.v[i], y.v[i]);
          }
          s.r[tid] = rv;
          s.y[tid] = y;
          if (form_x) {                                 // rows of 4k cells: both layouts index alike
            const double* XR = A.tbuf[sh.role[2]];
            double* XW = A.tbuf[sh.role[3]];
            const float sig = (float)sh.sigma_prev;
#pragma unroll
            for (int i = 0; i < V; ++i) {
              if constexpr (sizeof(T) == 8) XW[l + i] = fma(A.sinv[l + i], y.v[i], XR[l + i]);
              else XW[l + i] = XR[l + i] + f32_to_f64(sig * A.sinv32[l + i] * y.v[i]);
            }
          }
        }
        if constexpr (WEIGHTED) {
          const T v[2] = {rr, rw};
          cluster_put<T, 2>(s, v);
        } else {
          const T v[1] = {rr};
          cluster_put<T, 1>(s, v);
        }
      }
      cluster_post<T, NRV>(slot, slots, task0, C, table + kClusterTasks);
    }
    cluster_sync();                                     // the sums of every block are there
    if (tid < 32) {
      // one task a lane: the order of instance_sum
      double tot[2] = {0.0, 0.0};
      const double* p = table + (ph == PH_CG_PQ ? 0 : kClusterTasks);
      if (tid < nt) {
        tot[0] = 0.0 + p[tid];
        if (WEIGHTED && ph == PH_CG_B) tot[1] = 0.0 + p[kClusterTasks + tid];
      }
      for (int o = 16; o > 0; o >>= 1) {
        if (o >= nt) continue;                          // (lanes past the tasks hold zeros)
        tot[0] += __shfl_xor_sync(kFull, tot[0], o);
        if (WEIGHTED) tot[1] += __shfl_xor_sync(kFull, tot[1], o);
      }
      round_epilogue<T, WEIGHTED>(sh, A.opts, ph, tot, lim);
    } else if (tid == 32 && rank == 0 && round0 + r < kRoundLog) {
      ctl->phase_log[round0 + r] = logged;
      ctl->t_round[round0 + r] = gtimer();
    }
    __syncthreads();
  }
  if (sh.iter > 0) {
    for (int j = 0; j < slots; ++j) {
      const int4 o = origin[j];
      if (active(o)) {
        const int l = HF_IXV(A, o.w + lt, n4, V);
        st16(Vec<T>::y(A) + l, slot[j].y[tid]);
      }
    }
  }
  cluster_sync();                                       // no block leaves while its memory may be read
  if (rank != 0) return;
  if (tid == 0) sh.ypend = 0;
  __syncthreads();
  if (tid < kScalWords)
    reinterpret_cast<unsigned long long*>(A.scal)[tid] = reinterpret_cast<const unsigned long long*>(&sh)[tid];
  if (tid == 0) {
    ctl->rounds = round0 + r;
    A.stamps[kStampSolveEnd] = gtimer();
  }
}

typedef void (*SolveKernel)(DevArrays, SolveCtl*, int64_t, unsigned long long, int);
template <typename T, bool FULL, bool WEIGHTED>
static SolveKernel solve_kernel_of(const Ctx& c, bool xout) {
  if (c.ninst == 1) return k_solve_one<T, WEIGHTED>;
  return FULL && xout ? k_solve_batch<T, FULL, FULL, WEIGHTED> : k_solve_batch<T, false, FULL, WEIGHTED>;
}
static SolveKernel solve_kernel(const Ctx& c, int fp32, bool xout, bool full) {
  if (fp32) return full ? solve_kernel_of<float, true, false>(c, xout) : solve_kernel_of<float, false, false>(c, xout);
  if (c.opts.criterion == HF_STOP_RECURSIVE)
    return full ? solve_kernel_of<double, true, true>(c, xout) : solve_kernel_of<double, false, true>(c, xout);
  return full ? solve_kernel_of<double, true, false>(c, xout) : solve_kernel_of<double, false, false>(c, xout);
}

template <typename K>
static cudaError_t allow_smem(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// Largest co-resident grid of the persistent solve (cooperative launch bound), capped by tasks.
int solve_grid_blocks(Ctx& c, int fp32, bool full) {
  int& cached = c.solve_blocks[full ? 1 : 0][fp32 ? 1 : 0];
  if (cached > 0) return cached;
  int per_sm = INT_MAX, nsm = 0;
  const int smem = fp32 ? kPqSmem<float> : kPqSmem<double>;
  for (bool x : {false, true}) {               // one grid size for both variants
    int n = 0;
    if (allow_smem(solve_kernel(c, fp32, x, full), smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, solve_kernel(c, fp32, x, full), kBlock, smem) != cudaSuccess)
      return -1;
    per_sm = std::min(per_sm, n);
  }
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device) != cudaSuccess) return -1;
  // every SM holds the same number of blocks; tasks are handed out one at a time, so the blocks
  // of busier SMs take fewer of them
  int64_t g = (int64_t)per_sm * nsm;
  g = std::min(g, full && c.ninst > 1 ? std::max(c.ntasks, c.ncg) : c.ncg);
  if (g < 1) return -1;
  cached = (int)g;
  return cached;
}

// k_solve_cluster's launch: C blocks, one cluster.
template <typename T, bool WEIGHTED>
static cudaError_t cluster_config(Ctx& c, int C, cudaLaunchConfig_t& cfg, cudaLaunchAttribute& at) {
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)C;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg = {};
  cfg.gridDim = dim3((unsigned)C);
  cfg.blockDim = dim3(kBlock);
  cfg.dynamicSmemBytes = kClusterSlots * sizeof(ClusterSlot<T, WEIGHTED>);
  cfg.stream = c.stream;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  auto kernel = k_solve_cluster<T, WEIGHTED>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e == cudaSuccess ? allow_smem(kernel, (int)cfg.dynamicSmemBytes) : e;
}
// Blocks of the cluster that runs a grid's inner solves, or 0.
template <typename T, bool WEIGHTED>
static int cluster_blocks_of(Ctx& c) {
  const InstDesc& d = c.h_inst[0];
  if (d.cgnz != d.nz || d.cgn > (sizeof(T) == 8 ? kClusterMax : kClusterTasks)) return 0;
  const int C = std::min(kClusterMax, d.cgn);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  int n = 0;
  if (cluster_config<T, WEIGHTED>(c, C, cfg, at) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, k_solve_cluster<T, WEIGHTED>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n >= 1 ? C : 0;
}
template <typename T, bool WEIGHTED>
static cudaError_t launch_cluster(Ctx& c, int64_t limit) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  const cudaError_t e = cluster_config<T, WEIGHTED>(c, c.cluster_blocks, cfg, at);
  return e == cudaSuccess ? cudaLaunchKernelEx(&cfg, k_solve_cluster<T, WEIGHTED>, c.A, c.d_sctl, limit) : e;
}

// The dynamic shared memory a block of `kernel` may have beside its static one, which becomes its limit;
// or 0.  The limit belongs to the process: with one value for every context, no thread lowers it between
// another's occupancy query or launch and its own.
template <typename K>
static int most_smem(const Ctx& c, K kernel) {
  int most = 0;
  cudaFuncAttributes fa;
  if (cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device) == cudaSuccess &&
      cudaFuncGetAttributes(&fa, kernel) == cudaSuccess) {
    most -= (int)fa.sharedSizeBytes;
    if (allow_smem(kernel, most) == cudaSuccess) return most;
  }
  cudaGetLastError();                          // a refusal is an answer: no later launch reports it
  return 0;
}

// Planes of the deepest task where k_solve_res serves the inner solves of a grid, or 0: all of its
// blocks run at once with the task's state in shared memory.
template <typename T, bool WEIGHTED>
static int res_depth_of(Ctx& c) {
  const InstDesc& d = c.h_inst[0];
  const int D = (d.nz + d.cgnz - 1) / d.cgnz, smem = ResLayout<T>(D, WEIGHTED).n * 16;
  auto kernel = k_solve_res<T, WEIGHTED>;
  int n = 0, nsm = 0;
  if (smem > most_smem(c, kernel)) return 0;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kBlock, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return (int64_t)n * nsm >= d.cgn ? D : 0;
}
// Which kernel runs the inner solves of one grid: k_solve_cluster, k_solve_res or k_solve_one, each where
// the one before does not take the grid.  The cluster has 16 SMs, and its latency advantage is spent when
// each has more than one FP64 task (its pipe's work) or two FP32 ones; us per iteration, cluster against
// k_solve_res: FP64 under the reference's rule, 8 tasks 7.3 and 9.5, 16 tasks 7.7 and 9.5, 32 tasks 9.8
// and 9.4; FP32, 16 tasks 4.6 and 6.3, 32 tasks 5.5 and 6.3, 48 (three a block) 7.8 and 6.7.
template <typename T, bool WEIGHTED>
static void choose_of(Ctx& c) {
  c.cluster_blocks = c.inner_from <= HF_INNER_CLUSTER ? cluster_blocks_of<T, WEIGHTED>(c) : 0;
  c.res_depth = c.inner_from <= HF_INNER_RESIDENT ? res_depth_of<T, WEIGHTED>(c) : 0;
}
static void choose_solve(Ctx& c) {
  if (c.res_depth >= 0) return;
  if (c.opts.precision == HF_PREC_MIXED) choose_of<float, false>(c);
  else if (c.opts.criterion == HF_STOP_RECURSIVE) choose_of<double, true>(c);
  else choose_of<double, false>(c);
}
int inner_kernel(Ctx& c) {
  if (c.opts.use_graph == 0 && c.inner_from == HF_INNER_LAUNCHES) return HF_INNER_LAUNCHES;
  if (c.ninst > 1) return HF_INNER_GENERAL;
  choose_solve(c);
  return c.cluster_blocks > 0 ? HF_INNER_CLUSTER : c.res_depth > 0 ? HF_INNER_RESIDENT : HF_INNER_GENERAL;
}

// Zero the control block (its counters: full = false), then launch the persistent solve cooperatively
// on the context stream.
cudaError_t launch_solve(Ctx& c, bool full, unsigned long long wait_ns, int leaver) {
  const bool fp32 = c.opts.precision == HF_PREC_MIXED;
  const int g = solve_grid_blocks(c, fp32 ? 1 : 0, full);
  if (g < 1) return cudaErrorInvalidConfiguration;
  const size_t skip = full ? 0 : offsetof(SolveCtl, arrived);
  cudaError_t e = cudaSuccess;
  if (full || c.ninst > 1 || leaver >= 0) {    // (one grid's counter: k_finalize)
    e = cudaMemsetAsync(reinterpret_cast<char*>(c.d_sctl) + skip, 0, solve_ctl_bytes(c.ninst, c.ncg) - skip, c.stream);
    if (e != cudaSuccess) return e;
  }
  const int64_t per = fp32 ? c.opts.inner_itmax : c.opts.itmax;
  const int64_t limit = (int64_t)(c.opts.max_refine + 3) * (2 * per + 6) + 8;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)g);
  cfg.blockDim = dim3(kBlock);
  cfg.dynamicSmemBytes = fp32 ? kPqSmem<float> : kPqSmem<double>;
  cfg.stream = c.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const bool weighted = !fp32 && c.opts.criterion == HF_STOP_RECURSIVE;
  if (c.ninst == 1) {
    choose_solve(c);
    if (c.cluster_blocks > 0 && leaver < 0)    // (the failure-path check is of the waits of the others)
      return fp32 ? launch_cluster<float, false>(c, limit)
                  : weighted ? launch_cluster<double, true>(c, limit) : launch_cluster<double, false>(c, limit);
    if (const int D = c.res_depth) {
      auto kernel = fp32 ? k_solve_res<float, false> : weighted ? k_solve_res<double, true> : k_solve_res<double, false>;
      cfg.gridDim = dim3((unsigned)c.h_inst[0].cgn);
      cfg.dynamicSmemBytes = (size_t)16 * (fp32 ? ResLayout<float>(D, false).n : ResLayout<double>(D, weighted).n);
      return cudaLaunchKernelEx(&cfg, kernel, c.A, c.d_sctl, limit, wait_ns, leaver, D);
    }
  }
  e = allow_smem(solve_kernel(c, fp32 ? 1 : 0, c.A.xout != nullptr, full), (int)cfg.dynamicSmemBytes);
  if (e != cudaSuccess) return e;
  return cudaLaunchKernelEx(&cfg, solve_kernel(c, fp32 ? 1 : 0, c.A.xout != nullptr, full), c.A, c.d_sctl, limit,
                            wait_ns, leaver);
}

#ifdef HF_CHECKED
// One failed check and no memory access (the index is only compared with its range), so a test
// can see a failed check recorded and reported.
__global__ void k_check_probe(DevArrays A) { (void)HF_IX(A, -1, 1); }
cudaError_t launch_check_probe(Ctx& c) {
  k_check_probe<<<1, 1, 0, c.stream>>>(c.A);
  return cudaGetLastError();
}
#endif

// ---- launchers ---------------------------------------------------------------------------------
cudaError_t launch_step_begin(Ctx& c, int64_t itime, int) {
  k_step_begin<<<(unsigned)((c.ninst + 127) / 128), 128, 0, c.stream>>>(c.A, itime);
  return cudaGetLastError();
}

cudaError_t launch_step_end(Ctx& c) {
  k_step_end<<<(unsigned)((c.ninst + 127) / 128), 128, 0, c.stream>>>(c.A);
  return cudaGetLastError();
}

// mode 0: initial residual (+ finalize); mode 1: solution update + residual (+ finalize)
template <typename T>
static void launch_res(Ctx& c, int mode, int log) {
  const unsigned nb = (unsigned)c.ntasks;
  if (mode == 0) {
    k_residual<true, T><<<nb, kBlock, 0, c.stream>>>(c.A, log);
    return;
  }
  k_xupdate<T><<<nb * kFine, kBlock, 0, c.stream>>>(c.A);
  if (c.A.xout) k_residual<false, T, true><<<nb, kBlock, 0, c.stream>>>(c.A, log);
  else k_residual<false, T><<<nb, kBlock, 0, c.stream>>>(c.A, log);
}
cudaError_t launch_residual(Ctx& c, int mode, CtrlState* ctrl, cudaGraphConditionalHandle hw,
                            int graph) {
  if (c.opts.precision == HF_PREC_MIXED) launch_res<float>(c, mode, graph);
  else launch_res<double>(c, mode, graph);
  return launch_finalize(c, mode == 0 ? FIN_RES_INIT : FIN_RES, ctrl, hw, graph);
}

template <typename T>
static cudaError_t launch_cg_pq(Ctx& c) {
  const cudaError_t e = allow_smem(k_cg_pq<T>, kPqSmem<T>);
  if (e != cudaSuccess) return e;
  k_cg_pq<T><<<(unsigned)c.ncg, kBlock, kPqSmem<T>, c.stream>>>(c.A);
  return cudaGetLastError();
}

template <typename T>
static cudaError_t launch_cg_upd(Ctx& c) {
  const cudaError_t e = allow_smem(k_cg_upd<T>, kPqSmem<T>);
  if (e != cudaSuccess) return e;
  k_cg_upd<T><<<(unsigned)c.ncg, kBlock, kPqSmem<T>, c.stream>>>(c.A);
  return cudaGetLastError();
}

cudaError_t launch_inner_iteration(Ctx& c) {
  const bool fp32 = c.opts.precision == HF_PREC_MIXED;
  cudaError_t e = fp32 ? launch_cg_pq<float>(c) : launch_cg_pq<double>(c);
  if (e == cudaSuccess) e = launch_finalize(c, FIN_PQ, nullptr, 0, 0);
  if (e == cudaSuccess) e = fp32 ? launch_cg_upd<float>(c) : launch_cg_upd<double>(c);
  return e == cudaSuccess ? launch_finalize(c, FIN_UPD, nullptr, 0, 0) : e;
}

cudaError_t launch_graph_step_begin(Ctx& c, CtrlState* ctrl, int launches_per_step) {
  k_graph_step_begin<<<(unsigned)((c.ninst + 127) / 128), 128, 0, c.stream>>>(c.A, ctrl,
                                                                               launches_per_step);
  return cudaGetLastError();
}
cudaError_t launch_graph_step_end(Ctx& c, CtrlState* ctrl, const SolveCtl* sctl,
                                  cudaGraphConditionalHandle hloop, int loop) {
  k_graph_step_end<<<1, 256, 0, c.stream>>>(c.A, ctrl, sctl, hloop, loop);
  return cudaGetLastError();
}
cudaError_t launch_finalize(Ctx& c, int kind, CtrlState* ctrl, cudaGraphConditionalHandle hw,
                            int graph) {
  const unsigned nb = (unsigned)c.ninst;
  switch (kind) {
    case FIN_RHS: k_finalize<FIN_RHS><<<nb, 256, 0, c.stream>>>(c.A, ctrl, hw, graph); break;
    case FIN_RHS_DIAG: k_finalize<FIN_RHS_DIAG><<<nb, 256, 0, c.stream>>>(c.A, ctrl, hw, graph); break;
    case FIN_RES_INIT: k_finalize<FIN_RES_INIT><<<nb, 256, 0, c.stream>>>(c.A, ctrl, hw, graph); break;
    case FIN_RES: k_finalize<FIN_RES><<<nb, 256, 0, c.stream>>>(c.A, ctrl, hw, graph); break;
    case FIN_PQ: k_finalize<FIN_PQ><<<nb, 256, 0, c.stream>>>(c.A, ctrl, hw, graph); break;
    case FIN_UPD: k_finalize<FIN_UPD><<<nb, 256, 0, c.stream>>>(c.A, ctrl, hw, graph); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// One kernel of the step, for timing (hf_time_kernel).
cudaError_t launch_single(Ctx& c, int which) {
  const unsigned nb = (unsigned)c.ntasks;
  const bool fp32 = c.opts.precision == HF_PREC_MIXED;
  switch (which) {
    case HF_KERNEL_RHS: return launch_rhs(c);
    case HF_KERNEL_RESIDUAL:
      if (fp32) k_residual<false, float><<<nb, kBlock, 0, c.stream>>>(c.A, 0);
      else k_residual<false, double><<<nb, kBlock, 0, c.stream>>>(c.A, 0);
      break;
    case HF_KERNEL_RESIDUAL_INIT:
      if (fp32) k_residual<true, float><<<nb, kBlock, 0, c.stream>>>(c.A, 0);
      else k_residual<true, double><<<nb, kBlock, 0, c.stream>>>(c.A, 0);
      break;
    case HF_KERNEL_XUPDATE:
      if (fp32) k_xupdate<float><<<nb * kFine, kBlock, 0, c.stream>>>(c.A);
      else k_xupdate<double><<<nb * kFine, kBlock, 0, c.stream>>>(c.A);
      break;
    // the direction update and the SpMV are one pass
    case HF_KERNEL_CG_P:
    case HF_KERNEL_CG_SPMV:
    case HF_KERNEL_CG_PQ: return fp32 ? launch_cg_pq<float>(c) : launch_cg_pq<double>(c);
    case HF_KERNEL_CG_UPDATE: return fp32 ? launch_cg_upd<float>(c) : launch_cg_upd<double>(c);
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace hf
