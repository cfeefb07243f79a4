// Assembled FP64 path: 3x3 block sliced-ELL (SELL-32) stiffness built on the
// device from element matrices, its SpMV, and a Jacobi-PCG whose whole loop
// runs on the device.
//
// Replaces the skyline assembler (GlobalMatrixAssemblerSkyline.cs:51-103), the
// skyline product (SkylineMatrix2D.Multiply :224-286) and the PCG loop of
// SolverPCG.Solve (PCG/SolverPCG.cs:105-149) with the simple search vector
// (SolverPCGSimpleSearchVectorCalculator.cs:18-41) and the diagonal
// preconditioner z_j = r_j / K_jj (PolynomialChaosSolverPCGMatrixCalculator.cs:467-495).
//
// Layout: block row = mesh node; vectors in node layout v[3*node + comp]
// (constrained components hold 0 and their matrix rows/columns are identity).
// SELL values: val[((slot)*9 + k)*32 + lane], k = 3*row_comp + col_comp, so a
// warp reads each of the 9 block entries of 32 consecutive rows as one 256-byte
// coalesced load; the matrix stream is the whole HBM traffic of the product.
#include <algorithm>

#include <cstddef>
#include <cstring>

#include "msg_internal.h"

namespace msg {
namespace {


// One thread per (flat position, block entry k): sum the element
// contributions (e, a, b) of this block in their fixed order, then apply the
// Dirichlet mask (identity on constrained rows/columns).
__global__ void k_bsr_assemble(int64_t n_pos, const int* __restrict__ /*col*/, const int64_t* __restrict__ cptr,
                               const int* __restrict__ contrib, const double* __restrict__ Ke,
                               double* __restrict__ val) {
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (tid >= n_pos * 9) return;
  const int64_t pos = tid / 9;
  const int k = (int)(tid - pos * 9);
  const int64_t slot = pos >> 5;
  const int lane = (int)(pos & 31);
  const int cr = k / 3, cc = k - 3 * cr;
  double acc = 0.0;
  for (int64_t q = cptr[pos]; q < cptr[pos + 1]; ++q) {
    const int code = contrib[q];
    const int e = code >> 6, a = (code >> 3) & 7, b = code & 7;
    acc += Ke[(size_t)e * 300 + packed_index(3 * a + cr, 3 * b + cc)];
  }
  val[(slot * 9 + k) * 32 + lane] = acc;
}

// Dirichlet masking pass: row node = slice*32 + lane, column node = col[pos].
__global__ void k_bsr_mask(int n_rows, const int64_t* __restrict__ slice_ptr, const int* __restrict__ col,
                           const uint8_t* __restrict__ mask, double* __restrict__ val) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= n_rows) return;
  const int slice = row >> 5, lane = row & 31;
  const int64_t s0 = slice_ptr[slice], s1 = slice_ptr[slice + 1];
  const uint8_t mr = mask[row];
  for (int64_t s = s0; s < s1; ++s) {
    const int c = col[s * 32 + lane];
    if (c < 0) break;
    const uint8_t mc = mask[c];
    if ((mr | mc) == 0) continue;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int cr = k / 3, cc = k % 3;
      if (((mr >> cr) & 1) || ((mc >> cc) & 1)) val[(s * 9 + k) * 32 + lane] = (c == row && cr == cc) ? 1.0 : 0.0;
    }
  }
}

__global__ void k_bsr_diag_inv(int n_rows, const int* __restrict__ diag_pos, const double* __restrict__ val,
                               double* __restrict__ dinv) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= n_rows) return;
  const int64_t pos = diag_pos[row];
  const int64_t slot = pos >> 5;
  const int lane = (int)(pos & 31);
#pragma unroll
  for (int c = 0; c < 3; ++c) dinv[3 * row + c] = 1.0 / val[(slot * 9 + 4 * c) * 32 + lane];
}

// One warp per (32-row slice, output component): 3x the threads of a
// row-per-thread product, each warp still reading its 3 block entries per
// slot as coalesced 256-byte lines.
__device__ __forceinline__ double sell_row_comp(int slice, int lane, int c, const int64_t* __restrict__ slice_ptr,
                                                const int* __restrict__ col, const double* __restrict__ val,
                                                const double* __restrict__ x) {
  const int64_t s0 = slice_ptr[slice], s1 = slice_ptr[slice + 1];
  double acc = 0;
  for (int64_t s = s0; s < s1; ++s) {
    const int cc = __ldg(col + s * 32 + lane);
    if (cc < 0) break;
    const double* v = val + (s * 9 + 3 * c) * 32 + lane;
    acc += __ldg(v) * __ldg(x + 3 * cc) + __ldg(v + 32) * __ldg(x + 3 * cc + 1) + __ldg(v + 64) * __ldg(x + 3 * cc + 2);
  }
  return acc;
}

__global__ void __launch_bounds__(96) k_bsr_spmv3(int n_rows, const int64_t* __restrict__ slice_ptr,
                                                  const int* __restrict__ col, const double* __restrict__ val,
                                                  const double* __restrict__ x, double* __restrict__ y) {
  const int slice = blockIdx.x, c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = slice * 32 + lane;
  if (row >= n_rows) return;
  y[3 * row + c] = sell_row_comp(slice, lane, c, slice_ptr, col, val, x);
}

__global__ void k_dof_to_node(int n_dofs, const int* __restrict__ free_rows, const double* __restrict__ in,
                              double* __restrict__ out, int64_t in_stride, int64_t out_stride) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int v = blockIdx.y;
  if (i >= n_dofs) return;
  out[v * out_stride + free_rows[i]] = in[v * in_stride + i];
}

__global__ void k_node_to_dof(int n_dofs, const int* __restrict__ free_rows, const double* __restrict__ in,
                              double* __restrict__ out, int64_t in_stride, int64_t out_stride) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int v = blockIdx.y;
  if (i >= n_dofs) return;
  out[v * out_stride + i] = in[v * in_stride + free_rows[i]];
}

// ------------------------------------------------------------------ PCG
// Device-resident Jacobi-PCG. FP64 loop, two sums an iteration:
//   1: p_new = z + beta p_old (formed at the gathered columns, written for own
//      rows), q = K p_new, sum p.q -> alpha = z.r / p.q (breakdown check)
//   2: r -= alpha q, x += alpha p_new, z = D^-1 r, sums r.r and z.r -> err =
//      ||r||/||b||, convergence, beta
// p is double-buffered by iteration parity so gathered columns are never read
// while being overwritten. All sums are taken in a fixed order (deterministic
// results).
//
// k_pcg_resident: a matrix whose values fit the shared memory of a third of the SMs
// (3 slices an SM in FP64, 6 in FP32: 4,700 and 9,400 lattice nodes on 148) is copied
// there once, the whole solve is one cooperative launch, and its phases are separated
// by grid-wide sums, in which every CTA adds all CTAs' partials itself; bound by the two
// sums (2.5 us each): 10 x 4 x 4 5.8 us an iteration, 14^3 7.8, 20^3 mixed 10.7. It holds its
// SMs until it ends, so it gets no more of them: with all 148, or with a cooperative
// loop that streams larger matrices, a batch of 24^3 x 256 on another stream took 136
// ms beside 20^3 solves and 1,296 beside 64^3 ones, and 13 to 39 beside launches that
// end.
//
// k_pcg_product and k_pcg_step (k_pcgm_*): two launches an iteration for all other
// matrices, repeated by a graph's WHILE node; a launch after the end of the solve
// returns at once. The CTA that finishes last adds the partials. A launch starts while
// the one before it ends and loads its first values meanwhile. Bound by HBM, or by L2
// and the two launches' latency for matrices that stay there: 20^3 12.3 us an iteration,
// 37 x 22 x 29 16.2 (mixed 14.2), 32^3 18.2 (15.4), 48^3 51 (35), 64^3 102 (62; HBM
// alone 88 and 47).

constexpr int kPcgThreads = 256, kPcgWarps = kPcgThreads / 32;
constexpr int kPcgSums = 3;        // values of a sum at most
constexpr int kPcgMaxCtas = 8;     // CTAs an SM of a launch at most (sizes the partial sums)
constexpr int kPcgSpin = 1 << 22;  // polls of a grid-wide sum before it gives up

// v[k] of the CTA's threads summed and left in part[k][CTA] (thread 0 of the CTA has
// passed a fence after it). NW: warps of the CTA.
template <int NW, int K>
__device__ __forceinline__ void leave_partials(double* part, const double (&v)[K]) {
  __shared__ double sh[NW][K];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, G = gridDim.x;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double t = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (l == 0) sh[w][k] = t;
  }
  __syncthreads();  // (and every thread's stores of this phase are ordered before the fence)
  if (w == 0) {
    if (l < K) {
      double t = 0;
#pragma unroll
      for (int i = 0; i < NW; ++i) t += sh[i][l];
      part[(size_t)l * G + blockIdx.x] = t;
    }
    __syncwarp();
    if (l == 0) __threadfence();
  }
}

// out[k] = the CTAs' partials added: thread t takes t, t + 32 NW, ... in order, then the
// block's fixed tree. Every thread of the CTA gets it.
template <int NW, int K>
__device__ __forceinline__ void add_partials(const double* part, double (&out)[K]) {
  __shared__ double sh[NW][K];
  constexpr int T = 32 * NW;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, G = gridDim.x;
  double t[K];
#pragma unroll
  for (int k = 0; k < K; ++k) t[k] = threadIdx.x < G ? __ldcg(part + (size_t)k * G + threadIdx.x) : 0.0;
  int i = threadIdx.x + T;
  for (; i + 3 * T < G; i += 4 * T) {  // four loads in flight, added in order
    double u[K][4];
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) u[k][j] = __ldcg(part + (size_t)k * G + i + j * T);
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) t[k] += u[k][j];
  }
  for (; i < G; i += T)
#pragma unroll
    for (int k = 0; k < K; ++k) t[k] += __ldcg(part + (size_t)k * G + i);
#pragma unroll
  for (int k = 0; k < K; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t[k] += __shfl_down_sync(0xffffffffu, t[k], o);
    if (l == 0) sh[w][k] = t[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double x = 0;
#pragma unroll
    for (int j = 0; j < NW; ++j) x += sh[j][k];
    out[k] = x;
  }
}

// Grid-wide sums of one cooperative solve: the CTAs' partial sums (two buffers, used in
// turn: a CTA can be at most one sum ahead of another) and the arrival counter, cleared
// before the launch.
struct PcgGrid {
  double* part;       // [2][kPcgSums][grid]
  unsigned* arrived;
  unsigned target;    // arrivals that complete the next sum
  int buf;
  int spin = kPcgSpin;  // polls of a wait
};

// out[k] = sum over the grid of v[k], every thread of every CTA; what the CTAs
// wrote before is visible after. False when the bounded wait expired (the kernel
// then returns).
template <int NW, int K>
__device__ __forceinline__ bool grid_sum(PcgGrid& g, const double (&v)[K], double (&out)[K]) {
  __shared__ int ok;
  const int G = gridDim.x;
  double* part = g.part + (size_t)g.buf * kPcgSums * G;
  g.buf ^= 1;
  g.target += G;
  leave_partials<NW, K>(part, v);
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(g.arrived) : "memory");
    int good = 0;
    for (int i = 0; i < g.spin && !good; ++i) {
      unsigned n;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(g.arrived) : "memory");
      good = (int)(n - g.target) >= 0;
    }
    __threadfence();
    ok = good;
  }
  __syncthreads();
  if (!ok) return false;
  add_partials<NW, K>(part, out);
  return true;
}

// The sum of a launch: true in the CTA that finishes last, which gets it.
template <int NW, int K>
__device__ __forceinline__ bool last_sum(double* part, unsigned* counter, const double (&v)[K], double (&out)[K]) {
  __shared__ int last;
  leave_partials<NW, K>(part, v);
  if (threadIdx.x == 0) {
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return false;
  add_partials<NW, K>(part, out);
  if (threadIdx.x == 0) *counter = 0;  // for the next launch
  return true;
}

// y += the 3x3 block a times u. FP32 values multiply in FP32 and add in FP64.
template <class V>
__device__ __forceinline__ void block_row(const V (&a)[9], const V (&u)[3], double (&y)[3]) {
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    if constexpr (sizeof(V) == 8)
      y[r] += a[3 * r] * u[0] + a[3 * r + 1] * u[1] + a[3 * r + 2] * u[2];
    else
      y[r] += (double)fmaf(a[3 * r + 2], u[2], fmaf(a[3 * r + 1], u[1], a[3 * r] * u[0]));
  }
}

// Part of a slice's row sums y = K u formed by warp w of the W that share the
// slice (slots w, w + W, ...): U slots at a time, all their values requested
// before use (kStream: evict-first, for matrices that do not stay in L2).
// gather(c, u3) gives u at node c; first() runs when the first group's loads are under way.
template <int W, int U, bool kStream, class V, class Gather, class First>
__device__ __forceinline__ void slice_rows(int64_t s0, int64_t s1, int w, int lane, const int* __restrict__ col,
                                           const V* __restrict__ val, Gather gather, double (&y)[3], First first) {
  y[0] = y[1] = y[2] = 0.0;
  bool begin = true;
  for (int64_t s = s0 + w; s < s1; s += U * W) {
    V a[U][9];
    int c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      c[u] = -1;
      if (s + u * W >= s1) continue;
      c[u] = __ldg(col + (s + u * W) * 32 + lane);
      const V* v = val + (s + u * W) * 288 + lane;
#pragma unroll
      for (int k = 0; k < 9; ++k) a[u][k] = kStream ? __ldcs(v + k * 32) : __ldg(v + k * 32);
    }
    if (begin) first();
    begin = false;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c[u] >= 0) {  // (padding: -1)
        V x[3];
        gather(c[u], x);
        block_row(a[u], x, y);
      }
  }
}

struct PcgMat {
  int n_rows, n_slices;
  const int64_t* slice_ptr;
  const int* col;
};

// Visits the CTA's slices: f(slice) by all warps together, W warps a slice (kPcgWarps / W
// slices at a time). kOnce: the launch has a CTA for every kPcgWarps / W slices.
template <int W, bool kOnce, class F>
__device__ __forceinline__ void for_slices(int n_slices, F f) {
  constexpr int S = kPcgWarps / W;
  if constexpr (kOnce)
    f(blockIdx.x * S + (int)(threadIdx.x >> 5) / W);
  else
    for (int base = blockIdx.x * S; base < n_slices; base += gridDim.x * S) f(base + (int)(threadIdx.x >> 5) / W);
}

// y of the W warps of each slice summed in warp order; valid in warp 0 of the slice.
// (ys: [warps of the CTA][3][32] of shared memory.)
template <int W>
__device__ __forceinline__ void join_warps(double (&y)[3], double (*ys)[3][32]) {
  if constexpr (W > 1) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 3; ++c) ys[warp][c][lane] = y[c];
    __syncthreads();
    if (warp % W == 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
        for (int i = 1; i < W; ++i) y[c] += ys[warp + i][c][lane];
    }
  }
}

struct PcgEnd {  // how a solve ended (CTA 0 writes it)
  __device__ static void write(PcgState* st, double err, int status, int iterations, int matvecs) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->err = err;
      st->status = status;
      st->iterations = iterations;
      st->matvecs = matvecs;
      st->done = 1;
    }
  }
};

// Programmatic dependent launch: a launch's CTAs start while those of the launch before
// it finish, load what no launch changes, and wait for its results here.
__device__ __forceinline__ void wait_for_launch() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Whether the solve had ended before the launch began (it waits all the same).
__device__ __forceinline__ bool over(const PcgState* st) {
  if (!*reinterpret_cast<const volatile int*>(&st->done)) return false;
  wait_for_launch();
  return true;
}

// Elements i of a launch's vectors: f(i).
template <class F>
__device__ __forceinline__ void for_elements(int n, F f) {
  for (int i = blockIdx.x * kPcgThreads + threadIdx.x; i < n; i += gridDim.x * kPcgThreads) f(i);
}

// The loop of a solve whose launches a graph's WHILE node repeats (on = 0: the host
// enqueues them).
struct PcgLoop {
  int on;
  cudaGraphConditionalHandle handle;
  __device__ void end() const {
    if (on) cudaGraphSetConditional(handle, 0);
  }
  // One launch of the step: the loop's bound, and its end once the solve is over. (At
  // most two steps an iteration, so that the bound is never the reason to stop.)
  __device__ void step(PcgState* st, bool over) const {
    if (!on || blockIdx.x > 0 || threadIdx.x > 0) return;
    if (over || ++st->steps > 2LL * st->max_it + 2) cudaGraphSetConditional(handle, 0);
  }
};
struct PcgLimits {
  double tol, delta;  // delta: the mixed loop's reliable-update factor
  int max_it;
};

// Start of an FP64 solve: x = 0, r = b, z = D^-1 r, sums b.b and z.b.
__global__ void __launch_bounds__(kPcgThreads)
    k_pcg_start(int n3, const double* __restrict__ b, const double* __restrict__ dinv, double* x, double* r, double* z,
                double* p0, double* part, PcgState* st, PcgLimits lim) {
  double v[2] = {0.0, 0.0}, t[2];
  for_elements(n3, [&](int i) {
    const double bi = b[i], zi = dinv[i] * bi;
    r[i] = bi; x[i] = 0; z[i] = zi; p0[i] = 0;
    v[0] += bi * bi;
    v[1] += zi * bi;
  });
  if (!last_sum<kPcgWarps, 2>(part, &st->counter, v, t) || threadIdx.x) return;
  st->tol = lim.tol;
  st->max_it = lim.max_it;
  st->bnorm = sqrt(t[0]);
  st->zr = t[1];
  st->done = !(st->bnorm > 1e-25);  // SolverPCG.cs:112
}

// p_new = z + beta p_old, q = K p_new, alpha.
template <int W, bool kStream>
__global__ void __launch_bounds__(kPcgThreads, 3)
    k_pcg_product(PcgMat M, const double* __restrict__ val, const double* z, double* p0, double* p1,
                  double* __restrict__ q, double* part, PcgState* st) {
  __shared__ double ys[W > 1 ? kPcgWarps : 1][3][32];
  if (over(st)) return;
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) % W;
  double beta = 0.0, v[1] = {0.0}, t[1];
  const double* pold = nullptr;
  double* pnew = nullptr;
  int it = 0, done = 0;
  auto start = [&] {  // (once; the first slice's values are under way)
    if (pnew) return;
    wait_for_launch();
    beta = st->beta;
    it = st->it;
    done = st->done;
    pold = (it & 1) ? p1 : p0;
    pnew = (it & 1) ? p0 : p1;
  };
  auto dir = [&](int c, double (&u)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) u[k] = z[3 * c + k] + beta * pold[3 * c + k];
  };
  for_slices<W, (W > 2)>(M.n_slices, [&](int slice) {
    const int row = slice * 32 + lane;
    const bool live = slice < M.n_slices && row < M.n_rows;
    double y[3] = {0.0, 0.0, 0.0};
    if (live) slice_rows<W, 2, kStream>(M.slice_ptr[slice], M.slice_ptr[slice + 1], w, lane, M.col, val, dir, y, start);
    start();
    join_warps<W>(y, ys);
    if (w == 0 && live) {
      double pn[3];
      dir(row, pn);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        pnew[3 * row + k] = pn[k];
        q[3 * row + k] = y[k];
      }
      v[0] += pn[0] * y[0] + pn[1] * y[1] + pn[2] * y[2];
    }
  });
  if (done || !last_sum<kPcgWarps, 1>(part, &st->counter, v, t) || threadIdx.x) return;
  st->matvecs = it + 1;
  if (!(t[0] > 0) || isnan(t[0])) {  // breakdown: p.q <= 0 or NaN
    st->status = MSG_ERR_BREAKDOWN;
    st->iterations = it;
    st->done = 1;
  } else {
    st->alpha = st->zr / t[0];
  }
}

// r -= alpha q, x += alpha p_new, z = D^-1 r, err, beta.
__global__ void __launch_bounds__(kPcgThreads)
    k_pcg_step(int n3, const double* __restrict__ dinv, double* x, double* r, double* z, const double* p0,
               const double* p1, const double* q, double* part, PcgState* st, PcgLoop loop) {
  wait_for_launch();
  const bool over = st->done;
  loop.step(st, over);
  if (over) return;
  const int it = st->it;
  const double alpha = st->alpha;
  const double* p = (it & 1) ? p0 : p1;
  double v[2] = {0.0, 0.0}, t[2];
  for_elements(n3, [&](int i) {
    const double ri = r[i] - alpha * q[i], zi = dinv[i] * ri;
    r[i] = ri;
    x[i] += alpha * p[i];
    z[i] = zi;
    v[0] += ri * ri;
    v[1] += zi * ri;
  });
  if (!last_sum<kPcgWarps, 2>(part, &st->counter, v, t) || threadIdx.x) return;
  const int limit = st->max_it;
  st->err = sqrt(t[0]) / st->bnorm;
  if (st->err < st->tol) {
    st->iterations = it;
    st->done = 1;
  } else if (it + 1 >= limit) {
    st->iterations = limit;
    st->status = MSG_ERR_NOT_CONVERGED;
    st->done = 1;
  }
  if (st->done) loop.end();
  st->beta = t[1] / st->zr;
  st->zr = t[1];
  st->it = it + 1;
}

// The same loop for matrices whose values fit the shared memory of a third of the SMs:
// a CTA, alone on its SM, copies the values and columns of its S slices there once (W
// warps a slice), and each thread keeps the r, x, D^-1 of its own component in
// registers, so that an iteration reads only z and p_old at the gathered columns from
// L2.
constexpr int kPcgResidentSmem = 204 * 1024;
template <class V>
inline size_t pcg_resident_smem(int64_t slots) {  // of a CTA with that many slots
  return (size_t)slots * 32 * (9 * sizeof(V) + sizeof(int));
}

// What the two resident kernels share: the copy of a CTA's slices, and a row's sum
// from it.
template <int S, int W, class V>
struct Resident {
  V* vals;
  int* cols;
  int sl, w, lane, slice, row, t0, t1, n_slots;
  bool have, live;
  __device__ Resident(const PcgMat& M, const V* __restrict__ val, void* smem) {
    const int warp = threadIdx.x >> 5, first = blockIdx.x * S;
    lane = threadIdx.x & 31;
    w = warp % W;
    sl = warp / W;
    slice = first + sl;
    row = slice * 32 + lane;
    have = slice < M.n_slices;
    live = have && row < M.n_rows;
    const int64_t a0 = M.slice_ptr[first], a1 = M.slice_ptr[min(first + S, M.n_slices)];
    n_slots = (int)(a1 - a0);
    t0 = have ? (int)(M.slice_ptr[slice] - a0) : 0;
    t1 = have ? (int)(M.slice_ptr[slice + 1] - a0) : 0;
    vals = static_cast<V*>(smem);
    cols = reinterpret_cast<int*>(vals + (size_t)n_slots * 288);
    for (int i = threadIdx.x; i < n_slots * 32; i += 32 * S * W) cols[i] = M.col[a0 * 32 + i];
    for (int i = threadIdx.x; i < n_slots * 288; i += 32 * S * W) vals[i] = val[a0 * 288 + i];
    __syncthreads();
  }
  // y = the part of the row's sum in the slots of this warp, four slots' gathers at a time
  template <class Gather>
  __device__ __forceinline__ void sum(Gather gather, double (&y)[3]) const {
    constexpr int U = 4;
    y[0] = y[1] = y[2] = 0.0;
    if (!live) return;
    for (int s = t0 + w; s < t1; s += U * W) {
      V u[U][3];
      int c[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        c[q] = s + q * W < t1 ? cols[(s + q * W) * 32 + lane] : -1;
        if (c[q] >= 0) gather(c[q], u[q]);
      }
#pragma unroll
      for (int q = 0; q < U; ++q)
        if (c[q] >= 0) {
          V a[9];
#pragma unroll
          for (int k = 0; k < 9; ++k) a[k] = vals[(s + q * W) * 288 + k * 32 + lane];
          block_row(a, u[q], y);
        }
    }
  }
};

template <int S, int W>
__global__ void __launch_bounds__(32 * S * W, 1)
    k_pcg_resident(PcgMat M, const double* __restrict__ val, const double* __restrict__ b,
                   const double* __restrict__ dinv, double* x, double* z, double* p0, double* p1, PcgGrid grid,
                   PcgState* st, double tol, int max_it) {
  constexpr int NW = S * W;
  extern __shared__ __align__(16) unsigned char pcg_smem[];
  __shared__ double ys[NW][3][32];
  __shared__ double qs[S][96], ps[S][96];
  const Resident<S, W, double> A(M, val, pcg_smem);
  const int lane = A.lane, sl = A.sl, row = A.row;
  // the thread's own component of its slice (warps 0, 1, 2 of it)
  const int e = A.w * 32 + lane, i = A.slice * 96 + e;
  const bool own = A.have && A.w < 3 && i < 3 * M.n_rows;
  double r = 0.0, xi = 0.0, dv = 0.0;
  double s2[2] = {0.0, 0.0}, t2[2], u1[1];
  if (own) {
    r = b[i];
    dv = dinv[i];
    const double zi = dv * r;
    z[i] = zi;
    p0[i] = 0;
    s2[0] = r * r;
    s2[1] = zi * r;
  }
  if (!grid_sum<NW, 2>(grid, s2, t2)) return;
  const double bnorm = sqrt(t2[0]);
  double zr = t2[1], beta = 0.0, err = 0.0;
  int status = MSG_OK, iterations = 0, it = 0;
  const bool solve = bnorm > 1e-25;  // SolverPCG.cs:112
  while (solve) {
    double* pold = (it & 1) ? p1 : p0;
    double* pnew = (it & 1) ? p0 : p1;
    auto dir = [&](int c, double (&u)[3]) {
#pragma unroll
      for (int k = 0; k < 3; ++k) u[k] = z[3 * c + k] + beta * pold[3 * c + k];
    };
    double y[3], pn[3] = {0.0, 0.0, 0.0};
    const bool first = A.w == 0 && A.live;
    if (first) dir(row, pn);
    A.sum(dir, y);
    join_warps<W>(y, ys);
    const double v1[1] = {first ? pn[0] * y[0] + pn[1] * y[1] + pn[2] * y[2] : 0.0};
    if (first) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        pnew[3 * row + k] = pn[k];
        ps[sl][3 * lane + k] = pn[k];
        qs[sl][3 * lane + k] = y[k];
      }
    }
    if (!grid_sum<NW, 1>(grid, v1, u1)) return;
    if (!(u1[0] > 0) || isnan(u1[0])) {  // breakdown: p.q <= 0 or NaN
      status = MSG_ERR_BREAKDOWN;
      iterations = it;
      break;
    }
    const double alpha = zr / u1[0];
    s2[0] = s2[1] = 0.0;
    if (own) {
      r -= alpha * qs[sl][e];
      xi += alpha * ps[sl][e];
      const double zi = dv * r;
      z[i] = zi;
      s2[0] = r * r;
      s2[1] = zi * r;
    }
    if (!grid_sum<NW, 2>(grid, s2, t2)) return;
    err = sqrt(t2[0]) / bnorm;
    if (err < tol) {
      iterations = it;
      break;
    }
    if (++it >= max_it) {
      iterations = max_it;
      status = MSG_ERR_NOT_CONVERGED;
      break;
    }
    beta = t2[1] / zr;
    zr = t2[1];
  }
  if (own) x[i] = xi;
  PcgEnd::write(st, err, status, iterations, it);
}

// ------------------------------------------------------------------ mixed-precision PCG
// MSG_PCG_SOLVE_MIXED's loop: FP32 matrix values and FP32 vectors (r, p, q, the
// correction d and D^-1) inside the loop, the iterate x in FP64 (x += d at each
// FP64 true residual) and FP64 sums for every dot product. Two sums an iteration:
//   1: q = K32 p, sums p.q, (D r).q and q.D q -> alpha = gamma / p.q (breakdown
//      check) and, since r' = r - alpha q, gamma' = (D r').r' = gamma - 2 alpha
//      (D r).q + alpha^2 q.D q, hence beta = gamma' / gamma before the update;
//   2: r -= alpha q, d += alpha p, z = D r, p = z + beta p (the next direction,
//      formed in the same pass), exact sums z.r and r.r -> gamma = z.r, and a
//      true residual when ||r||/||b|| has dropped by delta since the last one or
//      below tol: x += d, r = b - K64 x with the FP64 values (stop when
//      ||r||/||b|| < tol in FP64), the direction kept. The true residual takes the
//      place of an iteration's two launches (x += d in the product's, r in the step's).
__global__ void __launch_bounds__(kPcgThreads)
    k_pcgm_start(int n3, const double* __restrict__ b, const double* __restrict__ dinv, double* x, float* r32,
                 float* p32, float* d32, float* dinv32, double* part, PcgState* st, PcgLimits lim) {
  double v[2] = {0.0, 0.0}, t[2];
  for_elements(n3, [&](int i) {
    const double bi = b[i];
    const float rv = (float)bi, dv = (float)dinv[i], zv = dv * rv;
    x[i] = 0;
    r32[i] = rv;
    dinv32[i] = dv;
    p32[i] = zv;
    d32[i] = 0.f;
    v[0] += bi * bi;
    v[1] += (double)zv * (double)rv;
  });
  if (!last_sum<kPcgWarps, 2>(part, &st->counter, v, t) || threadIdx.x) return;
  st->tol = lim.tol;
  st->delta = lim.delta;
  st->max_it = lim.max_it;
  st->bnorm = sqrt(t[0]);
  st->zr = t[1];
  st->err_ref = 1.0;
  st->done = !(st->bnorm > 1e-25);  // SolverPCG.cs:112
}

template <int W, bool kStream>
__global__ void __launch_bounds__(kPcgThreads, 4)
    k_pcgm_product(PcgMat M, const float* __restrict__ val32, double* x, const float* r32, const float* p32,
                   float* q32, float* d32, const float* dinv32, double* part, PcgState* st) {
  __shared__ double ys[W > 1 ? kPcgWarps : 1][3][32];
  if (over(st)) return;
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) % W;
  bool waited = false;
  int need = 0, done = 0;
  auto start = [&] {  // (once; the first slice's values are under way)
    if (waited) return;
    wait_for_launch();
    waited = true;
    need = st->need;
    done = st->done;
  };
  double v[3] = {0.0, 0.0, 0.0}, t[3];
  auto dir = [&](int c, float (&u)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) u[k] = p32[3 * c + k];
  };
  for_slices<W, (W > 2)>(M.n_slices, [&](int slice) {
    if (need) return;
    const int row = slice * 32 + lane;
    const bool live = slice < M.n_slices && row < M.n_rows;
    double y[3] = {0.0, 0.0, 0.0};
    if (live) slice_rows<W, (W > 2 ? 4 : 3), kStream>(M.slice_ptr[slice], M.slice_ptr[slice + 1], w, lane, M.col, val32, dir, y, start);
    start();
    join_warps<W>(y, ys);
    if (w == 0 && live && !need) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int i = 3 * row + k;
        const float qf = (float)y[k], dv = dinv32[i];
        q32[i] = qf;
        v[0] += (double)p32[i] * (double)qf;
        v[1] += (double)(dv * r32[i]) * (double)qf;
        v[2] += (double)(dv * qf) * (double)qf;
      }
    }
  });
  if (done) return;
  if (need) {
    for_elements(3 * M.n_rows, [&](int i) {
      x[i] += (double)d32[i];
      d32[i] = 0.f;
    });
    return;
  }
  if (!last_sum<kPcgWarps, 3>(part, &st->counter, v, t) || threadIdx.x) return;
  st->matvecs += 1;
  if (!(t[0] > 0) || isnan(t[0])) {  // breakdown: p.q <= 0 or NaN
    st->status = MSG_ERR_BREAKDOWN;
    st->iterations = st->it;
    st->done = 1;
    return;
  }
  const double zr = st->zr, alpha = zr / t[0];
  const double g1 = zr - 2.0 * alpha * t[1] + alpha * alpha * t[2];
  st->alpha = alpha;
  st->beta = g1 > 0.0 ? g1 / zr : 0.0;  // a non-positive estimate restarts from z
}

template <int W>
__global__ void __launch_bounds__(kPcgThreads, 4)
    k_pcgm_step(PcgMat M, const double* __restrict__ val, const double* __restrict__ b, const double* x, float* r32,
                float* p32, const float* q32, float* d32, const float* dinv32, double* part, PcgState* st, PcgLoop loop) {
  __shared__ double ys[W > 1 ? kPcgWarps : 1][3][32];
  wait_for_launch();
  const bool over = st->done;
  loop.step(st, over);
  if (over) return;
  const bool need = st->need;
  double v[2] = {0.0, 0.0}, t[2];
  if (need) {
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) % W;
    for_slices<W, false>(M.n_slices, [&](int slice) {
      const int row = slice * 32 + lane;
      const bool live = slice < M.n_slices && row < M.n_rows;
      double y[3] = {0.0, 0.0, 0.0};
      auto at = [&](int c, double (&u)[3]) {
#pragma unroll
        for (int k = 0; k < 3; ++k) u[k] = x[3 * c + k];
      };
      if (live) slice_rows<W, 1, true>(M.slice_ptr[slice], M.slice_ptr[slice + 1], w, lane, M.col, val, at, y, [] {});
      join_warps<W>(y, ys);
      if (w == 0 && live) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const int i = 3 * row + k;
          const double ri = b[i] - y[k];
          const float rv = (float)ri;
          r32[i] = rv;
          v[0] += ri * ri;
          v[1] += (double)(dinv32[i] * rv) * (double)rv;
        }
      }
    });
  } else {
    const float al = (float)st->alpha, be = (float)st->beta;
    for_elements(3 * M.n_rows, [&](int i) {
      const float pv = p32[i], rn = fmaf(-al, q32[i], r32[i]), zv = dinv32[i] * rn;
      d32[i] = fmaf(al, pv, d32[i]);
      p32[i] = fmaf(be, pv, zv);
      r32[i] = rn;
      v[0] += (double)rn * (double)rn;
      v[1] += (double)zv * (double)rn;
    });
  }
  if (!last_sum<kPcgWarps, 2>(part, &st->counter, v, t) || threadIdx.x) return;
  const double err = sqrt(t[0]) / st->bnorm, tol = st->tol;
  const int it = st->it, limit = st->max_it;
  st->err = err;
  if (!need && (err < tol || err < st->delta * st->err_ref)) {
    st->zr = t[1];
    st->need = 1;  // the next two launches
    return;
  }
  if (need) {
    st->need = 0;
    if (err < tol) {
      st->iterations = it;
      st->done = 1;
      loop.end();
      return;
    }
    st->err_ref = err;
  }
  st->zr = t[1];
  if (it + 1 >= limit) {
    st->iterations = limit;
    st->status = MSG_ERR_NOT_CONVERGED;
    st->done = 1;
    loop.end();
  }
  st->it = it + 1;
}

// A correction left by a solve that ended without a true residual.
__global__ void __launch_bounds__(kPcgThreads) k_pcgm_fold(int n3, double* x, const float* __restrict__ d32) {
  for_elements(n3, [&](int i) { x[i] += (double)d32[i]; });
}

// The mixed loop on resident FP32 values (Resident): the thread keeps r, p, d, D^-1,
// b and x of its component in registers; the FP64 values of the true residuals
// stream from memory.
template <int S, int W>
__global__ void __launch_bounds__(32 * S * W, 1)
    k_pcg_mixed_resident(PcgMat M, const double* __restrict__ val, const float* __restrict__ val32,
                         const double* __restrict__ b, const double* __restrict__ dinv, double* x, float* p32,
                         PcgGrid grid, PcgState* st, double tol, double delta, int max_it) {
  constexpr int NW = S * W;
  extern __shared__ __align__(16) unsigned char pcg_smem[];
  __shared__ double ys[NW][3][32];
  __shared__ double qs[S][96];
  const Resident<S, W, float> A(M, val32, pcg_smem);
  const int lane = A.lane, sl = A.sl;
  const int e = A.w * 32 + lane, i = A.slice * 96 + e;
  const bool own = A.have && A.w < 3 && i < 3 * M.n_rows, first = A.w == 0 && A.live;
  double bi = 0.0, xi = 0.0;
  float r = 0.f, p = 0.f, d = 0.f, dv = 0.f;
  double s2[2] = {0.0, 0.0}, t2[2], t3[3];
  if (own) {
    bi = b[i];
    r = (float)bi;
    dv = (float)dinv[i];
    p = dv * r;
    p32[i] = p;
    s2[0] = bi * bi;
    s2[1] = (double)p * (double)r;
  }
  if (!grid_sum<NW, 2>(grid, s2, t2)) return;
  const double bnorm = sqrt(t2[0]);
  double zr = t2[1], err = 0.0, err_ref = 1.0;
  int status = MSG_OK, iterations = 0, it = 0, products = 0;
  bool done = !(bnorm > 1e-25);  // SolverPCG.cs:112
  // the row sums of the slices' first warps, as the components of the own threads
  auto spread = [&](double (&y)[3]) {
    join_warps<W>(y, ys);
    if (first)
#pragma unroll
      for (int k = 0; k < 3; ++k) qs[sl][3 * lane + k] = y[k];
    __syncthreads();
  };
  while (!done) {
    double y[3], s3[3] = {0.0, 0.0, 0.0};
    A.sum([&](int c, float (&u)[3]) {
#pragma unroll
      for (int k = 0; k < 3; ++k) u[k] = p32[3 * c + k];
    }, y);
    spread(y);
    float q = 0.f;
    if (own) {
      q = (float)qs[sl][e];
      s3[0] = (double)p * (double)q;
      s3[1] = (double)(dv * r) * (double)q;
      s3[2] = (double)(dv * q) * (double)q;
    }
    if (!grid_sum<NW, 3>(grid, s3, t3)) return;
    ++products;
    if (!(t3[0] > 0) || isnan(t3[0])) {  // breakdown: p.q <= 0 or NaN
      status = MSG_ERR_BREAKDOWN;
      iterations = it;
      break;
    }
    const double alpha = zr / t3[0];
    const double g1 = zr - 2.0 * alpha * t3[1] + alpha * alpha * t3[2];
    const float al = (float)alpha, be = (float)(g1 > 0.0 ? g1 / zr : 0.0);  // a non-positive estimate restarts from z
    s2[0] = s2[1] = 0.0;
    if (own) {
      r = fmaf(-al, q, r);
      const float zv = dv * r;
      d = fmaf(al, p, d);
      p = fmaf(be, p, zv);
      p32[i] = p;
      s2[0] = (double)r * (double)r;
      s2[1] = (double)zv * (double)r;
    }
    if (!grid_sum<NW, 2>(grid, s2, t2)) return;
    err = sqrt(t2[0]) / bnorm;
    zr = t2[1];
    if (err < tol || err < delta * err_ref) {
      if (own) {
        xi += (double)d;
        d = 0.f;
        x[i] = xi;
      }
      s2[0] = s2[1] = 0.0;
      if (!grid_sum<NW, 2>(grid, s2, t2)) return;  // x is complete
      y[0] = y[1] = y[2] = 0.0;
      if (A.live)
        slice_rows<W, 1, true>(M.slice_ptr[A.slice], M.slice_ptr[A.slice + 1], A.w, lane, M.col, val,
                               [&](int c, double (&u)[3]) {
#pragma unroll
                                 for (int k = 0; k < 3; ++k) u[k] = x[3 * c + k];
                               }, y, [] {});
      spread(y);
      if (own) {
        const double ri = bi - qs[sl][e];
        r = (float)ri;
        s2[0] = ri * ri;
        s2[1] = (double)(dv * r) * (double)r;
      }
      if (!grid_sum<NW, 2>(grid, s2, t2)) return;
      err = sqrt(t2[0]) / bnorm;
      if (err < tol) {
        iterations = it;
        done = true;
      } else {
        zr = t2[1];
        err_ref = err;
      }
    }
    if (!done && it + 1 >= max_it) {
      iterations = max_it;
      status = MSG_ERR_NOT_CONVERGED;
      done = true;
    }
    ++it;
  }
  if (own) x[i] = xi + (double)d;  // (a correction left by a solve that ended without a true residual)
  PcgEnd::write(st, err, status, iterations, products);
}

// Self-test of the sum's bounded wait: one CTA, one arrival short of the target
// (grid.target on entry), so that the sum gives up and the state stays not done, as a
// solve's would.
__global__ void __launch_bounds__(kPcgThreads) k_pcg_wait_selftest(PcgGrid grid, PcgState* st) {
  const double v[1] = {1.0};
  double t[1];
  if (!grid_sum<kPcgWarps, 1>(grid, v, t)) return;
  PcgEnd::write(st, t[0], MSG_OK, 0, 0);
}

__global__ void k_to_f32(size_t n, const double* __restrict__ a, float* __restrict__ b) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}

}  // namespace

int launch_to_f32(Context* ctx, size_t n, const double* a, float* b) {
  k_to_f32<<<ctx->sm_count * 8, 256, 0, ctx->stream>>>(n, a, b);
  count_launch(ctx);
  MSG_CUDA(ctx, cudaGetLastError());
  return MSG_OK;
}

int launch_bsr_assemble(Context* ctx, const Mesh* m, const double* d_Ke, double* d_val) {
  const int64_t n_pos = m->pat.n_slots * 32;
  if (n_pos == 0) return MSG_OK;
  const int64_t nt = n_pos * 9;
  k_bsr_assemble<<<(unsigned)((nt + 255) / 256), 256, 0, ctx->stream>>>(
      n_pos, m->d_col.as<int>(), m->d_contrib_ptr.as<int64_t>(), m->d_contrib.as<int>(), d_Ke, d_val);
  k_bsr_mask<<<(m->n_nodes + 127) / 128, 128, 0, ctx->stream>>>(m->n_nodes, m->d_slice_ptr.as<int64_t>(),
                                                                m->d_col.as<int>(), m->d_mask.as<uint8_t>(), d_val);
  count_launch(ctx, 2);
  MSG_CUDA(ctx, cudaGetLastError());
  return MSG_OK;
}

int launch_bsr_diag_inv(Context* ctx, const Mesh* m, const double* d_val, double* d_dinv) {
  k_bsr_diag_inv<<<(m->n_nodes + 127) / 128, 128, 0, ctx->stream>>>(m->n_nodes, m->d_diag_pos.as<int>(), d_val,
                                                                    d_dinv);
  count_launch(ctx);
  MSG_CUDA(ctx, cudaGetLastError());
  return MSG_OK;
}

int launch_bsr_spmv(Context* ctx, const Mesh* m, const double* d_val, const double* d_x, double* d_y) {
  k_bsr_spmv3<<<m->pat.n_slices, 96, 0, ctx->stream>>>(m->n_nodes, m->d_slice_ptr.as<int64_t>(), m->d_col.as<int>(),
                                                        d_val, d_x, d_y);
  count_launch(ctx);
  MSG_CUDA(ctx, cudaGetLastError());
  return MSG_OK;
}

int launch_dof_to_node(Context* ctx, const Mesh* m, const double* d_in, double* d_out, int n_vec, int64_t in_stride,
                       int64_t out_stride) {
  if (m->n_dofs == 0 || n_vec == 0) return MSG_OK;
  dim3 grid((m->n_dofs + 255) / 256, n_vec);
  k_dof_to_node<<<grid, 256, 0, ctx->stream>>>(m->n_dofs, m->d_free_rows.as<int>(), d_in, d_out, in_stride,
                                               out_stride);
  count_launch(ctx);
  MSG_CUDA(ctx, cudaGetLastError());
  return MSG_OK;
}

int launch_node_to_dof(Context* ctx, const Mesh* m, const double* d_in, double* d_out, int n_vec, int64_t in_stride,
                       int64_t out_stride) {
  if (m->n_dofs == 0 || n_vec == 0) return MSG_OK;
  dim3 grid((m->n_dofs + 255) / 256, n_vec);
  k_node_to_dof<<<grid, 256, 0, ctx->stream>>>(m->n_dofs, m->d_free_rows.as<int>(), d_in, d_out, in_stride,
                                               out_stride);
  count_launch(ctx);
  MSG_CUDA(ctx, cudaGetLastError());
  return MSG_OK;
}

namespace {

// Warps that share a slice (a warp alone takes its 27 slots one after another): as many
// as keep the product's CTAs, `per_sm` an SM, in one round, 2 where none do. FP64, us an
// iteration: 20^3 12.6 with 8, 13.3 with 4; 25^3 16.5 and 14.6; 32^3 25.6 with 8, 22.9
// with 4, 18.2 with 2; 40^3 38.3 with 4, 39.1 with 2, 36.2 with 1; 48^3 54.8, 52.2, 56.6.
constexpr int kPcgCtas = 3, kPcgmCtas = 4;  // CTAs an SM of the FP64 and the mixed product
int pcg_warps(const Context* ctx, const Mesh* m, int per_sm) {
  for (int W : {8, 4, 2, 1})
    if ((int64_t)m->pat.n_slices * W <= (int64_t)kPcgWarps * per_sm * ctx->sm_count) return W;
  return 2;
}

PcgMat pcg_mat(const Mesh* m) {
  return {m->n_nodes, m->pat.n_slices, m->d_slice_ptr.as<int64_t>(), m->d_col.as<int>()};
}

// CTAs of the launches over slices (one round of them: 64^3 102 us an iteration, 107
// with a CTA for every four slices) and over elements.
int pcg_slice_ctas(const Context* ctx, const Mesh* m, int W, int per_sm) {
  const int per = kPcgWarps / W;
  return std::max(1, std::min((m->pat.n_slices + per - 1) / per, ctx->sm_count * per_sm));
}
int pcg_element_ctas(const Context* ctx, const Mesh* m) {
  return std::max(1, std::min((3 * m->n_nodes + kPcgThreads - 1) / kPcgThreads, ctx->sm_count * kPcgMaxCtas));
}

// bytes of the partial sums (two buffers of a cooperative solve's CTAs, at most one an
// SM; one of a launch's), then the state
size_t pcg_head_bytes(const Context* ctx) { return sizeof(double) * kPcgSums * kPcgMaxCtas * ctx->sm_count + 256; }
PcgState* pcg_state(const Context* ctx, void* head) {
  return reinterpret_cast<PcgState*>(static_cast<char*>(head) + pcg_head_bytes(ctx) - 256);
}

// Values that do not stay in L2 between iterations stream through it evict-first
// (a 71 MB matrix: 18.2 us an iteration without, 18.7 with; 240 MB: 56 and 48).
bool pcg_stream(const Mesh* m, size_t value_bytes) { return (size_t)m->pat.n_slots * 288 * value_bytes > (size_t)100 << 20; }

// Slices an SM (at most `most`, the kernels' widest CTA) if the CTAs of a resident
// solve fit a third of the SMs, one an SM, with their slots in shared memory; 0
// otherwise.
template <class V>
int pcg_resident(const Context* ctx, const Mesh* m, int most, size_t* smem) {
  const std::vector<int64_t>& sp = m->pat.slice_ptr;
  const int sms = std::max(1, ctx->sm_count / 3), ns = m->pat.n_slices, S = (ns + sms - 1) / sms;
  if (S > most) return 0;
  int64_t slots = 0;
  for (int i = 0; i < ns; i += S) slots = std::max(slots, sp[std::min(i + S, ns)] - sp[i]);
  *smem = pcg_resident_smem<V>(slots);
  return *smem <= (size_t)kPcgResidentSmem ? S : 0;
}

struct PcgLaunch {
  const void* kernel = nullptr;
  int grid = 0, threads = kPcgThreads;
  size_t smem = 0;
};

// The shared memory of a resident kernel, allowed when a context first launches it
// (the limit is a device's, and other devices' contexts may live in the process) and
// always the same: other threads' solves of other sizes share it.
int pcg_resident_limit(Context* ctx, const void* kernel) {
  std::vector<const void*>& done = ctx->pcg_limits;
  if (std::find(done.begin(), done.end(), kernel) != done.end()) return MSG_OK;
  MSG_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPcgResidentSmem));
  done.push_back(kernel);
  return MSG_OK;
}

int pcg_cooperative(Context* ctx, const PcgLaunch& l, void** args, cudaStream_t s) {
  if (l.smem) MSG_TRY(pcg_resident_limit(ctx, l.kernel));
  MSG_CUDA(ctx, cudaLaunchCooperativeKernel(l.kernel, dim3(l.grid), dim3(l.threads), args, l.smem, s));
  count_launch(ctx);
  return MSG_OK;
}

// A launch that may begin while the one before it ends (its kernel waits for it).
template <class... Params, class... Args>
void dependent(void (*kernel)(Params...), int grid, cudaStream_t s, Args... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(kPcgThreads);
  c.stream = s;
  c.attrs = at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, Params(args)...);  // (its error is the next cudaGetLastError)
}

// The iterations of a solve, iteration(loop) enqueues one. With a matrix (A) they are a
// graph of its own, kept for its next solves with the same vectors, whose WHILE node
// repeats kPcgRound of them until the solve ends, with no host in between (launched by
// the host, 64^3 took 206 ms instead of 119 on a host with more busy processes than
// processors). Without one (nothing may be allocated) the host enqueues them, two
// rounds of about 0.4 ms ahead of its look at the state.
constexpr int kPcgRound = 8;
template <class F>
int pcg_iterate(Context* ctx, const Mesh* m, Matrix* A, const void* b, const void* x, bool mixed, PcgState* st,
                int max_it, F iteration, cudaStream_t s) {
  if (A) {
    PcgGraph& g = A->pcg_graph[mixed ? 1 : 0];
    if (g.exec && (g.b != b || g.x != x)) {
      cudaGraphExecDestroy(g.exec);
      g.exec = nullptr;
    }
    if (!g.exec) {
      struct Hold {
        cudaGraph_t g = nullptr;
        ~Hold() {
          if (g) cudaGraphDestroy(g);
        }
      } graph;
      MSG_CUDA(ctx, cudaGraphCreate(&graph.g, 0));
      PcgLoop loop{1, 0};
      MSG_CUDA(ctx, cudaGraphConditionalHandleCreate(&loop.handle, graph.g, 1, cudaGraphCondAssignDefault));
      cudaGraphNodeParams wp = {};
      wp.type = cudaGraphNodeTypeConditional;
      wp.conditional.handle = loop.handle;
      wp.conditional.type = cudaGraphCondTypeWhile;
      wp.conditional.size = 1;
      cudaGraphNode_t node = nullptr;
      MSG_CUDA(ctx, cudaGraphAddNode(&node, graph.g, nullptr, 0, &wp));
      cudaGraph_t body = wp.conditional.phGraph_out[0];
      MSG_CUDA(ctx, cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
      for (int i = 0; i < kPcgRound; ++i) iteration(loop);
      const cudaError_t le = cudaGetLastError(), ce = cudaStreamEndCapture(s, &body);
      if (le != cudaSuccess || ce != cudaSuccess) return cuda_error(ctx, le != cudaSuccess ? le : ce, "PCG loop capture");
      const cudaError_t ie = cudaGraphInstantiate(&g.exec, graph.g, 0);
      if (ie != cudaSuccess) {
        g.exec = nullptr;
        return cuda_error(ctx, ie, "cudaGraphInstantiate");
      }
      g.b = b;
      g.x = x;
    }
    MSG_CUDA(ctx, cudaGraphLaunch(g.exec, s));
    return MSG_OK;
  }
  static_assert(sizeof(PcgState) <= 128, "two states in the flag page's first 256 bytes");
  const double us = 10.0 + (double)m->pat.n_slots * 288 * (mixed ? sizeof(float) : sizeof(double)) / 6e6;
  const int round = std::min(max_it, (int)std::max(2.0, std::min(64.0, 400.0 / us)));
  PcgState* h[2] = {reinterpret_cast<PcgState*>(ctx->h_flags), reinterpret_cast<PcgState*>(ctx->h_flags + 32)};
  auto enqueue = [&](int k) -> int {
    for (int i = 0; i < round; ++i) iteration(PcgLoop{0, 0});
    MSG_CUDA(ctx, cudaGetLastError());
    MSG_CUDA(ctx, cudaMemcpyAsync(h[k], st, sizeof(PcgState), cudaMemcpyDeviceToHost, s));
    MSG_CUDA(ctx, cudaEventRecord(ctx->ev[k], s));
    return MSG_OK;
  };
  MSG_TRY(enqueue(0));
  for (int64_t n = 0, k = 0; n <= 2 * (int64_t)max_it + 2 * round; n += round, k ^= 1) {
    MSG_TRY(enqueue((int)k ^ 1));
    MSG_CUDA(ctx, cudaEventSynchronize(ctx->ev[k]));
    if (h[k]->done) break;
  }
  return MSG_OK;
}

// One FP64 solve on stream s (A: the matrix, where a graph may be allocated).
int pcg_launch(Context* ctx, const Mesh* m, const double* val, const double* b, const double* dinv, double* x,
               double* r, double* z, double* p0, double* p1, double* q, void* head, double tol, int max_it,
               cudaStream_t s, Matrix* A) {
  PcgMat M = pcg_mat(m);
  PcgState* st = pcg_state(ctx, head);
  double* part = static_cast<double*>(head);
  MSG_CUDA(ctx, cudaMemsetAsync(head, 0, pcg_head_bytes(ctx), s));
  PcgLaunch l;
  if (const int S = pcg_resident<double>(ctx, m, 3, &l.smem)) {
    PcgGrid g{part, &st->counter, 0u, 0};
    l.kernel = S == 1 ? (const void*)k_pcg_resident<1, 8> : S == 2 ? (const void*)k_pcg_resident<2, 4>
                                                                   : (const void*)k_pcg_resident<3, 4>;
    l.threads = S == 1 ? 256 : 128 * S;
    l.grid = (m->pat.n_slices + S - 1) / S;
    void* args[] = {&M, &val, &b, &dinv, &x, &z, &p0, &p1, &g, &st, &tol, &max_it};
    return pcg_cooperative(ctx, l, args, s);
  }
  const int W = pcg_warps(ctx, m, kPcgCtas), gs = pcg_slice_ctas(ctx, m, W, kPcgCtas), ge = pcg_element_ctas(ctx, m);
  const int n3 = 3 * m->n_nodes;
  const bool stream = pcg_stream(m, sizeof(double));
  auto product = W == 8   ? k_pcg_product<8, false>  // (never that large)
                 : W == 4 ? k_pcg_product<4, false>
                 : W == 2 ? (stream ? k_pcg_product<2, true> : k_pcg_product<2, false>)
                          : (stream ? k_pcg_product<1, true> : k_pcg_product<1, false>);
  k_pcg_start<<<ge, kPcgThreads, 0, s>>>(n3, b, dinv, x, r, z, p0, part, st, PcgLimits{tol, 0.0, max_it});
  count_launch(ctx);
  return pcg_iterate(ctx, m, A, b, x, false, st, max_it, [&](PcgLoop loop) {
    dependent(product, gs, s, M, val, z, p0, p1, q, part, st);
    dependent(k_pcg_step, ge, s, n3, dinv, x, r, z, p0, p1, q, part, st, loop);
  }, s);
}

// The state after a solve (its copy on the host); a cooperative solve whose grid barrier
// expired leaves it not done. Copied to pinned memory and then waited for: a copy to
// pageable memory waits inside the driver, and calls of other contexts with it (a batch
// beside long solves took the whole time of one in three of four processes).
int pcg_finish(Context* ctx, PcgState* st, PcgState* host, cudaStream_t s) {
  MSG_CUDA(ctx, cudaMemcpyAsync(ctx->h_flags, st, sizeof(PcgState), cudaMemcpyDeviceToHost, s));
  MSG_CUDA(ctx, cudaStreamSynchronize(s));
  std::memcpy(host, ctx->h_flags, sizeof(PcgState));
  if (!host->done) return set_error(ctx, MSG_ERR_TIMEOUT, "PCG: a bounded grid barrier expired");
  if (host->it > 0) count_launch(ctx, 2 * host->matvecs);  // of a solve in launches
  return MSG_OK;
}

}  // namespace

int pcg_wait_selftest(Context* ctx, int polls) {
  MSG_TRY(context_resources(ctx));
  DevMem head;
  MSG_TRY(head.alloc(ctx, pcg_head_bytes(ctx)));
  PcgState* st = pcg_state(ctx, head.ptr);
  MSG_CUDA(ctx, cudaMemsetAsync(head.ptr, 0, pcg_head_bytes(ctx), ctx->stream));
  PcgGrid g{head.as<double>(), &st->counter, 1u, 0, polls};
  k_pcg_wait_selftest<<<1, kPcgThreads, 0, ctx->stream>>>(g, st);
  count_launch(ctx);
  MSG_CUDA(ctx, cudaGetLastError());
  PcgState hs;
  return pcg_finish(ctx, st, &hs, ctx->stream);
}

// Runs the device PCG on node-layout vectors.
int pcg_solve_device(Context* ctx, Matrix* A, const double* d_b, double* d_x, int max_it, double tol, int* iterations,
                     double* rel_res, int* status, bool mixed) {
  Mesh* m = A->mesh;
  const size_t n = 3 * (size_t)m->n_nodes;
  cudaStream_t s = ctx->stream;
  MSG_TRY(context_resources(ctx));
  // one allocation for the partial sums, the state and the solve's vectors: r, z, p
  // (two), q in FP64, or in the mixed loop r, p, q, d and D^-1 in FP32
  const size_t nv = (n + 31) / 32 * 32, head = pcg_head_bytes(ctx);
  if (!A->d_work.ptr) MSG_TRY(A->d_work.alloc(ctx, head + sizeof(double) * 5 * nv));
  PcgState* st = pcg_state(ctx, A->d_work.ptr);
  double* v = reinterpret_cast<double*>(A->d_work.as<char>() + head);
  if (mixed) {
    const size_t nval = (size_t)m->pat.n_slots * 32 * 9;
    if (!A->d_val32.ptr) {
      MSG_TRY(A->d_val32.alloc(ctx, sizeof(float) * std::max<size_t>(1, nval)));
      k_to_f32<<<ctx->sm_count * 8, 256, 0, s>>>(nval, A->d_val.as<double>(), A->d_val32.as<float>());
      count_launch(ctx);
    }
    float* f = reinterpret_cast<float*>(v);
    PcgMat M = pcg_mat(m);
    PcgGrid g{A->d_work.as<double>(), &st->counter, 0u, 0};
    const double *val = A->d_val.as<double>(), *dinv = A->d_dinv.as<double>();
    const float* val32 = A->d_val32.as<float>();
    float *r32 = f, *p32 = f + nv, *q32 = f + 2 * nv, *d32 = f + 3 * nv, *dinv32 = f + 4 * nv;
    double delta = ctx->reliable_delta;
    MSG_CUDA(ctx, cudaMemsetAsync(A->d_work.ptr, 0, head, s));
    PcgLaunch l;
    if (const int S = pcg_resident<float>(ctx, m, 6, &l.smem)) {
      const void* ks[] = {(const void*)k_pcg_mixed_resident<1, 8>, (const void*)k_pcg_mixed_resident<2, 4>,
                          (const void*)k_pcg_mixed_resident<3, 4>, (const void*)k_pcg_mixed_resident<4, 3>,
                          (const void*)k_pcg_mixed_resident<5, 3>, (const void*)k_pcg_mixed_resident<6, 3>};
      l.kernel = ks[S - 1];
      l.threads = S == 1 ? 256 : S < 4 ? 128 * S : 96 * S;
      l.grid = (m->pat.n_slices + S - 1) / S;
      void* args[] = {&M, &val, &val32, &d_b, &dinv, &d_x, &p32, &g, &st, &tol, &delta, &max_it};
      MSG_TRY(pcg_cooperative(ctx, l, args, s));
    } else {
      const int W = pcg_warps(ctx, m, kPcgmCtas), gs = pcg_slice_ctas(ctx, m, W, kPcgmCtas), ge = pcg_element_ctas(ctx, m);
      const int n3 = (int)n;
      double* part = A->d_work.as<double>();
      const bool stream = pcg_stream(m, sizeof(float));
      auto product = W == 8   ? k_pcgm_product<8, false>
                     : W == 4 ? k_pcgm_product<4, false>
                     : W == 2 ? (stream ? k_pcgm_product<2, true> : k_pcgm_product<2, false>)
                              : (stream ? k_pcgm_product<1, true> : k_pcgm_product<1, false>);
      auto step = W == 8 ? k_pcgm_step<8> : W == 4 ? k_pcgm_step<4> : W == 2 ? k_pcgm_step<2> : k_pcgm_step<1>;
      k_pcgm_start<<<ge, kPcgThreads, 0, s>>>(n3, d_b, dinv, d_x, r32, p32, d32, dinv32, part, st,
                                              PcgLimits{tol, delta, max_it});
      MSG_TRY(pcg_iterate(ctx, m, A, d_b, d_x, true, st, max_it, [&](PcgLoop loop) {
        dependent(product, gs, s, M, val32, d_x, r32, p32, q32, d32, dinv32, part, st);
        dependent(step, ge, s, M, val, d_b, d_x, r32, p32, q32, d32, dinv32, part, st, loop);
      }, s));
      k_pcgm_fold<<<ge, kPcgThreads, 0, s>>>(n3, d_x, d32);
      count_launch(ctx, 2);
    }
  } else {
    MSG_TRY(pcg_launch(ctx, m, A->d_val.as<double>(), d_b, A->d_dinv.as<double>(), d_x, v, v + nv, v + 2 * nv,
                       v + 3 * nv, v + 4 * nv, A->d_work.ptr, tol, max_it, s, A));
  }
  PcgState hs;
  MSG_TRY(pcg_finish(ctx, st, &hs, s));
  if (iterations) *iterations = hs.iterations;
  if (rel_res) *rel_res = hs.err;
  if (status) *status = hs.status;
  return MSG_OK;
}

// ------------------------------------------------------------------ PCG without allocation
// Scratch of MSG_PCG_SOLVE_NOALLOC: a fixed array in device memory, so the call
// needs no cudaMalloc. Sized for meshes of up to kNoAllocMaxNodes nodes: seven
// node-layout FP64 vectors (b, x, r, z, two search directions, K p), the CTAs'
// partial sums and the scalar state, about 11 MB. Every GPU that loads the
// library holds this array until the process exits.
constexpr int kNoAllocMaxNodes = 65536;
constexpr size_t kNoAllocVecBytes = sizeof(double) * 3 * (size_t)kNoAllocMaxNodes;
constexpr size_t kNoAllocBytes = 7 * kNoAllocVecBytes + sizeof(double) * kPcgSums * kPcgMaxCtas * 256 + 256;  // up to 256 SMs
static_assert(sizeof(PcgState) <= 256, "the scalar state fits its slot");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// Device address of the scratch array on the current device (host code cannot
// use the array's name as a device address). MSG_CREATE looks it up once per
// context, with the context's device current, so no solve call triggers the
// module load that the first lookup may cause.
cudaError_t noalloc_scratch_address(unsigned char** out) {
  void* p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  *out = static_cast<unsigned char*>(p);
  return e;
}

}  // namespace msg

using namespace msg;

// The device Jacobi-PCG of MSG_PCG_SOLVE, for callers that must not allocate
// device memory during the solve: the solve's working vectors live in the
// fixed scratch array above instead of buffers from cudaMalloc, and the
// right-hand side and solution are the caller's device buffers. The kernels and
// their launch shapes are MSG_PCG_SOLVE's; the host enqueues them (a graph takes device
// memory).
extern "C" int MSG_PCG_SOLVE_NOALLOC(MSG_MAT A, const double* b_dev, double* x_dev, int max_it, double tol,
                                     int* iterations, double* rel_res) {
  if (!A || !b_dev || !x_dev || max_it <= 0 || !(tol > 0)) return MSG_ERR_INVALID_ARGUMENT;
  Mesh* m = A->mesh;
  Context* ctx = m->ctx;
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  MSG_CUDA(ctx, cudaSetDevice(ctx->device));
  MSG_TRY(context_resources(ctx));  // (host memory and events)
  const int nr = m->n_nodes;
  if (nr > kNoAllocMaxNodes)
    return set_error(ctx, MSG_ERR_INVALID_ARGUMENT,
                     "MSG_PCG_SOLVE_NOALLOC: mesh has %d nodes, the fixed scratch holds at most %d", nr,
                     kNoAllocMaxNodes);
  unsigned char* base = ctx->noalloc_scratch;
  if (!base) return set_error(ctx, MSG_ERR_CUDA, "MSG_PCG_SOLVE_NOALLOC: scratch address not resolved");
  const size_t n = 3 * (size_t)nr;
  double* bn = reinterpret_cast<double*>(base);
  double* xn = reinterpret_cast<double*>(base + kNoAllocVecBytes);
  double* v[5];  // r, z, p (two), q
  for (int i = 0; i < 5; ++i) v[i] = reinterpret_cast<double*>(base + (2 + i) * kNoAllocVecBytes);
  void* head = base + 7 * kNoAllocVecBytes;
  if (ctx->sm_count > 256) return set_error(ctx, MSG_ERR_INVALID_ARGUMENT, "MSG_PCG_SOLVE_NOALLOC: device too large");
  PcgState* st = pcg_state(ctx, head);
  cudaStream_t s = ctx->stream;
  // the array keeps the previous call's contents: clear what must start at zero
  MSG_CUDA(ctx, cudaMemsetAsync(bn, 0, sizeof(double) * n, s));
  MSG_TRY(launch_dof_to_node(ctx, m, b_dev, bn, 1, 0, 0));
  MSG_TRY(pcg_launch(ctx, m, A->d_val.as<double>(), bn, A->d_dinv.as<double>(), xn, v[0], v[1], v[2], v[3], v[4],
                     head, tol, max_it, s, nullptr));
  MSG_TRY(launch_node_to_dof(ctx, m, xn, x_dev, 1, 0, 0));
  PcgState hs;
  MSG_TRY(pcg_finish(ctx, st, &hs, s));
  if (iterations) *iterations = hs.iterations;
  if (rel_res) *rel_res = hs.err;
  if (hs.status != MSG_OK)
    return set_error(ctx, hs.status,
                     hs.status == MSG_ERR_BREAKDOWN ? "PCG breakdown (p.q <= 0 or NaN)" : "PCG did not converge");
  return MSG_OK;
}
