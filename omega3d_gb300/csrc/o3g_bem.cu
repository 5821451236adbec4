// o3g_bem.cu -- the BEM system of the boundary solve: BEM<S,I> (BEM.h:44-234).
//
// The reference holds a dense Eigen matrix and solves it with GMRES (BEM.h:182-202),
// checking ||Ax-b||/||b|| afterwards (:227-230).  Here the matrix lives on the device and
// is solved by
//   * an FP32 LU factorisation with partial pivoting (row-by-row the same pivot choice
//     as LAPACK's getrf: largest magnitude, first index on ties), panels of kNb columns:
//       - k_panel_cluster: panels of up to 10,240 rows, 64 columns at a time, in one thread-block
//         cluster: rows in registers, pivot candidates through distributed shared memory;
//       - k_panel_lu: taller ones; one cooperative kernel factors the whole kNb-column panel; each
//         block keeps its slab of rows in shared memory; per column every block publishes
//         its pivot candidate (the whole row, and the diagonal row if it holds it) and then
//         a tagged 64-bit key with release semantics; every block polls all keys (relaxed
//         loads issued together, then a fence), so one round of stores and polls is the
//         column's grid barrier and its exchange.
//         Each block updates the next column first, publishes its next candidate, and runs
//         the rest of the rank-1 update while the other blocks publish;
//       - k_laswp: the panel's row interchanges applied to the other columns;
//       - k_trsm_unit_lower, k_left_gemm: U12 = L11^-1 A12, one warp per column, or by the explicit
//         inverse for the columns beyond the outer panel;
//       - trailing update A22 -= L21 U12 on the tensor cores (o3g_tcgemm.cu: tcgen05, TF32
//         products, FP32 sums), two-level blocking so the big updates have k = 512;
//   * iterative refinement: residuals r = b - A x formed FP64-accurately (double-single
//     FP32 arithmetic, k_matvec_ds) from the unfactored FP32 matrix and the FP64 iterate,
//     corrections from the FP32 factors (k_trsv: forward/back substitution in one cooperative
//     kernel each, 512 columns a step by explicit inverses of the diagonal blocks), until ||r||/||b|| <= tol;
//   * or, without any factorisation, restarted GMRES -- the reference's own solver
//     (BEM.h:182-202) -- with FP64 Krylov vectors, classical Gram-Schmidt with one
//     reorthogonalisation, and the same FP64-accurate products (o3g_bem_solve_gmres).
// Every grid barrier and key poll here spins at most kSpinLimit rounds, then sets an error
// flag that all blocks check, so a fault in the barrier logic ends the kernel instead of
// hanging.
#include "o3g_common.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

namespace o3g {

constexpr int kNb = 128;              // panel width
constexpr int kNbOuter = 512;         // outer panel width: k of the big trailing updates
constexpr int kPanelThreads = 512;
constexpr int kSolveThreads = 1024;
constexpr unsigned long long kSpinLimit = 1ull << 25;

constexpr unsigned long long kTestSpinLimit = 1ull << 14;   // the wait test's limit (~1 ms)

struct Barrier {
  unsigned* count;
  int* err;
  unsigned long long limit;   // polls before giving up
  unsigned extra;             // 0; 1 in the wait test: one more arrival than blocks, never met
};

// the barrier over the handle's flag words (arrival counter, error), with the spin limit,
// or in the wait test the unreachable count and the short limit
inline Barrier make_barrier(int* flags) {
  const bool test = wait_test_on();
  return Barrier{(unsigned*)(flags + 2), flags, test ? kTestSpinLimit : kSpinLimit, test ? 1u : 0u};
}

// Grid-wide barrier on one arrival counter that only grows.  The host zeroes the counter
// before each cooperative launch (zero_barrier); the k-th barrier of the launch is passed
// when the counter reaches k * gridDim.x.  One atomic per block and acquire loads of one
// word: no reset or generation step on the critical path.  Bounded: the wait returns false
// (in every thread) once the error flag is set, by a timeout here or anywhere else.
//
// grid_arrive (thread 0, after a __syncthreads that orders the block's writes before it)
// returns the count that passes this barrier; grid_wait (every thread) waits for it.  Work
// between the two overlaps the other blocks' arrivals.  Consecutive waits must be separated
// by a __syncthreads (the result word is shared).
__device__ __forceinline__ unsigned grid_arrive(const Barrier& b) {
  __threadfence();
  const unsigned arrived = atomicAdd(b.count, 1u) + 1u;
  return (arrived + gridDim.x - 1u) / gridDim.x * gridDim.x + b.extra;
}

__device__ bool grid_wait(const Barrier& b, unsigned target) {
  __shared__ int ok;
  if (threadIdx.x == 0) {
    unsigned long long it = 0;
    for (;;) {
      unsigned c;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(b.count) : "memory");
      if (c >= target) break;
      if ((it & 63ull) == 63ull && *(volatile int*)b.err) break;
      if (++it > b.limit) {
        atomicExch(b.err, 1);
        break;
      }
    }
    __threadfence();
    ok = (*(volatile int*)b.err == 0);
  }
  __syncthreads();
  return ok != 0;
}

__device__ bool grid_sync(const Barrier& b) {
  __syncthreads();
  unsigned target = 0;
  if (threadIdx.x == 0) target = grid_arrive(b);
  return grid_wait(b, target);
}

// zeroes the arrival counter of make_barrier(flags) before a cooperative launch
inline cudaError_t zero_barrier(int* flags, cudaStream_t st) { return cudaMemsetAsync(flags + 2, 0, sizeof(int), st); }

// global -> shared copy of a column-major rows x cols block (leading dimension ld), with 8
// loads in flight per thread before the stores (a plain load->store loop is latency-bound)
__device__ __forceinline__ void stage_in(float* __restrict__ dst, int ldd, const float* __restrict__ src, long long ld,
                                         int rows, int cols) {
  const int nw = blockDim.x / 32, lane = threadIdx.x & 31;
  const int nrb = (rows + 31) / 32, dcol = nw / nrb, drb = nw % nrb;
  int col = (threadIdx.x >> 5) / nrb, rb = (threadIdx.x >> 5) % nrb;
  while (col < cols) {
    float v[8];
    int d[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = 32 * rb + lane;
      const bool in = col < cols && r < rows;
      v[q] = in ? __ldg(src + (size_t)col * ld + r) : 0.f;
      d[q] = in ? col * ldd + r : -1;
      col += dcol;
      rb += drb;
      if (rb >= nrb) { rb -= nrb; ++col; }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (d[q] >= 0) dst[d[q]] = v[q];
  }
}
__device__ __forceinline__ void stage_out(float* __restrict__ dst, long long ld, const float* __restrict__ src, int lds,
                                          int rows, int cols) {
  const int total = rows * cols;
  for (int e = threadIdx.x; e < total; e += blockDim.x) dst[(size_t)(e / rows) * ld + (e % rows)] = src[(size_t)(e / rows) * lds + (e % rows)];
}

struct PanelArgs {
  float* A;
  long long ld;
  int n, k0, jb, R;        // matrix order, first panel column, panel width, rows per block
  int* piv;                // absolute pivot row of each column
  unsigned long long* keys;  // [2][G] tagged pivot candidates (panel_key)
  unsigned long long* crows; // [2][G][jb] candidate rows, tagged words (panel_word)
  unsigned long long* drow;  // [2][jb] diagonal rows, tagged words
  int* singular;           // first singular column + 1, or 0
  unsigned tag0;           // tag of column 0 of this panel (nonzero; see panel_key)
  Barrier bar;             // error word, poll limit and the wait test's offset
};

// A block's pivot candidate for one panel column as one 64-bit word:
//   bits 42-63  tag = (tag0 + column) mod 2^22: which launch and column the word is for;
//   bits 10-41  |value| bits + 1 (0: no finite candidate);
//   bits 0-9    the candidate's row offset inside the block's slab (R <= 1023).
// The rows themselves travel as 64-bit words too (panel_word): the value's bits and the
// full 32-bit tag.  Every word names its column, so no store needs to be ordered before
// another: readers poll the keys, then read the winner's row and re-read any word whose
// tag is not yet the column's.  One round of relaxed stores and polls is the grid barrier
// and the exchange.  The host zeroes keys and rows before each factorisation and numbers
// the panels from 1, so no word is ever mistaken for a later column's.
__device__ __forceinline__ unsigned long long panel_key(unsigned tag, float v, int rowoff) {
  const unsigned long long vk = v >= 0.f ? (unsigned long long)__float_as_uint(v) + 1ull : 0ull;
  return ((unsigned long long)(tag & 0x3FFFFFu) << 42) | (vk << 10) | (unsigned long long)rowoff;
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
constexpr int kMaxKeysPerLane = 8;   // up to 256 panel blocks
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long panel_word(unsigned tag, float v) {
  return ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(v);
}

__device__ __forceinline__ void argmax_merge(float& v, int& i, float ov, int oi) {
  if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}

// The block's candidate for panel column jc: the block argmax of (best, bi), then warp 0
// writes the whole candidate row and its key, and warp 1 the diagonal row k0 + jc if this
// block holds it; no barrier after (every word is tagged).  Rows go out in their state
// after column jc - 1's elimination: in the slab that update is still pending for the
// columns beyond jc, so warps 0 and 1 apply it to their row here (the same fmaf as the
// rest of the slab) and write it back; the other rows get it in the caller's loop, which
// skips the two returned rows (-1: none).
__device__ __forceinline__ void panel_publish(const PanelArgs& a, float* slab, const float* prow, int jc,
                                              bool pending, float best, int bi, float* rv, int* ri, int r0, int nr,
                                              int& done_cand, int& done_diag) {
  const int G = gridDim.x, b = blockIdx.x, jb = a.jb, R = a.R, par = jc & 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned tag = a.tag0 + (unsigned)jc;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    argmax_merge(best, bi, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o));
  if (lane == 0) { rv[warp] = best; ri[warp] = bi; }
  __syncthreads();
  // the block's candidate, found by every warp alike
  float v = lane < kPanelThreads / 32 ? rv[lane] : -1.f;
  int i = lane < kPanelThreads / 32 ? ri[lane] : 0x7fffffff;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    argmax_merge(v, i, __shfl_xor_sync(0xffffffffu, v, o), __shfl_xor_sync(0xffffffffu, i, o));
  const int c = a.k0 + jc;
  const bool has_cand = v >= 0.f;
  const bool has_diag = c >= r0 && c < r0 + nr;
  done_cand = has_cand ? i - r0 : -1;
  done_diag = (has_diag && !(has_cand && i == c)) ? c - r0 : -1;
  // one warp per published row: the update applied and written back, the words out to
  // dst (and to dst2 when the candidate is the diagonal row itself)
  auto put_row = [&](unsigned long long* dst, unsigned long long* dst2, int rr) {
    const float l = pending ? slab[(size_t)(jc - 1) * R + rr] : 0.f;
    for (int jj = lane; jj < jb; jj += 32) {
      float x = slab[(size_t)jj * R + rr];
      if (pending && jj > jc) {
        x = fmaf(-l, prow[jj], x);
        slab[(size_t)jj * R + rr] = x;
      }
      st_relaxed_u64(dst + jj, panel_word(tag, x));
      if (dst2) st_relaxed_u64(dst2 + jj, panel_word(tag, x));
    }
  };
  if (warp == 0) {
    if (has_cand)
      put_row(a.crows + ((size_t)par * G + b) * jb, (has_diag && i == c) ? a.drow + par * jb : nullptr, i - r0);
    if (lane == 0) st_relaxed_u64(a.keys + (size_t)par * G + b, panel_key(tag, v, has_cand ? i - r0 : 0));
  } else if (warp == 1 && done_diag >= 0) {
    put_row(a.drow + par * jb, nullptr, c - r0);
  }
}

// Warp 0: waits (bounded) until every block's key for column j is out, then the pivot
// (largest |value|, first row on ties; the same answer in every block), the pivot row into
// prow and, when this block holds the pivot row, the diagonal row into dsw.  Returns the
// pivot row (absolute), or -1 after a timeout or another block's error.
__device__ int panel_collect(const PanelArgs& a, int j, float* prow, float* dsw, int r0, int nr) {
  const int G = gridDim.x, jb = a.jb, par = j & 1, lane = threadIdx.x & 31;
  const int c = a.k0 + j;
  const unsigned tag = (a.tag0 + (unsigned)j + a.bar.extra) & 0x3FFFFFu;
  float v = -1.f;
  int i = 0x7fffffff, ow = -1;
  // this lane's keys (G <= 32 kMaxKeysPerLane blocks), polled together with relaxed loads
  unsigned long long k[kMaxKeysPerLane];
  unsigned pending = 0;
#pragma unroll
  for (int q = 0; q < kMaxKeysPerLane; ++q)
    if (lane + 32 * q < G) pending |= 1u << q;
  bool ok = true;
  for (unsigned long long it = 0; pending; ++it) {
#pragma unroll
    for (int q = 0; q < kMaxKeysPerLane; ++q)
      if (pending & (1u << q)) k[q] = ld_relaxed_u64(a.keys + (size_t)par * G + lane + 32 * q);
#pragma unroll
    for (int q = 0; q < kMaxKeysPerLane; ++q)
      if ((pending & (1u << q)) && (unsigned)(k[q] >> 42) == tag) pending &= ~(1u << q);
    if (!pending) break;
    if ((it & 63ull) == 63ull && *(volatile int*)a.bar.err) { ok = false; break; }
    if (it > a.bar.limit) {
      atomicExch(a.bar.err, 1);
      ok = false;
      break;
    }
  }
  if (__any_sync(0xffffffffu, !ok)) return -1;
#pragma unroll
  for (int q = 0; q < kMaxKeysPerLane; ++q) {
    const int g = lane + 32 * q;
    if (g >= G) break;
    const unsigned vk = (unsigned)(k[q] >> 10);
    if (vk != 0u) {
      const float gv = __uint_as_float(vk - 1u);
      const int gi = a.k0 + g * a.R + (int)(k[q] & 1023ull);
      if (gv > v || (gv == v && gi < i)) { v = gv; i = gi; ow = g; }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, i, o);
    const int oo = __shfl_xor_sync(0xffffffffu, ow, o);
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; ow = oo; }
  }
  if (!(v >= 0.f) || i < c || i >= a.n || ow < 0) {   // no finite candidate (a NaN column): keep the row
    i = c;
    ow = -1;
    v = 0.f;
  }
  // the rows: every word read until it carries this column's tag (the stores are not
  // ordered with the key's); bounded like the keys
  const unsigned wtag = a.tag0 + (unsigned)j + a.bar.extra;
  const bool mine = i >= r0 && i < r0 + nr && i != c;
  const unsigned long long* src = ow >= 0 ? a.crows + ((size_t)par * G + ow) * jb : a.drow + par * jb;
  // this lane's words of a row (jb <= 128: at most 4), loaded together, stale ones again
  auto fetch = [&](const unsigned long long* p, float* out) -> bool {
    constexpr int kW = kNb / 32;
    unsigned long long w[kW];
    unsigned stale = 0;
#pragma unroll
    for (int q = 0; q < kW; ++q)
      if (lane + 32 * q < jb) stale |= 1u << q;
    for (unsigned long long it = 0; stale; ++it) {
#pragma unroll
      for (int q = 0; q < kW; ++q)
        if (stale & (1u << q)) w[q] = ld_relaxed_u64(p + lane + 32 * q);
#pragma unroll
      for (int q = 0; q < kW; ++q)
        if ((stale & (1u << q)) && (unsigned)(w[q] >> 32) == wtag) stale &= ~(1u << q);
      if (!stale) break;
      if (it > a.bar.limit || ((it & 63ull) == 63ull && *(volatile int*)a.bar.err)) {
        atomicExch(a.bar.err, 1);
        return false;
      }
    }
#pragma unroll
    for (int q = 0; q < kW; ++q)
      if (lane + 32 * q < jb) out[lane + 32 * q] = __uint_as_float((unsigned)w[q]);
    return true;
  };
  ok = fetch(src, prow);
  if (ok && mine) ok = fetch(a.drow + par * jb, dsw);
  if (__any_sync(0xffffffffu, !ok)) return -1;
  if (lane == 0 && blockIdx.x == 0) {
    a.piv[c] = i;
    if (!(v > 0.f) && *a.singular == 0) *a.singular = c + 1;
  }
  return i;
}

// Partial-pivoting LU of the panel's jb columns, rows k0..n-1 spread over the blocks (R rows
// each, kept in shared memory).  Per column: every block publishes its candidate (its key
// last, with release semantics), then polls all blocks' keys; every block finds the same
// pivot, swaps, forms its multipliers and updates the next column first -- enough for the
// next candidate, which is published at once -- and only then updates the rest of its
// rows, while the other blocks publish.
__global__ void __launch_bounds__(kPanelThreads) k_panel_lu(PanelArgs a) {
  extern __shared__ float smem[];
  const int jb = a.jb, R = a.R;
  const int warp = threadIdx.x >> 5;
  float* slab = smem;                       // [jb][R]
  float* prow = smem + (size_t)jb * R;      // [jb] pivot row
  float* dsw = prow + jb;                   // [jb] diagonal row, for the swap
  __shared__ float rv[kPanelThreads / 32];
  __shared__ int ri[kPanelThreads / 32];
  __shared__ int sg_row;
  const int r0 = a.k0 + blockIdx.x * R;
  const int nr = max(0, min(a.n, r0 + R) - r0);
  if (nr > 0) stage_in(slab, R, a.A + (size_t)a.k0 * a.ld + r0, a.ld, nr, jb);
  __syncthreads();
  {
    float best = -1.f;
    int bi = 0x7fffffff;
    for (int r = threadIdx.x; r < nr; r += blockDim.x) argmax_merge(best, bi, fabsf(slab[r]), r0 + r);
    int dc, dd;
    panel_publish(a, slab, prow, 0, false, best, bi, rv, ri, r0, nr, dc, dd);
  }
  for (int j = 0; j < jb; ++j) {
    const int c = a.k0 + j;
    if (warp == 0) {
      const int pi = panel_collect(a, j, prow, dsw, r0, nr);
      if ((threadIdx.x & 31) == 0) sg_row = pi;
    }
    __syncthreads();
    const int prow_i = sg_row;
    if (prow_i < 0) return;
    if (prow_i != c) {
      if (c >= r0 && c < r0 + nr)
        for (int jj = threadIdx.x; jj < jb; jj += blockDim.x) slab[(size_t)jj * R + (c - r0)] = prow[jj];
      if (prow_i >= r0 && prow_i < r0 + nr)
        for (int jj = threadIdx.x; jj < jb; jj += blockDim.x) slab[(size_t)jj * R + (prow_i - r0)] = dsw[jj];
      __syncthreads();
    }
    // multipliers and the next column, with the next column's local argmax on the fly
    const float p = prow[j];
    const bool nxt = (j + 1 < jb);
    float best = -1.f;
    int bi = 0x7fffffff;
    for (int r = threadIdx.x; r < nr; r += blockDim.x) {
      if (r0 + r <= c) continue;
      float* row = slab + r;
      if (p != 0.f) {
        const float l = row[(size_t)j * R] / p;
        row[(size_t)j * R] = l;
        if (nxt) row[(size_t)(j + 1) * R] = fmaf(-l, prow[j + 1], row[(size_t)(j + 1) * R]);
      }
      if (nxt) argmax_merge(best, bi, fabsf(row[(size_t)(j + 1) * R]), r0 + r);
    }
    if (!nxt) break;
    int done_cand, done_diag;
    panel_publish(a, slab, prow, j + 1, p != 0.f, best, bi, rv, ri, r0, nr, done_cand, done_diag);
    // the rest of the rank-1 update (the published rows have theirs), eight loads in flight
    // per thread
    if (p != 0.f) {
      for (int r = threadIdx.x; r < nr; r += blockDim.x) {
        if (r0 + r <= c || r == done_cand || r == done_diag) continue;
        float* row = slab + r;
        const float l = row[(size_t)j * R];
        int jj = j + 2;
        for (; jj + 8 <= jb; jj += 8) {
          float v[8], q[8];
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            v[t] = row[(size_t)(jj + t) * R];
            q[t] = prow[jj + t];
          }
#pragma unroll
          for (int t = 0; t < 8; ++t) row[(size_t)(jj + t) * R] = fmaf(-l, q[t], v[t]);
        }
        for (; jj < jb; ++jj) row[(size_t)jj * R] = fmaf(-l, prow[jj], row[(size_t)jj * R]);
      }
    }
    __syncthreads();
  }
  __syncthreads();
  if (nr > 0) stage_out(a.A + (size_t)a.k0 * a.ld + r0, a.ld, slab, R, nr, jb);
}

// ---- the panel factorisation in one thread-block cluster ---------------------------------
// What bounds a panel is latency: one pivot exchange per column.  Through global memory
// (k_panel_lu, 152 blocks) it costs 3.1 us a column; among the 16 blocks of one cluster the
// candidates travel through distributed shared memory, counted in on mbarriers.
// The rows then have to fit 16 SMs: up to 640 rows of W = 64 columns in a block's registers, so
// 10,240 rows fit; a kNb-column panel is factored W columns at a time (k_panel_next brings the
// second half up to date).  More rows than that go to k_panel_lu.  A column's steps are a chain that
// every warp runs for itself, so the fewer warps share a scheduler the faster: 64 columns take 90 us
// with 10 warps a block (10,240 rows), 77 with 8 (8,192), 69 with 4 (4,096), whatever the cluster's size.
//
// Rows do not move while the sub-panel is factored: each thread tracks the position its rows have
// after the interchanges so far (LAPACK's order); the sub-panel's rows are stored there at
// the end, and k_laswp moves the other columns'.  Pivot choice: largest |value|, lowest position on ties.
// Inside, columns go in groups of kCpGroup.  Per column only the group's columns are touched, a
// thread holding two rows of them: the warps' candidates (redux), the best of them sent by warp 0 to
// every block of the cluster (st.async, which counts its bytes on the receiver's mbarrier), the
// same winner found by every warp, the rank-1 update of the window.  Per group the pivot rows'
// later columns are sent to every block, solved against the group's L (U12), and the columns right
// of the group, held as tiles of 4 rows x 4 columns per thread and chunk, take the rank-8 update: a
// tile reads 4 multipliers and 4 elements of U for 16 products (two full rows per thread: 58 reads
// for 112 products, and this update a fifth of the kernel).
// Measured (one GB300), 64 columns with 10 warps: 112 -> 90 us (one warp's instructions in series
// are what is left); factorisation at n = 10,240: 43.2 -> 22.3 ms with the kernels below.  Not kept: full
// rows in every exchange with a rank-1 update of the whole width per column (2.3 us a column),
// the column's code unrolled (by 8: 108 against 97 us; fetching it takes longer than running
// it), a block barrier and a second search by every warp before the exchange (112 against
// 97 us), a cluster barrier instead of mbarriers (its release waits for the finished columns'
// global stores).
constexpr int kCpMax = 16;                  // blocks per cluster
constexpr int kCpGroup = 8;                 // columns between two updates of the rest
constexpr int kCpW = 64, kCpRows = 2;       // columns of a sub-panel, rows per thread
// threads per block, the fewest that hold a panel: 4,096 rows, 8,192, 10,240 in 16 blocks
constexpr int kCpThreads[] = {128, 256, 320};

struct ClusterPanelArgs {
  float* A;
  long long ld;
  int n, k0, c, w;        // matrix order, first column of the panel, of this sub-panel, its width
  int* piv;
  int* singular;
  int* err;               // set when a wait runs out
  const float* u;         // the rows of U above the sub-panel, (c - k0) x w column-major (k_panel_next)
  int test;               // the wait test: every wait runs out
};
template <int W, int NT> struct ClusterShared {
  static constexpr int RPT = kCpRows, warps = NT / 32;
  static constexpr int R = W - kCpGroup;          // columns right of the first group
  static constexpr int rows_n = RPT * NT;         // rows of a block
  float xch[2][kCpGroup][kCpMax][kCpGroup];       // the blocks' candidate windows, by group parity and column
  float rows[2][kCpGroup][R];                     // the pivot rows' later columns, by group parity
  float u12[2][kCpGroup][R];                      // the same after the solve
  float own[kCpGroup][R];                         // those that this block sends
  float cand[warps][kCpGroup];                    // the warps' candidate windows
  float l[kCpGroup][rows_n];                      // the group's multipliers, 0 where a row takes no update
  float4 turn[2][rows_n];                         // the next group's columns, from tiles to rows
  uint2 head[2][kCpGroup][kCpMax];                // candidates' |value| bits + 1 (0: none) and positions
  uint2 whead[warps];                             // the warps'
  unsigned long long bar[4];                      // mbarriers: a column's candidates (by parity), a group's rows, none (wait test)
  int prow[kCpGroup];                             // the group's k-th pivot row, if it is one of this block's (-1)
  float done[W * RPT * NT];                       // the finished columns
};
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_map(const void* p, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}

__device__ __forceinline__ void cluster_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// 8 bytes into another block's shared memory, counted there
__device__ __forceinline__ void cluster_send(unsigned dst, unsigned v0, unsigned v1, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(dst),
               "r"(v0), "r"(v1), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cluster_send4(unsigned dst, const float4& v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)),
               "r"(bar)
               : "memory");
}
// the lane with the largest key and, among those that have it, the lowest position (distinct
// but for keys of 0)
__device__ __forceinline__ int best_lane(unsigned key, unsigned pos, unsigned& m) {
  constexpr unsigned full = 0xffffffffu;
  m = __reduce_max_sync(full, key);
  unsigned eq = __ballot_sync(full, key == m);
  if ((eq & (eq - 1u)) != 0u && m != 0u) {
    const unsigned p = __reduce_min_sync(full, key == m ? pos : full);
    eq = __ballot_sync(full, key == m && pos == p);
  }
  return __ffs(eq) - 1;
}
__device__ __forceinline__ unsigned cluster_test(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(done)
               : "r"(bar), "r"(parity)
               : "memory");
  return done;
}
// suspends for up to 1 us
__device__ __forceinline__ unsigned cluster_try(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done;
}
// A warp's wait (bounded) for the phase of mbarrier `bar`.  All blocks of a cluster are resident, so it can
// only run out if one of them faults, or in the wait test, where it polls `never` (parity 0: a phase that
// nothing completes) for a short time.  A wait that runs out sets the error word, gives the copies in flight to
// this block time to land (in the wait test they all do) and returns false in the whole warp.
constexpr unsigned kClusterTries = 1u << 21, kClusterTestTries = 1u << 6, kClusterDrain = 1u << 16;
__device__ __forceinline__ bool cluster_wait(unsigned bar, unsigned parity, int* err, unsigned never) {
  const unsigned wb = never ? never : bar, limit = never ? kClusterTestTries : kClusterTries;
  unsigned done = 0u;
  for (int it = 0; it < 4096 && !done; ++it) done = cluster_test(wb, parity);   // (a suspended wait wakes up later)
  for (unsigned it = 0; it < limit && !done; ++it) done = cluster_try(wb, parity);
  if (__all_sync(0xffffffffu, done != 0u)) return true;
  atomicExch(err, 1);
  for (unsigned it = 0; it < kClusterDrain && !cluster_try(bar, parity); ++it) {}
  __syncwarp();
  return false;
}

// A block's rows right of the group, NRB = NT / 64 row blocks of 128: warp w holds the rows 128 (w % NRB) +
// lane + 32 i, i < 4, and of every group's 8 columns the half w / NRB (chunk c: columns 8 (c + 1) +
// 4 (w / NRB) .. + 3).
template <int W> struct PanelTile {
  static constexpr int NCH = W / kCpGroup - 1;
  float4 y[4][NCH];
};
// their rank-kCpGroup update after group g: y -= l u
template <int W, int NT>
__device__ __forceinline__ void panel_update(PanelTile<W>& t, const ClusterShared<W, NT>& sh, int g, int gp, int rb, int cb) {
  constexpr int KS = NT > 256 ? kCpGroup / 2 : kCpGroup;   // multipliers in registers at a time
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int k0 = 0; k0 < kCpGroup; k0 += KS) {
    float l[KS][4];
#pragma unroll
    for (int k = 0; k < KS; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) l[k][i] = -sh.l[k0 + k][128 * rb + lane + 32 * i];
#pragma unroll
    for (int c = 0; c < PanelTile<W>::NCH; ++c)
      if (c >= g)
#pragma unroll
        for (int k = 0; k < KS; ++k) {
          const float4 u = *reinterpret_cast<const float4*>(&sh.u12[gp][k0 + k][8 * c + 4 * cb]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float4& y = t.y[i][c];
            const float2 lo = __ffma2_rn(make_float2(l[k][i], l[k][i]), make_float2(u.x, u.y), make_float2(y.x, y.y));
            const float2 hi = __ffma2_rn(make_float2(l[k][i], l[k][i]), make_float2(u.z, u.w), make_float2(y.z, y.w));
            y = make_float4(lo.x, lo.y, hi.x, hi.y);
          }
        }
  }
}

// One group of columns; x[.][0..kCpGroup) are the rows tid and tid + NT, t what lies right of it.
template <int W, int NT>
__device__ __forceinline__ void panel_group(const ClusterPanelArgs& a, ClusterShared<W, NT>& sh, float (*x)[kCpGroup],
                                            PanelTile<W>& t, int* pos, int g0, unsigned rank, unsigned C, bool& dead) {
  constexpr unsigned full = 0xffffffffu;
  constexpr int B = kCpGroup, R = W - B, RPT = kCpRows, NRB = NT / 64;
  auto off = [&](const void* p) { return (unsigned)((const char*)p - (const char*)&sh); };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cg = a.c + g0, gp = (g0 / B) & 1;
  const int nb = min(B, a.w - g0);
  const unsigned peer = cluster_map(&sh, (unsigned)(lane & 15) < C ? lane & 15 : 0);
  const unsigned never = a.test ? (unsigned)__cvta_generic_to_shared(&sh.bar[3]) : 0u;
  unsigned win = 0u;   // the winners' blocks, 4 bits each
  // one copy of the column's code (unrolled eight times, fetching it took longer than running
  // it): the current column is always x[.][0], and the group's window turns by one per column
#pragma unroll 1
  for (int jj = 0; jj < B; ++jj) {
    if (jj < nb) {
      const int cj = cg + jj, par = jj & 1;
      // this thread's candidate, the warp's
      unsigned key = 0u, mp = full;
      int mq = 0;
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const unsigned v = __float_as_uint(x[q][0]) & 0x7fffffffu;
        const unsigned kq = (pos[q] >= cj) & (v <= 0x7f800000u) ? v + 1u : 0u;   // NaN: no candidate
        const bool take = (kq > key) | ((kq == key) & ((unsigned)pos[q] < mp));
        key = take ? kq : key;
        mp = take ? (unsigned)pos[q] : mp;
        mq = take ? q : mq;
      }
      unsigned m;
      if (lane == best_lane(key, mp, m)) {
#pragma unroll
        for (int v = 0; v < B / 4; ++v) {
          float4 r = make_float4(x[0][4 * v], x[0][4 * v + 1], x[0][4 * v + 2], x[0][4 * v + 3]);
#pragma unroll
          for (int q = 1; q < RPT; ++q)
            if (mq == q) r = make_float4(x[q][4 * v], x[q][4 * v + 1], x[q][4 * v + 2], x[q][4 * v + 3]);
          reinterpret_cast<float4*>(sh.cand[warp])[v] = r;
        }
        sh.whead[warp] = make_uint2(key, mp);
      }
      __syncwarp();
      // warp 0 finds the block's and sends its window and head to every block
      if (warp == 0) {
        asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
        const uint2 hw = lane < NT / 32 ? sh.whead[lane] : make_uint2(0u, full);
        const int wi = best_lane(hw.x, hw.y, m);
        const uint2 hs = make_uint2(m, __shfl_sync(full, hw.y, wi));
        // (after a wait that ran out nothing is sent or armed any more: the phases before may be open)
        if (lane == 0 && !dead) cluster_expect((unsigned)__cvta_generic_to_shared(&sh.bar[par]), C * (B * 4 + 8));
        const int to = lane & 15, h = lane >> 4;
        if (to < (int)C && !dead) {
          const unsigned bar = peer + off(&sh.bar[par]);
          cluster_send4(peer + off(&sh.xch[gp][jj][rank][4 * h]), reinterpret_cast<const float4*>(sh.cand[wi])[h], bar);
          if (h == 0) cluster_send(peer + off(&sh.head[gp][jj][rank]), hs.x, hs.y, bar);
        }
      } else if (!dead) {
        asm volatile("bar.arrive 1, %0;" ::"n"(NT) : "memory");
      } else {
        // no exchange holds this warp back: it waits here, or it would arrive twice in one turn
        asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
      }
      const unsigned bar = (unsigned)__cvta_generic_to_shared(&sh.bar[par]);
      if (!dead) dead = !cluster_wait(bar, (unsigned)((g0 + jj) >> 1) & 1u, a.err, never);
      // the cluster's pivot, found by every warp alike
      const uint2 hd = lane < (int)C ? sh.head[gp][jj][lane] : make_uint2(0u, full);
      const unsigned wb = (unsigned)best_lane(hd.x, hd.y, m) % kCpMax;
      const unsigned p = __shfl_sync(full, hd.y, wb);
      win |= wb << (4 * jj);
      const float* u = sh.xch[gp][jj][wb];
      // no finite candidate (or a wait that ran out): keep the row
      const int pw = m != 0u && !dead && (int)p >= cj && (int)p < a.n ? (int)p : cj;
      const float pv = m > 1u ? u[0] : 0.f;
      if (rank == 0 && tid == 0) {
        a.piv[cj] = pw;
        if (m <= 1u && *a.singular == 0) *a.singular = cj + 1;
      }
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        pos[q] = pos[q] == cj ? pw : pos[q] == pw ? cj : pos[q];
      }
      if (pv != 0.f) {
        float ue[B];
#pragma unroll
        for (int v = 0; v < B / 4; ++v) {
          const float4 uv = reinterpret_cast<const float4*>(u)[v];
          ue[4 * v] = uv.x; ue[4 * v + 1] = uv.y; ue[4 * v + 2] = uv.z; ue[4 * v + 3] = uv.w;
        }
        // the finished columns at the window's end take no update
#pragma unroll
        for (int k = 1; k < B; ++k)
          if (k >= B - jj) ue[k] = 0.f;
        // x / pv as the division rounds it: a reciprocal rounded to nearest, and per row two corrections by
        // the exact residual (P. Markstein, IBM J. Res. Dev. 34, 1990: the first leaves the quotient within
        // an ulp, the second then rounds it correctly), where nothing underflows on the way.  A division per
        // row costs 1.4 ms more of a factorisation at n = 10,240 (23.5 ms).
        const float rp = __frcp_rn(pv), ap = fabsf(pv);
        float l[RPT];
        bool good = ap > 1e-30f && ap < 1e30f;
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          l[q] = x[q][0] * rp;
          good = good && ((fabsf(x[q][0]) > 1e-28f && fabsf(l[q]) > 1e-30f) || x[q][0] == 0.f);
#pragma unroll
          for (int e = 0; e < 2; ++e) l[q] = fmaf(fmaf(-l[q], pv, x[q][0]), rp, l[q]);
        }
        if (!good)
#pragma unroll
          for (int q = 0; q < RPT; ++q) l[q] = x[q][0] / pv;
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          const bool below = pos[q] > cj;
          if (below) x[q][0] = l[q];
#pragma unroll
          for (int k = 1; k < B; ++k)
            if (below) x[q][k] = fmaf(-l[q], ue[k], x[q][k]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const float t = x[q][0];
#pragma unroll
      for (int k = 0; k + 1 < B; ++k) x[q][k] = x[q][k + 1];
      x[q][B - 1] = t;
    }
  }
  const int g = g0 / B, rb = warp % NRB, cb = warp / NRB;
  const bool more = g0 + B < a.w;
  if (more) {
    // which rows the pivots are
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const int e = pos[q] - cg;
      if ((unsigned)e < (unsigned)B) sh.prow[e] = (tid + q * NT) | (g0 << 16);
    }
    if (tid == 0 && !dead) cluster_expect((unsigned)__cvta_generic_to_shared(&sh.bar[2]), B * (R - g0) * 4);
    __syncthreads();
    // their columns right of the group to every block, by the warps that hold them
    const unsigned barb = off(&sh.bar[2]);
    const int mine = sh.prow[lane & 7];
    unsigned todo = __ballot_sync(full, lane < B && (mine >> 16) == g0 && (mine & 0xffff) / 128 == rb);
    while (todo) {
      const int k = __ffs(todo) - 1;
      todo &= todo - 1u;
      const int r = __shfl_sync(full, mine, k) & 0xffff, ri = (r >> 5) & 3;
      if (lane == (r & 31))
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i == ri)
#pragma unroll
            for (int c = 0; c < PanelTile<W>::NCH; ++c) {
              float* o = &sh.own[k][8 * c + 4 * cb];
              asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"((unsigned)__cvta_generic_to_shared(o)),
                           "f"(t.y[i][c].x), "f"(t.y[i][c].y), "f"(t.y[i][c].z), "f"(t.y[i][c].w) : "memory");
            }
      __syncwarp();
      // 8 lanes per destination
      const int c = lane & 7;
      if (!dead && c >= g && c < PanelTile<W>::NCH) {
        const float4 v = *reinterpret_cast<const float4*>(&sh.own[k][8 * c + 4 * cb]);
        for (unsigned to = lane >> 3; to < C; to += 4) {
          const unsigned dst = cluster_map(&sh, to);
          cluster_send4(dst + off(&sh.rows[gp][k][8 * c + 4 * cb]), v, dst + barb);
        }
      }
      __syncwarp();
    }
    // the rows' multipliers: a pivot row of this group takes only the earlier ones, a finished row none
#pragma unroll
    for (int q = 0; q < RPT; ++q)
#pragma unroll
      for (int k = 0; k < B; ++k) sh.l[k][tid + q * NT] = pos[q] - cg > k ? x[q][k] : 0.f;
  }
#pragma unroll
  for (int q = 0; q < RPT; ++q)
#pragma unroll
    for (int k = 0; k < B; ++k) sh.done[((g0 + k) * RPT + q) * NT + tid] = x[q][k];
  if (!more) return;
  const unsigned bar = (unsigned)__cvta_generic_to_shared(&sh.bar[2]);
  if (!dead) dead = !cluster_wait(bar, (unsigned)gp, a.err, never);
  // U12 = L11^-1 A12 of the group, a thread per column; L11 from the pivots' windows
  if (tid >= g0 && tid < R) {
    float uu[B];
#pragma unroll
    for (int k = 0; k < B; ++k) {
      // the k-th pivot's window starts at its own column: its multipliers e < k are at B - k + e
      const float* lk = sh.xch[gp][k][(win >> (4 * k)) & 15u];
      float v = sh.rows[gp][k][tid];
#pragma unroll
      for (int e = 0; e < k; ++e) v = fmaf(-lk[B - k + e], uu[e], v);
      uu[k] = v;
      sh.u12[gp][k][tid] = v;
    }
  }
  __syncthreads();
  panel_update<W, NT>(t, sh, g, gp, rb, cb);
  // the next group's columns to the threads of their rows
#pragma unroll
  for (int c = 0; c < PanelTile<W>::NCH; ++c)
    if (c == g)
#pragma unroll
      for (int i = 0; i < 4; ++i) sh.turn[cb][128 * rb + lane + 32 * i] = t.y[i][c];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const float4 v0 = sh.turn[0][tid + q * NT], v1 = sh.turn[1][tid + q * NT];
    x[q][0] = v0.x; x[q][1] = v0.y; x[q][2] = v0.z; x[q][3] = v0.w;
    x[q][4] = v1.x; x[q][5] = v1.y; x[q][6] = v1.z; x[q][7] = v1.w;
  }
}

template <int W, int NT>
__global__ void __launch_bounds__(NT, 1) k_panel_cluster(const ClusterPanelArgs a) {
  constexpr int RPT = kCpRows, NRB = NT / 64;
  extern __shared__ __align__(16) char cpsm[];
  static_assert(kNb % W == 0 && W % 16 == 0, "whole sub-panels and groups");
  using Sh = ClusterShared<W, NT>;
  static_assert(offsetof(Sh, rows) % 16 == 0 && offsetof(Sh, u12) % 16 == 0 &&
                    offsetof(Sh, own) % 16 == 0 && offsetof(Sh, cand) % 16 == 0 && (W - kCpGroup) % 4 == 0 &&
                    offsetof(Sh, xch) % 16 == 0 && offsetof(Sh, turn) % 16 == 0 && offsetof(Sh, head) % 8 == 0 &&
                    offsetof(Sh, whead) % 8 == 0 && offsetof(Sh, bar) % 8 == 0,
                "vector accesses");
  static_assert(kCpMax <= 16 && kCpGroup == 8 && (W - kCpGroup) / 4 <= 32, "lanes per destination");
  static_assert(W - kCpGroup <= NT, "a thread per column of U12");
  ClusterShared<W, NT>& sh = *reinterpret_cast<ClusterShared<W, NT>*>(cpsm);
  const int tid = threadIdx.x;
  const unsigned rank = cluster_rank(), C = cluster_size();
  const int c = a.c, w = a.w, kp = a.c - a.k0;
  const int row0 = c + (int)rank * (NT * RPT) + tid;   // this thread's rows: row0 + q NT
  static_assert(W == 64 && RPT == 2 && NT % 64 == 0 && sizeof(Sh) <= 227 * 1024, "tiles of 128 rows, two column halves");
  float x[RPT][kCpGroup];
  PanelTile<W> t;
  int pos[RPT];
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int r = row0 + q * NT;
    const bool in = r < a.n;
    pos[q] = in ? r : -1;
#pragma unroll
    for (int k = 0; k < kCpGroup; ++k) x[q][k] = in && k < w ? a.A[(size_t)(c + k) * a.ld + r] : 0.f;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = c + (int)rank * (NT * RPT) + 128 * ((tid >> 5) % NRB) + (tid & 31) + 32 * i;
#pragma unroll
    for (int e = 0; e < PanelTile<W>::NCH; ++e) {
      const int k = 8 * (e + 1) + 4 * ((tid >> 5) / NRB);
      const float* g = a.A + (size_t)(c + k) * a.ld + r;
      t.y[i][e].x = r < a.n && k < w ? g[0] : 0.f;
      t.y[i][e].y = r < a.n && k + 1 < w ? g[a.ld] : 0.f;
      t.y[i][e].z = r < a.n && k + 2 < w ? g[2 * a.ld] : 0.f;
      t.y[i][e].w = r < a.n && k + 3 < w ? g[3 * a.ld] : 0.f;
    }
  }
  if (tid < kCpGroup) sh.prow[tid] = -1;
  if (tid == 0) {
#pragma unroll
    for (int b = 0; b < 4; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(&sh.bar[b])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the rows of U above this sub-panel (k_panel_next)
  if (rank == 0)
    for (int e = tid; e < kp * w; e += NT)
      a.A[(size_t)(c + e / kp) * a.ld + a.k0 + e % kp] = a.u[e];
  cluster_barrier();   // every block runs: its shared memory may be written
  bool dead = false;
#pragma unroll 1
  for (int g0 = 0; g0 < w; g0 += kCpGroup) panel_group<W, NT>(a, sh, x, t, pos, g0, rank, C, dead);
  // every row to the place the interchanges gave it
#pragma unroll 4
  for (int k = 0; k < w; ++k)
#pragma unroll
    for (int q = 0; q < RPT; ++q)
      if (pos[q] >= 0) a.A[(size_t)(c + k) * a.ld + pos[q]] = sh.done[(k * RPT + q) * NT + tid];
  cluster_barrier();   // no block leaves while another may still write to its shared memory
}

// Before a later sub-panel [c, c + w) of a panel: U = L11^-1 A12 for the rows [k0, c) and
// A22 -= L21 U for the rows below, in FP32 on all SMs (kp = c - k0 and w at most 64).  Every block
// solves U for itself (a warp per column, 8 side by side) and updates 64 rows; block 0 keeps U
// in `u` (kp x w), from where the sub-panel's factorisation stores it: in A other blocks still
// read A12.
constexpr int kNextRows = 64, kNextMax = 64, kNextLd = kNextMax + 4;
struct PanelNextShared {
  alignas(16) float L11[kNextMax * kNextMax];     // column-major
  alignas(16) float U[kNextMax][kNextLd];         // [k][column]
  alignas(16) float L21[kNextMax][kNextLd];       // [k][row]
};
__global__ void __launch_bounds__(256) k_panel_next(float* A, long long ld, int n, int k0, int kp, int w, float* u) {
  extern __shared__ __align__(16) char pnsm[];
  PanelNextShared& sh = *reinterpret_cast<PanelNextShared*>(pnsm);
  constexpr unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c = k0 + kp;
  const int r0 = c + blockIdx.x * kNextRows, nr = min(kNextRows, n - r0);
  stage_in(sh.L11, kp, A + (size_t)k0 * ld + k0, ld, kp, kp);
  constexpr int NQ = kNextMax / 8, NL = kNextMax / 32;
  float y[NQ][NL];
#pragma unroll
  for (int t = 0; t < NQ; ++t)
#pragma unroll
    for (int b = 0; b < NL; ++b) {
      const int col = warp + 8 * t, m = 32 * b + lane;
      y[t][b] = col < w && m < kp ? A[(size_t)(c + col) * ld + k0 + m] : 0.f;
    }
  // L21: 64 rows x kp columns, 16 loads in flight per thread
  {
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int e = tid + 256 * i, k = e / kNextRows, r = e % kNextRows;
      v[i] = k < kp && r < nr ? A[(size_t)(k0 + k) * ld + r0 + r] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int e = tid + 256 * i;
      sh.L21[e / kNextRows][e % kNextRows] = v[i];
    }
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < NL; ++b) {
#pragma unroll 4
    for (int il = 0; il < 32; ++il) {
      const int i = 32 * b + il;
      if (i >= kp) break;
      float lc[NL];
#pragma unroll
      for (int e = b; e < NL; ++e) {
        const int m = 32 * e + lane;
        lc[e] = m > i && m < kp ? sh.L11[(size_t)i * kp + m] : 0.f;
      }
#pragma unroll
      for (int t = 0; t < NQ; ++t) {
        const float yi = __shfl_sync(full, y[t][b], il);
#pragma unroll
        for (int e = b; e < NL; ++e) y[t][e] = fmaf(-lc[e], yi, y[t][e]);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < NQ; ++t)
#pragma unroll
    for (int b = 0; b < NL; ++b) {
      const int col = warp + 8 * t, m = 32 * b + lane;
      sh.U[m][col] = y[t][b];
      if (blockIdx.x == 0 && col < w && m < kp) u[(size_t)col * kp + m] = y[t][b];
    }
  __syncthreads();
  // thread (tr, tc) of 16 x 16: rows 4 tr .. + 3, columns 4 tc .. + 3
  const int tr = tid & 15, tc = tid >> 4;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = 4 * tr + i, col = 4 * tc + q;
      acc[i][q] = r < nr && col < w ? A[(size_t)(c + col) * ld + r0 + r] : 0.f;
    }
#pragma unroll 4
  for (int k = 0; k < kp; ++k) {
    const float4 l = *reinterpret_cast<const float4*>(&sh.L21[k][4 * tr]);
    const float4 v = *reinterpret_cast<const float4*>(&sh.U[k][4 * tc]);
    const float le[4] = {l.x, l.y, l.z, l.w}, ve[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(-le[i], ve[q], acc[i][q]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = 4 * tr + i, col = 4 * tc + q;
      if (r < nr && col < w) A[(size_t)(c + col) * ld + r0 + r] = acc[i][q];
    }
}

// The cluster kernels by the rows that they take: block size, shared memory and the largest cluster
// that can be resident on this device (0: none)
struct ClusterPlan {
  const void* kernel = nullptr;
  int threads = 0, blocks = 0;
  size_t smem = 0;
};
// sets the kernel's attributes, once per factorisation that may use it
template <int NT> static int32_t cluster_setup_of(ClusterPlan* p) {
  p->kernel = (const void*)&k_panel_cluster<kCpW, NT>;
  p->threads = NT;
  p->smem = sizeof(ClusterShared<kCpW, NT>);
  p->blocks = 0;
  O3G_CUDA_TRY(cudaFuncSetAttribute(p->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem));
  O3G_CUDA_TRY(cudaFuncSetAttribute(p->kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  for (int c = kCpMax; c >= 1 && p->blocks == 0; c /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = p->smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, p->kernel, &cfg) == cudaSuccess && nc > 0) p->blocks = c;
    else (void)cudaGetLastError();
  }
  return O3G_OK;
}
// those that a matrix of n rows can use (the first that holds a panel is taken)
static int32_t cluster_setup(int n, ClusterPlan (&p)[3]) {
  static_assert(sizeof(kCpThreads) / sizeof(int) == 3, "one setup each");
  O3G_TRY(cluster_setup_of<kCpThreads[0]>(&p[0]));
  if (n > p[0].blocks * kCpThreads[0] * kCpRows) O3G_TRY(cluster_setup_of<kCpThreads[1]>(&p[1]));
  if (n > p[1].blocks * kCpThreads[1] * kCpRows && p[1].kernel) O3G_TRY(cluster_setup_of<kCpThreads[2]>(&p[2]));
  return O3G_OK;
}
// the plan for a panel of m rows, or nothing when it fits none
static ClusterPlan cluster_for(int m, const ClusterPlan (&p)[3]) {
  for (const ClusterPlan& v : p) {
    const int rows = v.threads * kCpRows;
    if (v.kernel == nullptr || v.blocks * rows < m) continue;
    ClusterPlan r = v;
    r.blocks = 1;
    while (r.blocks * rows < m) r.blocks *= 2;
    return r;
  }
  return ClusterPlan();
}
static int32_t launch_cluster_panel(const ClusterPlan& p, ClusterPanelArgs a, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.blocks);
  cfg.blockDim = dim3(p.threads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = p.blocks;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {&a};
  O3G_CUDA_TRY(cudaLaunchKernelExC(&cfg, p.kernel, args));
  note_launch();
  return O3G_OK;
}

// Row interchanges p0..p1-1 (piv) as one gather: the rows they touch are [p0, p1) and the pivot
// rows below, and a row's final value comes from where the interchanges, undone one by one from
// the last to the first, lead back to.  Slot q of 2 np: row p0 + q, or the pivot row piv[p0 + q -
// np] (-1 where that is not below p1; a row named twice is moved twice, to the same effect).
// Every slot walks for itself: np steps of a few instructions on broadcast reads, where one thread
// applying the interchanges in turn took most of 10 us for 64 and 40 us for 512 (k_laswp then:
// 10.5 and 117 us at n = 10,240, now 5.4 and 9 + 13).
__device__ __forceinline__ int2 row_slot(const int* pv, int p0, int np_, int n, int q) {
  int row = q < np_ ? p0 + q : pv[q - np_];
  if (q >= np_ && row < p0 + np_) row = -1;
  int src = row;
#pragma unroll 8
  for (int e = np_ - 1; e >= 0; --e) {
    const int a = p0 + e, b = pv[e];
    src = src == a ? b : src == b ? a : src;
  }
  return make_int2(row, src);
}
// pv[e] = the pivot row of step e; one that is no interchange (or out of range) is the step's own row
__device__ __forceinline__ void stage_pivots(int* pv, const int* piv, int p0, int np_, int n) {
  for (int e = threadIdx.x; e < np_; e += blockDim.x) {
    const int b = piv[p0 + e];
    pv[e] = b < p0 + e || b >= n ? p0 + e : b;
  }
}
// the slots of many interchanges, for k_laswp's blocks to share
constexpr int kSwapInline = 128;   // up to this many, each block finds them itself
__global__ void __launch_bounds__(128) k_row_map(const int* __restrict__ piv, int p0, int np_, int n, int2* map) {
  extern __shared__ int rmsm[];
  stage_pivots(rmsm, piv, p0, np_, n);
  __syncthreads();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < 2 * np_) map[q] = row_slot(rmsm, p0, np_, n, q);
}
// The interchanges on the columns [c0, c1) outside [s0, s1): one warp per column gathers the rows
// that change and scatters them, 8 loads in flight per lane.  Rows that stay are left alone.
// dynamic shared memory for np interchanges: 8 warps' segments of 2 np floats, then the rows,
// their sources (2 np ints each) and the pivots (np)
inline size_t laswp_smem(int np_) { return (size_t)(8 * 2 * np_ + 5 * np_) * 4; }
__global__ void __launch_bounds__(256) k_laswp(float* A, long long ld, int n, int p0, int p1, const int* piv,
                                               const int2* map, int c0, int c1, int s0, int s1) {
  extern __shared__ float lsw[];
  const int np_ = p1 - p0;
  float* segs = lsw;                                         // [8][2 np]
  int* rowof = reinterpret_cast<int*>(segs + 8 * 2 * np_);   // [2 np]
  int* srcof = rowof + 2 * np_;                              // [2 np]
  int* pv = srcof + 2 * np_;                                 // [np]
  __shared__ int nslots;
  if (threadIdx.x == 0) nslots = 0;
  if (!map) stage_pivots(pv, piv, p0, np_, n);
  __syncthreads();
  // (the slots' order does not matter)
  for (int q = threadIdx.x; q < 2 * np_; q += blockDim.x) {
    const int2 m = map ? map[q] : row_slot(pv, p0, np_, n, q);
    if (m.x != m.y) {
      const int at = atomicAdd(&nslots, 1);
      rowof[at] = m.x;
      srcof[at] = m.y;
    }
  }
  __syncthreads();
  const int ns = nslots;
  if (ns == 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int skip = (s1 > s0) ? (s1 - s0) : 0;
  const int ncol = c1 - c0 - skip;
  for (int t = blockIdx.x * 8 + warp; t < ncol; t += gridDim.x * 8) {
    int col = c0 + t;
    if (skip && col >= s0) col += skip;
    float* a = A + (size_t)col * ld;
    float* seg = segs + (size_t)warp * 2 * np_;
    for (int q0 = lane; q0 < ns; q0 += 256) {
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = q0 + 32 * e < ns ? a[srcof[q0 + 32 * e]] : 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (q0 + 32 * e < ns) seg[q0 + 32 * e] = v[e];
    }
    __syncwarp();
    for (int q = lane; q < ns; q += 32) a[rowof[q]] = seg[q];
    __syncwarp();
  }
}

// x <- L^-1 x for a unit lower L (columns of kNb floats in shared memory, zero below row jb; what lies
// above its diagonal is not used), lane l holding rows l + 32 q: steps [32 b0, jb).  Both indices
// into x are constants after unrolling.
__device__ __forceinline__ void unit_lower_solve(float* x, const float* L, int jb, int b0) {
  constexpr int NQ = kNb / 32;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int b = 0; b < NQ; ++b) {
    if (b < b0 || 32 * b >= jb) continue;
#pragma unroll 8
    for (int il = 0; il < 32; ++il) {
      const float* col = L + (size_t)(32 * b + il) * kNb + lane;   // (a column beyond jb is zero)
      const float xi = __shfl_sync(0xffffffffu, x[b], il);
      x[b] = fmaf(lane > il ? -col[32 * b] : 0.f, xi, x[b]);
#pragma unroll
      for (int q = b + 1; q < NQ; ++q) x[q] = fmaf(-col[32 * q], xi, x[q]);
    }
  }
}
// the jb x jb block at src into columns of kNb floats, zero beyond it
__device__ __forceinline__ void stage_block(float* dst, const float* __restrict__ src, long long ld, int jb) {
  if (jb < kNb) {
    for (int e = threadIdx.x; e < kNb * kNb; e += blockDim.x)
      if (e % kNb >= jb || e / kNb >= jb) dst[e] = 0.f;
  }
  stage_in(dst, kNb, src, ld, jb, jb);
}
constexpr size_t kBlockBytes = (size_t)kNb * kNb * sizeof(float);

// B = L^-1 B for a unit lower jb x jb L (column-major at Lp, leading dimension ldl) and the
// ncols columns of B (jb rows at Bp, leading dimension ldb), or, with identity set, B = L^-1: one
// warp per column of B, L in shared memory.  Bound by its chain of jb shuffles and FMAs and by the
// latency of fetching L: 14 us for 384 columns; 24 us with run-time indices into x and an
// integer division per staged element.
__global__ void __launch_bounds__(256) k_trsm_unit_lower(const float* Lp, long long ldl, int jb, float* Bp,
                                                         long long ldb, int ncols, bool identity) {
  extern __shared__ float L[];   // [jb][kNb]
  constexpr int NQ = kNb / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x / 32;
  stage_block(L, Lp, ldl, jb);
  __syncthreads();
  for (int cidx = blockIdx.x * nw + warp; cidx < ncols; cidx += gridDim.x * nw) {
    float* col = Bp + (size_t)cidx * ldb;
    float x[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int m = q * 32 + lane;
      x[q] = identity ? (m == cidx ? 1.f : 0.f) : m < jb ? col[m] : 0.f;
    }
    unit_lower_solve(x, L, jb, identity ? cidx / 32 : 0);
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (q * 32 + lane < jb) col[q * 32 + lane] = x[q];
  }
}

// FP32 products of a 128 x 128 block with 64 columns, 256 threads: thread (tr, tc) of 16 x 16
// takes rows 4 tr .. + 3 and 64 + 4 tr .. + 3 and columns 4 tc .. + 3, summed in k order in packed
// pairs of rows.  Every operand is loaded in one go, 24 16-byte loads in flight per thread: with 8
// single words at a time the kernels spent their time on 12 rounds of memory latency (k_left_gemm
// 26 us, now 10).
static_assert(kNb == 128, "blocks of 128");
constexpr int kProdCols = 64, kProdLd = kNb + 4;
struct ProdShared {
  alignas(16) float A[kNb][kNb];              // [k][row]
  alignas(16) float B[kProdCols][kProdLd];    // [column][k]
};
// rows from rlim on and columns from clim on are zero; column k of the block at a + k lda
__device__ __forceinline__ void prod_load_a(float4 (&v)[16], const float* __restrict__ a, long long lda, int rlim, int clim) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int e = threadIdx.x + 256 * i, k = e >> 5, r = 4 * (e & 31);
    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < clim && r < rlim) v[i] = __ldcg(reinterpret_cast<const float4*>(a + (size_t)k * lda + r));
    if (r + 1 >= rlim) v[i].y = 0.f;
    if (r + 2 >= rlim) v[i].z = 0.f;
    if (r + 3 >= rlim) v[i].w = 0.f;
  }
}
__device__ __forceinline__ void prod_load_b(float4 (&v)[8], const float* __restrict__ b, long long ldb, int clim) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int e = threadIdx.x + 256 * i, c = e >> 5, k = 4 * (e & 31);
    v[i] = c < clim ? __ldcg(reinterpret_cast<const float4*>(b + (size_t)c * ldb + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
__device__ __forceinline__ void prod_store_a(ProdShared& sh, const float4 (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int e = threadIdx.x + 256 * i;
    *reinterpret_cast<float4*>(&sh.A[e >> 5][4 * (e & 31)]) = v[i];
  }
}
__device__ __forceinline__ void prod_store_b(ProdShared& sh, const float4 (&v)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int e = threadIdx.x + 256 * i;
    *reinterpret_cast<float4*>(&sh.B[e >> 5][4 * (e & 31)]) = v[i];
  }
}
// acc[c][2 h + p] += rows (64 h + 4 tr + 2 p, + 1) of column 4 tc + c
__device__ __forceinline__ void prod_add(float2 (&acc)[4][4], const ProdShared& sh) {
  const int tr = threadIdx.x & 15, tc = threadIdx.x >> 4;
#pragma unroll 1
  for (int k0 = 0; k0 < kNb; k0 += 4) {
    float4 b[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) b[c] = *reinterpret_cast<const float4*>(&sh.B[4 * tc + c][k0]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 a0 = *reinterpret_cast<const float4*>(&sh.A[k0 + k][4 * tr]);
      const float4 a1 = *reinterpret_cast<const float4*>(&sh.A[k0 + k][64 + 4 * tr]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float bv = k == 0 ? b[c].x : k == 1 ? b[c].y : k == 2 ? b[c].z : b[c].w;
        const float2 b2 = make_float2(bv, bv);
        acc[c][0] = __ffma2_rn(make_float2(a0.x, a0.y), b2, acc[c][0]);
        acc[c][1] = __ffma2_rn(make_float2(a0.z, a0.w), b2, acc[c][1]);
        acc[c][2] = __ffma2_rn(make_float2(a1.x, a1.y), b2, acc[c][2]);
        acc[c][3] = __ffma2_rn(make_float2(a1.z, a1.w), b2, acc[c][3]);
      }
    }
  }
}

// B = L B in place for ncols columns of kNb rows (16-byte aligned): each block has read its 64
// columns before it writes them
__global__ void __launch_bounds__(256) k_left_gemm(const float* __restrict__ L, float* B, long long ldb, int ncols) {
  extern __shared__ __align__(16) char lgsm[];
  ProdShared& sh = *reinterpret_cast<ProdShared*>(lgsm);
  const int tr = threadIdx.x & 15, tc = threadIdx.x >> 4;
  float4 va[16], vb[8];
  prod_load_a(va, L, kNb, kNb, kNb);
  int c0 = blockIdx.x * kProdCols;
  prod_load_b(vb, B + (size_t)c0 * ldb, ldb, ncols - c0);
  prod_store_a(sh, va);
  for (; c0 < ncols; c0 += gridDim.x * kProdCols) {
    prod_store_b(sh, vb);
    __syncthreads();
    const int next = c0 + gridDim.x * kProdCols;
    if (next < ncols) prod_load_b(vb, B + (size_t)next * ldb, ldb, ncols - next);
    float2 acc[4][4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[c][r] = make_float2(0.f, 0.f);
    prod_add(acc, sh);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int col = c0 + 4 * tc + c;
      if (col >= ncols) break;
      float* o = B + (size_t)col * ldb + 4 * tr;
      *reinterpret_cast<float4*>(o) = make_float4(acc[c][0].x, acc[c][0].y, acc[c][1].x, acc[c][1].y);
      *reinterpret_cast<float4*>(o + 64) = make_float4(acc[c][2].x, acc[c][2].y, acc[c][3].x, acc[c][3].y);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------
// solves with the factors: y = P b (gather), L y = y (unit lower), U x = y (upper)
__global__ void k_permute_to_float(const double* r, const int* perm, float* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = (float)r[perm[i]];
}

// Inverses of the diagonal blocks of the factors.  The solves use blocks of kDb columns: block b
// has its unit lower inverse at dinv + b 2 kDb^2 and its upper one kDb^2 further, both
// column-major with leading dimension kDb.  k_diag_inverses inverts the kNb x kNb blocks on
// their diagonals (one per CUDA block: columns of the identity, solved by one warp each),
// k_diag_merge fills in the blocks beside them.  The other triangles off those blocks are never
// written nor read.
constexpr int kDb = 512;
constexpr int kDbSub = kDb / kNb;
__host__ __device__ inline size_t dinv_floats(int n) { return (size_t)((n + kDb - 1) / kDb) * 2 * kDb * kDb; }
// blockIdx.y: lower and upper; blockIdx.z: every kInvSplit-th column
constexpr int kInvSplit = 4;
__global__ void __launch_bounds__(256) k_diag_inverses(const float* __restrict__ LU, long long ld, int n,
                                                       float* __restrict__ dinv) {
  extern __shared__ float D[];   // [jb][kNb] diagonal block
  constexpr int NQ = kNb / 32;
  const int kb = blockIdx.x, k0 = kb * kNb, jb = min(kNb, n - k0);
  const bool lower = blockIdx.y == 0;
  stage_block(D, LU + (size_t)k0 * ld + k0, ld, jb);
  __syncthreads();
  float* X = dinv + (size_t)(kb / kDbSub) * 2 * kDb * kDb + (size_t)(kb % kDbSub) * kNb * (kDb + 1) +
             (lower ? 0 : (size_t)kDb * kDb);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c = warp * kInvSplit + blockIdx.z; c < jb; c += blockDim.x / 32 * kInvSplit) {
    float x[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) x[q] = (q * 32 + lane == c) ? 1.f : 0.f;
    if (lower) {
      unit_lower_solve(x, D, jb, c / 32);
    } else {
      // U x = e_c, from row c up
#pragma unroll
      for (int b = NQ - 1; b >= 0; --b) {
        if (b > c / 32) continue;
#pragma unroll 4
        for (int il = 31; il >= 0; --il) {
          const int i = 32 * b + il;
          if (i > c) continue;
          const float* col = D + (size_t)i * kNb + lane;
          if (il == lane) x[b] = x[b] / col[32 * b];
          const float xi = __shfl_sync(0xffffffffu, x[b], il);
          x[b] = fmaf(lane < il ? -col[32 * b] : 0.f, xi, x[b]);
#pragma unroll
          for (int q = 0; q < b; ++q) x[q] = fmaf(-col[32 * q], xi, x[q]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int m = q * 32 + lane;
      X[(size_t)c * kDb + m] = m < jb ? x[q] : 0.f;
    }
  }
}

// The kNb x kNb blocks at distance d from the diagonal of every kDb block's inverses (d = 1, 2,
// ... in turn): X_ij = -X_ii sum_{j <= k < i} L_ik X_kj, and for the upper factor
// Y_ij = -Y_ii sum_{i < k <= j} U_ik Y_kj.  blockIdx.y: lower, upper; blockIdx.z: half of the columns.
__global__ void __launch_bounds__(256) k_diag_merge(const float* __restrict__ LU, long long ld, int n, float* dinv,
                                                    int d) {
  extern __shared__ __align__(16) char mgsm[];
  ProdShared& sh = *reinterpret_cast<ProdShared*>(mgsm);
  const int per = kDbSub - d, b = blockIdx.x / per, t = blockIdx.x % per;
  const bool lower = blockIdx.y == 0;
  const int i = lower ? t + d : t, j = lower ? t : t + d;
  const int o = b * kDb;                                   // first row and column of the kDb block
  if (o + kNb * max(i, j) >= n) return;
  float* X = dinv + (size_t)b * 2 * kDb * kDb + (lower ? 0 : (size_t)kDb * kDb);
  float* Xj = X + (size_t)(kNb * j + kProdCols * blockIdx.z) * kDb;   // this block's columns
  const int tr = threadIdx.x & 15, tc = threadIdx.x >> 4;
  float2 acc[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[c][r] = make_float2(0.f, 0.f);
  float4 va[16], vb[8];
  for (int k = lower ? j : i + 1; k <= (lower ? i - 1 : j); ++k) {
    prod_load_a(va, LU + (size_t)(o + kNb * k) * ld + o + kNb * i, ld, n - (o + kNb * i), n - (o + kNb * k));
    prod_load_b(vb, Xj + kNb * k, kDb, kProdCols);
    __syncthreads();
    prod_store_a(sh, va);
    prod_store_b(sh, vb);
    __syncthreads();
    prod_add(acc, sh);
  }
  // (columns of X_ii beyond the matrix hold nothing)
  prod_load_a(va, X + (size_t)kNb * i * (kDb + 1), kDb, kNb, n - (o + kNb * i));
  __syncthreads();
  prod_store_a(sh, va);
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      *reinterpret_cast<float4*>(&sh.B[4 * tc + c][64 * h + 4 * tr]) =
          make_float4(acc[c][2 * h].x, acc[c][2 * h].y, acc[c][2 * h + 1].x, acc[c][2 * h + 1].y);
      acc[c][2 * h] = acc[c][2 * h + 1] = make_float2(0.f, 0.f);
    }
  __syncthreads();
  prod_add(acc, sh);
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<float4*>(Xj + (size_t)(4 * tc + c) * kDb + kNb * i + 64 * h + 4 * tr) =
          make_float4(-acc[c][2 * h].x, -acc[c][2 * h].y, -acc[c][2 * h + 1].x, -acc[c][2 * h + 1].y);
}

struct TrsvArgs {
  const float* LU;
  const float* dinv;
  long long ld;
  int n;
  float* y;     // K right-hand sides (column c at c n), overwritten by the partial updates
  float* out;   // the solutions: each segment, once final
  Barrier bar;
};

// L w = y (LOWER) or U x = w for K right-hand sides, STEP columns at a time.  What bounds it is
// latency: per step the segment is multiplied by its block's inverse (a few rows per CUDA block),
// a grid barrier, the other rows take the segment's columns of the factor (each block its share
// of rows), a grid barrier.  The factor's elements are loaded before the barriers they do not
// depend on.  STEP is kDb: 128 columns a step, every block applying the whole 128 x 128 inverse for
// itself, took 8-10 us a step; 1024 would double the memory of the inverses (n kDb 8 bytes) to
// save a few barriers.  STEP kNb uses the kNb x kNb inverses alone, for systems that the bigger ones
// are too inaccurate for (refine_passes).  A whole solve with 3 refinements, before and after: n = 640 0.44 -> 0.36
// ms, 2,560 0.99 -> 0.56, 10,240 5.41 -> 1.59, 15,360 8.12 -> 2.56; the inverses cost 0.2 ms per factorisation.
constexpr int kTrRows = 64, kTrChunks = kSolveThreads / kTrRows;
constexpr size_t trsv_smem(int K, int step) { return (size_t)K * (step + kSolveThreads) * sizeof(float); }
template <int K, bool LOWER, int STEP>
__global__ void __launch_bounds__(kSolveThreads) k_trsv(TrsvArgs a) {
  static_assert(kDb % STEP == 0 && STEP % kNb == 0, "whole inverses");
  constexpr int kTrCols = STEP / kTrChunks, kColThreads = kSolveThreads / 4;
  extern __shared__ float trsm[];
  float* yd = trsm;                // [K][STEP]
  float* part = trsm + K * STEP;   // [K][kTrChunks][kTrRows]
  const int G = gridDim.x, tid = threadIdx.x, n = a.n;
  const int nblk = (n + STEP - 1) / STEP;
  for (int s = 0; s < nblk; ++s) {
    const int b = LOWER ? s : nblk - 1 - s;
    const int k0 = b * STEP, jb = min(STEP, n - k0);
    const float* D = a.dinv + (size_t)(k0 / kDb) * 2 * kDb * kDb + (size_t)(k0 % kDb) * (kDb + 1) +
                     (LOWER ? 0 : (size_t)kDb * kDb);
    // this block's rows of the update, and their elements for the first kTrRows of them
    const int lo = LOWER ? k0 + jb : 0, hi = LOWER ? n : k0;
    const int share = (hi - lo + G - 1) / G;
    const int i0 = lo + blockIdx.x * share, i1 = min(hi, i0 + share);
    const int r = tid % kTrRows, q = tid / kTrRows;
    float m[kTrCols];
    auto load = [&](int i) {
#pragma unroll
      for (int t = 0; t < kTrCols; ++t) {
        const int col = q * kTrCols + t;
        m[t] = i < i1 && col < jb ? __ldg(a.LU + (size_t)(k0 + col) * a.ld + i) : 0.f;
      }
    };
    load(i0 + r);
    // rows of the block's inverse times the segment: 4 rows at a time, a thread per row and pair
    // of columns
    const int rpb = (jb + G - 1) / G;
    const int d1 = min(jb, (int)(blockIdx.x + 1) * rpb);
    for (int d0 = blockIdx.x * rpb; d0 < d1; d0 += 4) {
      const int row = d0 + (tid & 3);
      float v[K];
#pragma unroll
      for (int c = 0; c < K; ++c) v[c] = 0.f;
#pragma unroll
      for (int h = 0; h < (STEP + kColThreads - 1) / kColThreads; ++h) {
        const int col = (tid >> 2) + h * kColThreads;
        const bool in = row < d1 && col < jb && (LOWER ? col <= row : col >= row);
        const float dv = in ? __ldg(D + (size_t)col * kDb + row) : 0.f;
        if (in)
#pragma unroll
          for (int c = 0; c < K; ++c) v[c] = fmaf(dv, __ldcg(a.y + (size_t)c * n + k0 + col), v[c]);
      }
#pragma unroll
      for (int c = 0; c < K; ++c) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
        if ((tid & 31) < 4) part[(c * 32 + (tid >> 5)) * 4 + (tid & 3)] = v[c];
      }
      __syncthreads();
      if (tid < 4 * K) {
        const int c = tid >> 2, rr = d0 + (tid & 3);
        float t = 0.f;
#pragma unroll 8
        for (int w = 0; w < 32; ++w) t += part[(c * 32 + w) * 4 + (tid & 3)];
        if (rr < d1) __stcg(a.out + (size_t)c * n + k0 + rr, t);
      }
      __syncthreads();
    }
    if (hi <= lo) break;   // the last segment (the same in every block)
    if (!grid_sync(a.bar)) return;
    for (int e = tid; e < K * jb; e += kSolveThreads) {
      const int c = e / jb, k = e - c * jb;
      yd[c * STEP + k] = __ldcg(a.out + (size_t)c * n + k0 + k);
    }
    for (int r0 = i0; r0 < i1; r0 += kTrRows) {
      if (r0 > i0) load(r0 + r);
      __syncthreads();
      float v[K];
#pragma unroll
      for (int c = 0; c < K; ++c) v[c] = 0.f;
#pragma unroll
      for (int t = 0; t < kTrCols; ++t)
#pragma unroll
        for (int c = 0; c < K; ++c) v[c] = fmaf(m[t], q * kTrCols + t < jb ? yd[c * STEP + q * kTrCols + t] : 0.f, v[c]);
#pragma unroll
      for (int c = 0; c < K; ++c) part[(c * kTrChunks + q) * kTrRows + r] = v[c];
      __syncthreads();
      for (int e = tid; e < K * kTrRows; e += kSolveThreads) {
        const int c = e / kTrRows, rr = e % kTrRows;
        if (r0 + rr < i1) {
          float t = 0.f;
#pragma unroll
          for (int w = 0; w < kTrChunks; ++w) t += part[(c * kTrChunks + w) * kTrRows + rr];
          float* yp = a.y + (size_t)c * n + r0 + rr;
          __stcg(yp, __ldcg(yp) - t);
        }
      }
    }
    if (!grid_sync(a.bar)) return;
  }
}

// both solves for K right-hand sides, `step` (kDb or kNb) columns at a time: lower.y -> lower.out =
// upper.y -> upper.out
template <int K, int STEP>
static int32_t launch_trsv(const TrsvArgs& lower, const TrsvArgs& upper, int G, cudaStream_t st) {
  const void* ks[2] = {(const void*)&k_trsv<K, true, STEP>, (const void*)&k_trsv<K, false, STEP>};
  TrsvArgs args[2] = {lower, upper};
  const size_t smem = trsv_smem(K, STEP);
  for (int e = 0; e < 2; ++e) {
    void* av[] = {&args[e]};
    O3G_CUDA_TRY(cudaFuncSetAttribute(ks[e], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    O3G_CUDA_TRY(zero_barrier(lower.bar.err, st));
    O3G_CUDA_TRY(cudaLaunchCooperativeKernel(ks[e], dim3(G), dim3(kSolveThreads), av, smem, st));
  }
  note_launch(2);
  return O3G_OK;
}
template <int K>
static int32_t launch_trsv(int step, const TrsvArgs& lower, const TrsvArgs& upper, int G, cudaStream_t st) {
  return step == kDb ? launch_trsv<K, kDb>(lower, upper, G, st) : launch_trsv<K, kNb>(lower, upper, G, st);
}
static int32_t trsv(int K, int step, const TrsvArgs& lower, const TrsvArgs& upper, int G, cudaStream_t st) {
  switch (K) {
    case 1: return launch_trsv<1>(step, lower, upper, G, st);
    case 2: return launch_trsv<2>(step, lower, upper, G, st);
    case 3: return launch_trsv<3>(step, lower, upper, G, st);
    case 4: return launch_trsv<4>(step, lower, upper, G, st);
    case 5: return launch_trsv<5>(step, lower, upper, G, st);
    case 6: return launch_trsv<6>(step, lower, upper, G, st);
    case 7: return launch_trsv<7>(step, lower, upper, G, st);
    default: return launch_trsv<8>(step, lower, upper, G, st);
  }
}
// The refinement's passes: with the kDb solves, and, for a system that does not reach its tolerance with
// them, once more from the start with the kNb solves (the same solves when n <= kNb).  An explicit
// inverse's error grows with its block's condition: unit lower triangles whose inverses grow to 1e4 over 512
// columns take up to 3 times the refinements or none are enough, where kNb columns converge.
static int refine_passes(int n) { return n > kNb ? 2 : 1; }
static int refine_step(int pass) { return pass == 0 ? kDb : kNb; }
// one block per SM (1024 threads and at most 48 KB each: always resident together)
static int trsv_grid(int num_sms) { return num_sms; }

__global__ void k_axpy_f2d(double* x, const float* d, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] += (double)d[i];
}
__global__ void k_f2d(const float* s, double* d, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) d[i] = (double)s[i];
}
__global__ void k_d2f(const double* s, float* d, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) d[i] = (float)s[i];
}

// ---- FP64-accurate products of the FP32 matrix without the FP64 pipe --------------------
// x (double) is split into xh + xl (floats, ~48 significant bits together).  Each product
// a * xh is formed error-free (p + e, e = fma(a, xh, -p)), a * xl in one fma, and the row
// sum is carried as a double-single pair (hi, lo) with Knuth's two-sum, renormalised every
// 8 columns.  About 10 FP32 instructions per matrix element: the kernel streams the matrix
// at HBM speed, where the same sum on the FP64 pipe is limited by its rate.
constexpr int kMvChunk = 1024;   // columns per block (blockIdx.y)

__global__ void k_split_f64(const double* __restrict__ x, float* xh, float* xl, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double v = x[i];
  const float h = (float)v;
  xh[i] = h;
  xl[i] = (float)(v - (double)h);
}

__device__ __forceinline__ void ds_add_product(float a, float h, float l, float& hi, float& lo) {
  const float p = __fmul_rn(a, h);
  const float e = fmaf(a, h, -p);
  const float s = __fadd_rn(hi, p);
  const float bb = __fsub_rn(s, hi);
  const float t = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(p, bb));
  hi = s;
  lo = fmaf(a, l, __fadd_rn(lo, __fadd_rn(t, e)));
}

// part[cb][i] = sum over the columns of chunk cb of A[i, j] x[j]
__global__ void __launch_bounds__(256) k_matvec_ds(const float* __restrict__ A, long long ld, int n,
                                                   const float* __restrict__ xh, const float* __restrict__ xl,
                                                   double* __restrict__ part) {
  __shared__ float sh[kMvChunk], sl[kMvChunk];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int cb = blockIdx.y;
  const int j0 = cb * kMvChunk, m = min(n - j0, kMvChunk);
  for (int k = threadIdx.x; k < m; k += blockDim.x) { sh[k] = xh[j0 + k]; sl[k] = xl[j0 + k]; }
  __syncthreads();
  if (i >= n) return;
  const float* a = A + (size_t)j0 * ld + i;
  float hi = 0.f, lo = 0.f;
  int k = 0;
  for (; k + 8 <= m; k += 8) {
    float av[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) av[q] = __ldg(a + (size_t)(k + q) * ld);
#pragma unroll
    for (int q = 0; q < 8; ++q) ds_add_product(av[q], sh[k + q], sl[k + q], hi, lo);
    // renormalise: move the bulk of lo into hi (Dekker's fast two-sum, |hi| >= |lo|)
    const float s2 = __fadd_rn(hi, lo);
    lo = __fsub_rn(lo, __fsub_rn(s2, hi));
    hi = s2;
  }
  for (; k < m; ++k) ds_add_product(__ldg(a + (size_t)k * ld), sh[k], sl[k], hi, lo);
  part[(size_t)cb * n + i] = (double)hi + (double)lo;
}

// y = b - sum_cb part (b != null) or y = sum_cb part; per-block sums of y^2 into nrm
__global__ void k_matvec_finish(const double* __restrict__ part, int ncb, int n, const double* __restrict__ b,
                                double* __restrict__ y, double* __restrict__ nrm) {
  __shared__ double s1[8];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double yy = 0.0;
  if (i < n) {
    double s = 0.0;
    for (int k = 0; k < ncb; ++k) s += part[(size_t)k * n + i];
    const double v = b ? b[i] - s : s;
    y[i] = v;
    yy = v * v;
  }
  for (int o = 16; o > 0; o >>= 1) yy += __shfl_xor_sync(0xffffffffu, yy, o);
  if ((threadIdx.x & 31) == 0) s1[threadIdx.x >> 5] = yy;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a1 = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) a1 += s1[w];
    if (nrm) nrm[blockIdx.x] = a1;
  }
}

// finalize_vels of the panel velocities (u = fs + u/(4 pi) in double, ElementBase.h:187-193
// via Surfaces.h:877-887) followed by vels_to_rhs_panels (RHS.h:92-110)
__global__ void k_vels_to_rhs(int np, int nunk, double fx, double fy, double fz, float* pu, float* pv, float* pw,
                              const float* __restrict__ x1x, const float* __restrict__ x1y,
                              const float* __restrict__ x1z, const float* __restrict__ x2x,
                              const float* __restrict__ x2y, const float* __restrict__ x2z,
                              const float* __restrict__ nx, const float* __restrict__ ny,
                              const float* __restrict__ nz, float* rhs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const double factor = 0.25 / 3.14159265358979323846;
  const float u = (float)(fx + (double)pu[i] * factor);
  const float v = (float)(fy + (double)pv[i] * factor);
  const float w = (float)(fz + (double)pw[i] * factor);
  pu[i] = u;
  pv[i] = v;
  pw[i] = w;
  if (nunk == 1) {
    rhs[i] = -(__fadd_rn(__fadd_rn(__fmul_rn(u, nx[i]), __fmul_rn(v, ny[i])), __fmul_rn(w, nz[i])));
    return;
  }
  rhs[(size_t)nunk * i] = -(__fadd_rn(__fadd_rn(__fmul_rn(u, x1x[i]), __fmul_rn(v, x1y[i])), __fmul_rn(w, x1z[i])));
  rhs[(size_t)nunk * i + 1] = -(__fadd_rn(__fadd_rn(__fmul_rn(u, x2x[i]), __fmul_rn(v, x2y[i])), __fmul_rn(w, x2z[i])));
  if (nunk == 3)
    rhs[(size_t)nunk * i + 2] = -(__fadd_rn(__fadd_rn(__fmul_rn(u, nx[i]), __fmul_rn(v, ny[i])), __fmul_rn(w, nz[i])));
}

}  // namespace o3g

extern "C" int32_t o3g_panel_vels_to_rhs(int32_t np, int32_t nunk, const double* fs, float* pu, float* pv, float* pw,
                                         const o3g_surface_t* surf, float* rhs, void* stream) {
  using namespace o3g;
  if (np < 0 || nunk < 1 || nunk > 3 || !surf || surf->np != np || !fs) {
    set_error("o3g_panel_vels_to_rhs: bad sizes or null arguments");
    return O3G_ERR_INVALID_ARG;
  }
  if (np == 0) return O3G_OK;
  if (!pu || !pv || !pw || !rhs || !surf->x1x || !surf->x2x || (nunk != 2 && !surf->nx)) {
    set_error("o3g_panel_vels_to_rhs: null array");
    return O3G_ERR_INVALID_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  k_vels_to_rhs<<<(np + 255) / 256, 256, 0, st>>>(np, nunk, fs[0], fs[1], fs[2], pu, pv, pw, surf->x1x, surf->x1y,
                                                 surf->x1z, surf->x2x, surf->x2y, surf->x2z, surf->nx, surf->ny,
                                                 surf->nz, rhs);
  note_launch();
  O3G_CUDA_TRY(cudaGetLastError());
  return O3G_OK;
}

// ======================================================================================
struct o3g_bem {
  int device = -1;
  int n = 0;
  long long ld = 0;
  float* A = nullptr;     // assembled matrix (kept for residuals)
  float* LU = nullptr;    // factors
  int* piv = nullptr;     // per-column pivot rows
  int* perm = nullptr;    // composed row permutation: (P b)[i] = b[perm[i]]
  float* dinv = nullptr;  // inverses of the diagonal blocks of L and U
  char* scratch = nullptr;
  size_t scratch_bytes = 0;
  int* flags = nullptr;   // [0] barrier error, [1] singular column + 1, [2] barrier arrivals,
                          // [4] tensor-core update error
  float* tcw = nullptr;   // K-major copies of the update's left operand (n x 512)
  bool factored = false;
  int panel_blocks = 0, solve_blocks = 0;
  int bs = 1;             // unknowns per panel: GMRES preconditions with the bs x bs diagonal blocks
};

using namespace o3g;

extern "C" int32_t o3g_bem_size(const o3g_bem_t* h, int64_t* n) {
  if (!h || !n) return O3G_ERR_INVALID_ARG;
  *n = h->n;
  return O3G_OK;
}

static int32_t bem_check(o3g_bem_t* h) {
  if (!h || !h->A) {
    set_error("o3g_bem: null or destroyed handle");
    return O3G_ERR_INVALID_ARG;
  }
  int dev = -1;
  O3G_CUDA_TRY(cudaGetDevice(&dev));
  if (dev != h->device) {
    set_error("o3g_bem: handle belongs to another device");
    return O3G_ERR_STATE;
  }
  return O3G_OK;
}

extern "C" int32_t o3g_bem_create(int64_t n, o3g_bem_t** out) {
  if (!out || n <= 0 || n > (int64_t)200000) {
    set_error("o3g_bem_create: n must be in 1..200000");
    return O3G_ERR_INVALID_ARG;
  }
  *out = nullptr;
  DeviceFacts df;
  O3G_TRY(device_facts(&df));
  o3g_bem_t* h = new o3g_bem_t();
  h->device = df.device;
  h->n = (int)n;
  h->ld = (n + 31) / 32 * 32;
  const size_t mat = (size_t)h->ld * n * sizeof(float);
  cudaError_t e = o3g::dev_alloc((void**)&h->A, mat);
  if (e == cudaSuccess) e = o3g::dev_alloc((void**)&h->LU, mat);
  if (e == cudaSuccess) e = o3g::dev_alloc((void**)&h->piv, n * sizeof(int));
  if (e == cudaSuccess) e = o3g::dev_alloc((void**)&h->perm, n * sizeof(int));
  if (e == cudaSuccess) e = o3g::dev_alloc((void**)&h->flags, 64 * sizeof(int));
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    set_error_cuda("o3g_bem_create: cudaMalloc", e);
    cudaFree(h->A); cudaFree(h->LU); cudaFree(h->piv); cudaFree(h->perm); cudaFree(h->flags); cudaFree(h->dinv);
    delete h;
    return O3G_ERR_ALLOC;
  }
  cudaMemset(h->A, 0, mat);
  *out = h;
  return O3G_OK;
}

extern "C" int32_t o3g_bem_destroy(o3g_bem_t* h) {
  if (!h) return O3G_OK;
  cudaDeviceSynchronize();
  cudaFree(h->A); cudaFree(h->LU); cudaFree(h->piv); cudaFree(h->perm); cudaFree(h->flags); cudaFree(h->scratch);
  cudaFree(h->dinv);
  cudaFree(h->tcw);
  h->A = nullptr;
  delete h;
  return O3G_OK;
}

extern "C" int32_t o3g_bem_matrix(o3g_bem_t* h, float** A, int64_t* ld) {
  O3G_TRY(bem_check(h));
  if (!A || !ld) return O3G_ERR_INVALID_ARG;
  *A = h->A;
  *ld = h->ld;
  h->factored = false;
  return O3G_OK;
}

extern "C" int32_t o3g_bem_set_unknowns_per_panel(o3g_bem_t* h, int32_t bs) {
  O3G_TRY(bem_check(h));
  if (bs < 1 || bs > 3 || h->n % bs != 0) {
    set_error("o3g_bem_set_unknowns_per_panel: bs must be 1..3 and divide n");
    return O3G_ERR_INVALID_ARG;
  }
  h->bs = bs;
  return O3G_OK;
}

extern "C" int32_t o3g_bem_set_block(o3g_bem_t* h, int64_t rstart, int64_t nrows, int64_t cstart, int64_t ncols,
                                     const float* blk, int32_t mem, void* stream) {
  O3G_TRY(bem_check(h));
  if (rstart < 0 || cstart < 0 || nrows < 0 || ncols < 0 || rstart + nrows > h->n || cstart + ncols > h->n ||
      (!blk && nrows * ncols > 0) || (mem != O3G_MEM_HOST && mem != O3G_MEM_DEVICE)) {
    set_error("o3g_bem_set_block: block outside the matrix or bad arguments");
    return O3G_ERR_INVALID_ARG;
  }
  if (nrows == 0 || ncols == 0) return O3G_OK;
  cudaStream_t st = (cudaStream_t)stream;
  O3G_CUDA_TRY(cudaMemcpy2DAsync(h->A + cstart * h->ld + rstart, h->ld * sizeof(float), blk, nrows * sizeof(float),
                                 nrows * sizeof(float), ncols,
                                 mem == O3G_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
  if (mem == O3G_MEM_HOST) O3G_CUDA_TRY(cudaStreamSynchronize(st));
  h->factored = false;
  return O3G_OK;
}

static int32_t bem_scratch(o3g_bem_t* h, size_t bytes) {
  if (h->scratch_bytes >= bytes) return O3G_OK;
  O3G_CUDA_TRY(cudaDeviceSynchronize());
  cudaFree(h->scratch);
  h->scratch = nullptr;
  h->scratch_bytes = 0;
  cudaError_t e = o3g::dev_alloc((void**)&h->scratch, bytes);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    set_error_cuda("o3g_bem: scratch", e);
    return O3G_ERR_ALLOC;
  }
  h->scratch_bytes = bytes;
  return O3G_OK;
}

extern "C" int32_t o3g_bem_factor(o3g_bem_t* h, void* stream) {
  O3G_TRY(bem_check(h));
  cudaStream_t st = (cudaStream_t)stream;
  const int n = h->n;
  const long long ld = h->ld;
  DeviceFacts df;
  O3G_TRY(device_facts(&df));
  // panel kernel: co-resident blocks, each keeping R rows x kNb columns in shared memory
  int per_sm = 0, optin = 0;
  O3G_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, df.device));
  cudaFuncAttributes fa;
  O3G_CUDA_TRY(cudaFuncGetAttributes(&fa, k_panel_lu));
  const size_t max_smem = (size_t)optin - fa.sharedSizeBytes;
  O3G_CUDA_TRY(cudaFuncSetAttribute(k_panel_lu, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem));
  // panels of up to 10,240 rows run in one cluster (k_panel_cluster); this sizes k_panel_lu
  int G = std::min(df.num_sms, 32 * kMaxKeysPerLane);
  int R = (n + G - 1) / G;
  size_t smem = ((size_t)kNb * R + 2 * kNb + 32) * sizeof(float);
  if (smem > max_smem) {
    set_error("o3g_bem_factor: matrix too large for the panel kernel's shared memory");
    return O3G_ERR_INVALID_ARG;
  }
  O3G_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_panel_lu, kPanelThreads, smem));
  if (per_sm < 1) {
    set_error("o3g_bem_factor: panel kernel cannot be resident");
    return O3G_ERR_INVALID_ARG;
  }
  const size_t cand = align_up((2 * (size_t)G + 2 * (size_t)G * kNb + 2 * (size_t)kNb) * sizeof(unsigned long long));
  O3G_TRY(bem_scratch(h, cand + align_up((size_t)kNb * kNb * 4) + align_up(2 * (size_t)kNbOuter * 8) + (1 << 20)));
  Carve cv(h->scratch);
  // keys and tagged rows back to back, zeroed together once per factorisation
  const size_t xwords = 2 * (size_t)G + 2 * (size_t)G * kNb + 2 * (size_t)kNb;
  unsigned long long* keys = cv.take<unsigned long long>(xwords);
  unsigned long long* crows = keys + 2 * (size_t)G;
  unsigned long long* drow = crows + 2 * (size_t)G * kNb;
  O3G_CUDA_TRY(cudaMemsetAsync(h->flags, 0, 64 * sizeof(int), st));
  O3G_CUDA_TRY(cudaMemsetAsync(keys, 0, xwords * sizeof(unsigned long long), st));
  O3G_CUDA_TRY(cudaMemcpy2DAsync(h->LU, ld * sizeof(float), h->A, ld * sizeof(float), n * sizeof(float), n,
                                 cudaMemcpyDeviceToDevice, st));
  KernelTimer& tm = thread_timer();
  tm.begin(st);
  O3G_CUDA_TRY(cudaFuncSetAttribute(k_trsm_unit_lower, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlockBytes));
  O3G_CUDA_TRY(cudaFuncSetAttribute(k_laswp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)laswp_smem(kNbOuter)));
  // C = C - A B on the tensor cores (o3g_tcgemm.cu: tcgen05, TF32 products, FP32 sums; all
  // operands column-major in LU); the error word of its pipeline waits is flags[4]
  if (!h->tcw) {
    const cudaError_t e = o3g::dev_alloc((void**)&h->tcw, tc_gemm_scratch_floats(n, kNbOuter) * sizeof(float));
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      h->tcw = nullptr;
      set_error_cuda("o3g_bem_factor: tensor-core scratch", e);
      return O3G_ERR_ALLOC;
    }
  }
  // the inverses of the diagonal blocks, 4 KB per row: what is only solved by GMRES has no use for them
  if (!h->dinv) {
    const cudaError_t e = o3g::dev_alloc((void**)&h->dinv, dinv_floats(n) * sizeof(float));
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      h->dinv = nullptr;
      set_error_cuda("o3g_bem_factor: diagonal inverses", e);
      return O3G_ERR_ALLOC;
    }
  }
  auto gemm = [&](int m, int nn, int kk, const float* Am, const float* Bm, float* Cm) -> int32_t {
    return tc_gemm_sub(m, nn, kk, Am, ld, Bm, ld, Cm, ld, h->tcw, h->flags + 4, st);
  };
  auto trsm = [&](int k0, int jb, int c0, int ncols) {
    if (ncols <= 0) return;
    int tb = (ncols + 7) / 8;
    if (tb > 4 * df.num_sms) tb = 4 * df.num_sms;
    k_trsm_unit_lower<<<tb, 256, kBlockBytes, st>>>(h->LU + (size_t)k0 * ld + k0, ld, jb, h->LU + (size_t)c0 * ld + k0,
                                                    ld, ncols, false);
    note_launch();
  };
  // the same solve for a wide right-hand side (whole blocks): Linv = L11^-1 once, then B <- Linv B
  // as an FP32 product
  float* linv = cv.take<float>((size_t)kNb * kNb);
  O3G_CUDA_TRY(cudaFuncSetAttribute(k_left_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ProdShared)));
  auto trsm_wide = [&](int k0, int c0, int ncols) {
    k_trsm_unit_lower<<<kNb / 8, 256, kBlockBytes, st>>>(h->LU + (size_t)k0 * ld + k0, ld, kNb, linv, kNb, kNb, true);
    const int lb = std::min((ncols + kProdCols - 1) / kProdCols, 2 * df.num_sms);
    k_left_gemm<<<lb, 256, sizeof(ProdShared), st>>>(linv, h->LU + (size_t)c0 * ld + k0, ld, ncols);
    note_launch(2);
  };
  int2* rowmap = cv.take<int2>(2 * (size_t)kNbOuter);
  auto laswp = [&](int p0, int p1, int c0, int c1, int s0, int s1) {
    const int cnt = (c1 - c0) - (s1 > s0 ? s1 - s0 : 0);
    if (cnt <= 0) return;
    const int lb = std::min((cnt + 7) / 8, 8 * df.num_sms);
    const bool shared_map = p1 - p0 > kSwapInline;
    if (shared_map) {
      k_row_map<<<(2 * (p1 - p0) + 127) / 128, 128, (size_t)(p1 - p0) * sizeof(int), st>>>(h->piv, p0, p1 - p0, n, rowmap);
      note_launch();
    }
    k_laswp<<<lb, 256, laswp_smem(p1 - p0), st>>>(h->LU, ld, n, p0, p1, h->piv, shared_map ? rowmap : nullptr, c0, c1, s0,
                                                  s1);
    note_launch();
  };
  auto at = [&](int r, int c) { return h->LU + (size_t)c * ld + r; };
  ClusterPlan plans[3];
  O3G_TRY(cluster_setup(n, plans));
  O3G_CUDA_TRY(cudaFuncSetAttribute(k_panel_next, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PanelNextShared)));
  static_assert(kNb == 2 * kCpW && kCpW <= kNextMax, "at most one earlier sub-panel");
  // two-level right-looking LU: kNb-column panels inside kNbOuter-column outer panels; the
  // big trailing update of each outer panel has k = kNbOuter
  for (int K0 = 0; K0 < n; K0 += kNbOuter) {
    const int KB = std::min(kNbOuter, n - K0), K1 = K0 + KB;
    for (int k0 = K0; k0 < K1; k0 += kNb) {
      const int jb = std::min(kNb, K1 - k0);
      const int m = n - k0;
      // (the wait test of the grid barriers, o3g_debug_wait_test(1), takes the kernel that polls them)
      ClusterPlan cp;
      if (!wait_test_on() || wait_test_clusters()) cp = cluster_for(m, plans);
      if (cp.kernel) {
        for (int c = k0; c < k0 + jb; c += kCpW) {
          ClusterPanelArgs ca;
          ca.A = h->LU; ca.ld = ld; ca.n = n; ca.k0 = k0; ca.c = c; ca.w = std::min(kCpW, k0 + jb - c);
          ca.piv = h->piv; ca.singular = h->flags + 1; ca.err = h->flags;
          ca.u = linv;
          ca.test = wait_test_clusters() ? 1 : 0;
          if (c > k0) {
            k_panel_next<<<(n - c + kNextRows - 1) / kNextRows, 256, sizeof(PanelNextShared), st>>>(h->LU, ld, n, k0, c - k0,
                                                                                               ca.w, linv);
            note_launch();
          }
          O3G_TRY(launch_cluster_panel(cp, ca, st));
          laswp(c, c + ca.w, K0, K1, c, c + ca.w);
        }
      } else {
        int g = G;
        int r = (m + g - 1) / g;
        if (r < 32) {   // short panels: fewer blocks
          g = (m + 31) / 32;
          r = (m + g - 1) / g;
        }
        PanelArgs pa;
        pa.A = h->LU; pa.ld = ld; pa.n = n; pa.k0 = k0; pa.jb = jb; pa.R = r;
        pa.piv = h->piv; pa.keys = keys; pa.crows = crows; pa.drow = drow;
        pa.singular = h->flags + 1;
        pa.tag0 = (unsigned)(k0 / kNb + 1) << 7;   // panels numbered from 1: zeroed keys never match
        pa.bar = make_barrier(h->flags);
        void* args[] = {&pa};
        const size_t sm = ((size_t)jb * r + 2 * jb + 32) * sizeof(float);
        O3G_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)k_panel_lu, dim3(g), dim3(kPanelThreads), args, sm, st));
        note_launch();
        // interchanges inside the outer panel; the other columns get them once per outer panel
        laswp(k0, k0 + jb, K0, K1, k0, k0 + jb);
      }
      if (k0 + jb < K1) {
        trsm(k0, jb, k0 + jb, K1 - k0 - jb);
        O3G_TRY(gemm(n - k0 - jb, K1 - k0 - jb, jb, at(k0 + jb, k0), at(k0, k0 + jb), at(k0 + jb, k0 + jb)));
      }
    }
    laswp(K0, K1, 0, n, K0, K1);
    if (K1 < n) {
      // U12 = L11^-1 A12 for the KB x KB unit lower L11, block by block
      for (int k0 = K0; k0 < K1; k0 += kNb) {
        trsm_wide(k0, K1, n - K1);   // (K1 < n: the outer panel is whole blocks)
        if (k0 + kNb < K1) O3G_TRY(gemm(K1 - k0 - kNb, n - K1, kNb, at(k0 + kNb, k0), at(k0, K1), at(k0 + kNb, K1)));
      }
      O3G_TRY(gemm(n - K1, n - K1, KB, at(K1, K0), at(K0, K1), at(K1, K1)));
    }
  }
  {
    O3G_CUDA_TRY(cudaFuncSetAttribute(k_diag_inverses, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlockBytes));
    k_diag_inverses<<<dim3((n + kNb - 1) / kNb, 2, kInvSplit), 256, kBlockBytes, st>>>(h->LU, ld, n, h->dinv);
    O3G_CUDA_TRY(cudaFuncSetAttribute(k_diag_merge, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ProdShared)));
    const int nbig = (n + kDb - 1) / kDb;
    note_launch();
    for (int d = 1; d < kDbSub && n > d * kNb; ++d) {
      k_diag_merge<<<dim3(nbig * (kDbSub - d), 2, kNb / kProdCols), 256, sizeof(ProdShared), st>>>(h->LU, ld, n, h->dinv, d);
      note_launch();
    }
  }
  tm.end(st);
  O3G_CUDA_TRY(cudaGetLastError());
  int fl[5] = {0, 0, 0, 0, 0};
  O3G_CUDA_TRY(cudaMemcpyAsync(fl, h->flags, 5 * sizeof(int), cudaMemcpyDeviceToHost, st));
  std::vector<int> piv(n);
  O3G_CUDA_TRY(cudaMemcpyAsync(piv.data(), h->piv, n * sizeof(int), cudaMemcpyDeviceToHost, st));
  O3G_CUDA_TRY(cudaStreamSynchronize(st));
  if (fl[0]) {
    set_error("o3g_bem_factor: a grid barrier or a panel's exchange timed out");
    return O3G_ERR_TIMEOUT;
  }
  if (fl[4]) {
    set_error("o3g_bem_factor: a wait of the tensor-core update timed out");
    return O3G_ERR_TIMEOUT;
  }
  // compose the interchanges into one gather permutation
  std::vector<int> perm(n);
  for (int i = 0; i < n; ++i) perm[i] = i;
  for (int i = 0; i < n; ++i) {
    const int p = piv[i];
    if (p < 0 || p >= n) {
      set_error("o3g_bem_factor: pivot index out of range");
      return O3G_ERR_CUDA;
    }
    std::swap(perm[i], perm[p]);
  }
  O3G_CUDA_TRY(cudaMemcpyAsync(h->perm, perm.data(), n * sizeof(int), cudaMemcpyHostToDevice, st));
  O3G_CUDA_TRY(cudaStreamSynchronize(st));
  if (fl[1]) {
    char msg[128];
    std::snprintf(msg, sizeof(msg), "o3g_bem_factor: zero pivot in column %d", fl[1] - 1);
    set_error(msg);
    return O3G_ERR_SINGULAR;
  }
  h->factored = true;
  return O3G_OK;
}

extern "C" int32_t o3g_bem_solve(o3g_bem_t* h, const float* b, float* x, double* x64, int32_t mem, double tol,
                                 int32_t max_iter, int32_t* iters, double* relres, void* stream) {
  O3G_TRY(bem_check(h));
  if (!h->factored) {
    set_error("o3g_bem_solve: factor the matrix first (o3g_bem_factor)");
    return O3G_ERR_STATE;
  }
  if (!b || (mem != O3G_MEM_HOST && mem != O3G_MEM_DEVICE) || max_iter < 1 || !(tol >= 0.0)) {
    set_error("o3g_bem_solve: bad arguments");
    return O3G_ERR_INVALID_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int n = h->n;
  const long long ld = h->ld;
  DeviceFacts df;
  O3G_TRY(device_facts(&df));
  const int ncb = (n + kMvChunk - 1) / kMvChunk;
  const int nrb = (n + 255) / 256;
  const size_t need = align_up((size_t)n * 8) * 3 + align_up((size_t)n * 4) * 5 + align_up((size_t)ncb * n * 8) +
                      align_up((size_t)nrb * 16);
  O3G_TRY(bem_scratch(h, need));
  Carve cv(h->scratch);
  double* bd = cv.take<double>(n);
  double* xd = cv.take<double>(n);
  double* rd = cv.take<double>(n);
  float* bf = cv.take<float>(n);
  float* y = cv.take<float>(n);
  float* xf = cv.take<float>(n);
  float* xh = cv.take<float>(n);
  float* xl = cv.take<float>(n);
  double* part = cv.take<double>((size_t)ncb * n);
  double* nrm = cv.take<double>(2 * (size_t)nrb);
  O3G_CUDA_TRY(cudaMemcpyAsync(bf, b, (size_t)n * 4, mem == O3G_MEM_HOST ? cudaMemcpyHostToDevice
                                                                           : cudaMemcpyDeviceToDevice, st));
  k_f2d<<<nrb, 256, 0, st>>>(bf, bd, n);
  O3G_CUDA_TRY(cudaMemsetAsync(xd, 0, (size_t)n * 8, st));
  O3G_CUDA_TRY(cudaMemcpyAsync(rd, bd, (size_t)n * 8, cudaMemcpyDeviceToDevice, st));
  O3G_CUDA_TRY(cudaMemsetAsync(h->flags, 0, 4 * sizeof(int), st));
  const int G = trsv_grid(df.num_sms);
  // L w = P r (y -> w; xh is free between the products), then U y = w (w -> y)
  TrsvArgs ta, tb;
  ta.LU = h->LU; ta.dinv = h->dinv; ta.ld = ld; ta.n = n; ta.y = y; ta.out = xh;
  ta.bar = make_barrier(h->flags);
  tb = ta;
  tb.y = xh; tb.out = y;
  std::vector<double> hn((size_t)nrb);
  double rel = 1.0, bnorm = 0.0;
  int it = 0;
  KernelTimer& tm = thread_timer();
  tm.begin(st);
  for (int pass = 0; pass < refine_passes(n); ++pass) {
    if (pass > 0) O3G_CUDA_TRY(cudaMemsetAsync(xd, 0, (size_t)n * 8, st));
    for (it = 0; it <= max_iter; ++it) {
      // r = b - A x in FP64-accurate double-single arithmetic (r = b at x = 0)
      if (it > 0) {
        k_split_f64<<<nrb, 256, 0, st>>>(xd, xh, xl, n);
        k_matvec_ds<<<dim3(nrb, ncb), 256, 0, st>>>(h->A, ld, n, xh, xl, part);
        note_launch(2);
      }
      k_matvec_finish<<<nrb, 256, 0, st>>>(part, it > 0 ? ncb : 0, n, bd, rd, nrm);
      note_launch();
      O3G_CUDA_TRY(cudaMemcpyAsync(hn.data(), nrm, (size_t)nrb * 8, cudaMemcpyDeviceToHost, st));
      O3G_CUDA_TRY(cudaStreamSynchronize(st));
      double rr = 0.0;
      for (int k = 0; k < nrb; ++k) rr += hn[k];
      if (it == 0) bnorm = std::sqrt(rr);
      rel = bnorm > 0.0 ? std::sqrt(rr) / bnorm : std::sqrt(rr);
      if (rel <= tol || it == max_iter || (!std::isfinite(rel) && pass + 1 < refine_passes(n))) break;
      k_permute_to_float<<<nrb, 256, 0, st>>>(rd, h->perm, y, n);
      O3G_TRY(trsv(1, refine_step(pass), ta, tb, G, st));
      k_axpy_f2d<<<nrb, 256, 0, st>>>(xd, y, n);
      note_launch(2);
    }
    if (rel <= tol) break;
  }
  tm.end(st);
  int fl = 0;
  O3G_CUDA_TRY(cudaMemcpyAsync(&fl, h->flags, sizeof(int), cudaMemcpyDeviceToHost, st));
  k_d2f<<<nrb, 256, 0, st>>>(xd, xf, n);
  note_launch();
  if (x)
    O3G_CUDA_TRY(cudaMemcpyAsync(x, xf, (size_t)n * 4, mem == O3G_MEM_HOST ? cudaMemcpyDeviceToHost
                                                                            : cudaMemcpyDeviceToDevice, st));
  if (x64)
    O3G_CUDA_TRY(cudaMemcpyAsync(x64, xd, (size_t)n * 8, mem == O3G_MEM_HOST ? cudaMemcpyDeviceToHost
                                                                              : cudaMemcpyDeviceToDevice, st));
  O3G_CUDA_TRY(cudaStreamSynchronize(st));
  if (iters) *iters = it;
  if (relres) *relres = rel;
  if (fl) {
    set_error("o3g_bem_solve: a grid barrier timed out");
    return O3G_ERR_TIMEOUT;
  }
  if (!(rel <= tol)) {
    char msg[160];
    std::snprintf(msg, sizeof(msg), "o3g_bem_solve: relative residual %.3e after %d refinements (tol %.1e)", rel, it,
                  tol);
    set_error(msg);
    return O3G_ERR_NOT_CONVERGED;
  }
  return O3G_OK;
}

// ---- the Krylov bases' FP64 operations (Gram-Schmidt, norms, updates), sums in a fixed order
namespace o3g {
constexpr int kKrylovRows = 4096;   // rows per block of the reductions

// part[b kc + j] = sum over the rows [b R, b R + R) of V[j n + i] w[i], j < kc
__global__ void __launch_bounds__(256) k_kry_dots(const double* __restrict__ V, int n, int kc,
                                                  const double* __restrict__ w, double* __restrict__ part) {
  __shared__ double red[8];
  const int r0 = blockIdx.x * kKrylovRows, r1 = min(n, r0 + kKrylovRows);
  for (int j = 0; j < kc; ++j) {
    double s = 0.0;
    for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) s = fma(V[(size_t)j * n + i], w[i], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      double a = 0.0;
      for (int q = 0; q < (int)(blockDim.x >> 5); ++q) a += red[q];
      part[(size_t)blockIdx.x * kc + j] = a;
    }
    __syncthreads();
  }
}

// h[j] = sum over the nb blocks, in block order, of part[b kc + j]
__global__ void k_kry_sum(const double* __restrict__ part, int nb, int kc, double* __restrict__ h) {
  for (int j = threadIdx.x; j < kc; j += blockDim.x) {
    double a = 0.0;
    for (int b = 0; b < nb; ++b) a += part[(size_t)b * kc + j];
    h[j] = a;
  }
}

// y[i] += alpha sum_j V[j n + i] h[j], kc <= 512
__global__ void __launch_bounds__(256) k_kry_update(const double* __restrict__ V, int n, int kc,
                                                    const double* __restrict__ h, double alpha, double* y) {
  __shared__ double hs[512];
  for (int j = threadIdx.x; j < kc; j += blockDim.x) hs[j] = h[j];
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
  for (int j = 0; j < kc; ++j) s = fma(V[(size_t)j * n + i], hs[j], s);
  y[i] = fma(alpha, s, y[i]);
}

__global__ void k_kry_scale(double* w, int n, double s) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) w[i] *= s;
}

// Block-Jacobi preconditioner of GMRES: the inverses (FP64) of the BS x BS diagonal blocks
// of A, one per panel (the panel's self-influence, Coefficients.h:414-436, when the blocks
// are surfaces on themselves).  A block that is singular or not finite gets the identity.
// Minv[p] is row-major.  BS is a template argument so the blocks stay in registers.
template <int BS>
__global__ void k_block_inv(const float* __restrict__ A, long long ld, int nb, double* __restrict__ Minv) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nb) return;
  double a[3][3] = {{1.0, 0.0, 0.0}, {0.0, 1.0, 0.0}, {0.0, 0.0, 1.0}};
  const size_t o = (size_t)p * BS;
#pragma unroll
  for (int r = 0; r < BS; ++r)
#pragma unroll
    for (int c = 0; c < BS; ++c) a[r][c] = (double)A[(o + c) * ld + o + r];
  double inv[3][3] = {{1.0, 0.0, 0.0}, {0.0, 1.0, 0.0}, {0.0, 0.0, 1.0}};
  // cofactors of the 3 x 3 (a 2 x 2 block sits in the leading corner of an identity, so
  // the same formula serves)
  const double c00 = a[1][1] * a[2][2] - a[1][2] * a[2][1];
  const double c01 = a[1][2] * a[2][0] - a[1][0] * a[2][2];
  const double c02 = a[1][0] * a[2][1] - a[1][1] * a[2][0];
  const double det = a[0][0] * c00 + a[0][1] * c01 + a[0][2] * c02;
  if (det != 0.0 && isfinite(det)) {
    const double id = 1.0 / det;
    inv[0][0] = c00 * id;
    inv[1][0] = c01 * id;
    inv[2][0] = c02 * id;
    inv[0][1] = (a[0][2] * a[2][1] - a[0][1] * a[2][2]) * id;
    inv[1][1] = (a[0][0] * a[2][2] - a[0][2] * a[2][0]) * id;
    inv[2][1] = (a[0][1] * a[2][0] - a[0][0] * a[2][1]) * id;
    inv[0][2] = (a[0][1] * a[1][2] - a[0][2] * a[1][1]) * id;
    inv[1][2] = (a[0][2] * a[1][0] - a[0][0] * a[1][2]) * id;
    inv[2][2] = (a[0][0] * a[1][1] - a[0][1] * a[1][0]) * id;
  }
#pragma unroll
  for (int r = 0; r < BS; ++r)
#pragma unroll
    for (int c = 0; c < BS; ++c) Minv[(size_t)p * BS * BS + r * BS + c] = inv[r][c];
}
// out = M^-1 in (acc = 0) or out += M^-1 in (acc = 1)
template <int BS>
__global__ void k_block_apply(const double* __restrict__ Minv, int nb, const double* __restrict__ in,
                              double* __restrict__ out, int acc) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nb) return;
  const double* x = in + (size_t)p * BS;
  double* y = out + (size_t)p * BS;
  const double* M = Minv + (size_t)p * BS * BS;
  double v[BS];
#pragma unroll
  for (int c = 0; c < BS; ++c) v[c] = x[c];
#pragma unroll
  for (int r = 0; r < BS; ++r) {
    double t = 0.0;
#pragma unroll
    for (int c = 0; c < BS; ++c) t += M[r * BS + c] * v[c];
    y[r] = acc ? y[r] + t : t;
  }
}
// launches for the unknowns per panel (2 or 3)
static void block_inv(const float* A, long long ld, int nb, int bs, double* Minv, cudaStream_t st) {
  const int g = (nb + 255) / 256;
  if (bs == 2) k_block_inv<2><<<g, 256, 0, st>>>(A, ld, nb, Minv);
  else         k_block_inv<3><<<g, 256, 0, st>>>(A, ld, nb, Minv);
  note_launch();
}
static void block_apply(const double* Minv, int nb, int bs, const double* in, double* out, int acc,
                        cudaStream_t st) {
  const int g = (nb + 255) / 256;
  if (bs == 2) k_block_apply<2><<<g, 256, 0, st>>>(Minv, nb, in, out, acc);
  else         k_block_apply<3><<<g, 256, 0, st>>>(Minv, nb, in, out, acc);
  note_launch();
}

namespace {
// one classical Gram-Schmidt pass: hp = V^T w (kc columns), w -= V hp
void gs_pass(const double* V, int n, int kc, double* w, double* hp, double* part, cudaStream_t st) {
  const int nb = (n + kKrylovRows - 1) / kKrylovRows;
  k_kry_dots<<<nb, 256, 0, st>>>(V, n, kc, w, part);
  k_kry_sum<<<1, 256, 0, st>>>(part, nb, kc, hp);
  k_kry_update<<<(n + 255) / 256, 256, 0, st>>>(V, n, kc, hp, -1.0, w);
  note_launch(3);
}
// per-block partial sums of w^2 into part (nb of them), summed on the host in order
void norm_partials(const double* w, int n, double* part, cudaStream_t st) {
  k_kry_dots<<<(n + kKrylovRows - 1) / kKrylovRows, 256, 0, st>>>(w, n, 1, w, part);
  note_launch();
}
double host_sum(const std::vector<double>& v) {
  double a = 0.0;
  for (double x : v) a += x;
  return a;
}
}  // namespace
}  // namespace o3g

// ---- GMRES: the reference's solver (Eigen GMRES, BEM.h:182-202) ----------------------------
// Restarted GMRES(m) on the unfactored FP32 matrix: FP64 Krylov vectors, classical
// Gram-Schmidt with one reorthogonalisation (k_kry_dots / k_kry_update on the n x (k+1)
// basis, sums in a fixed order), Givens
// rotations of the small Hessenberg matrix on the host, FP64-accurate matrix products
// (k_matvec_ds).  The true residual ||b - A x|| / ||b|| (BEM.h:227-230) is recomputed at
// every restart and decides convergence.  The vortex-sheet rows of the matrix have a zero
// diagonal (Coefficients.h:414-436), where a Jacobi preconditioner is the identity; with the
// unknowns per panel set (o3g_bem_set_unknowns_per_panel) GMRES is right-preconditioned by
// the inverses of the panels' diagonal blocks (A M^-1 u = b, x = M^-1 u), which keeps the
// residual the system's own.
extern "C" int32_t o3g_bem_solve_gmres(o3g_bem_t* h, const float* b, float* x, double* x64, int32_t mem, double tol,
                                       int32_t max_iter, int32_t restart, int32_t* iters, double* relres,
                                       void* stream) {
  O3G_TRY(bem_check(h));
  if (!b || (mem != O3G_MEM_HOST && mem != O3G_MEM_DEVICE) || max_iter < 1 || restart < 1 || restart > 500 ||
      !(tol >= 0.0)) {
    set_error("o3g_bem_solve_gmres: bad arguments (max_iter >= 1, restart 1..500, tol >= 0)");
    return O3G_ERR_INVALID_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int n = h->n;
  const long long ld = h->ld;
  const int m = std::min(restart, max_iter);
  const int ncb = (n + kMvChunk - 1) / kMvChunk;
  const int nrb = (n + 255) / 256;
  const int nkb = (n + kKrylovRows - 1) / kKrylovRows;
  const int bs = h->bs, npb = n / bs;
  const bool pre = bs > 1;
  const size_t need = align_up((size_t)(m + 1) * n * 8) + 2 * align_up((size_t)n * 8) + 4 * align_up((size_t)n * 4) +
                      align_up((size_t)ncb * n * 8) + align_up((size_t)nrb * 8) + align_up((size_t)2 * (m + 1) * 8) +
                      2 * align_up((size_t)nkb * (m + 1) * 8) + align_up((size_t)n * bs * 8) + align_up((size_t)n * 8);
  O3G_TRY(bem_scratch(h, need));
  Carve cv(h->scratch);
  double* V = cv.take<double>((size_t)(m + 1) * n);
  double* bd = cv.take<double>(n);
  double* xd = cv.take<double>(n);
  double* Minv = cv.take<double>((size_t)n * bs);   // the diagonal blocks' inverses (pre)
  double* zd = cv.take<double>(n);                  // M^-1 v, and V y before M^-1 (pre)
  if (pre) block_inv(h->A, ld, npb, bs, Minv, st);
  float* bf = cv.take<float>(n);
  float* xf = cv.take<float>(n);
  float* xh = cv.take<float>(n);
  float* xl = cv.take<float>(n);
  double* part = cv.take<double>((size_t)ncb * n);
  double* nrm = cv.take<double>(nrb);
  double* hd = cv.take<double>(2 * (size_t)(m + 1));
  double* kpart = cv.take<double>((size_t)nkb * (m + 1));
  double* npart = cv.take<double>((size_t)nkb * (m + 1));
  std::vector<double> hnp((size_t)nkb);
  O3G_CUDA_TRY(cudaMemcpyAsync(bf, b, (size_t)n * 4, mem == O3G_MEM_HOST ? cudaMemcpyHostToDevice
                                                                           : cudaMemcpyDeviceToDevice, st));
  k_f2d<<<nrb, 256, 0, st>>>(bf, bd, n);
  note_launch();
  O3G_CUDA_TRY(cudaMemsetAsync(xd, 0, (size_t)n * 8, st));
  std::vector<double> hn((size_t)nrb);
  // y = b - A xin (bin given) or y = A xin; the squared norm of y when asked (synchronises)
  auto matvec = [&](const double* xin, const double* bin, double* yout, double* norm2) -> int32_t {
    int nc = 0;
    if (xin) {
      k_split_f64<<<nrb, 256, 0, st>>>(xin, xh, xl, n);
      k_matvec_ds<<<dim3(nrb, ncb), 256, 0, st>>>(h->A, ld, n, xh, xl, part);
      note_launch(2);
      nc = ncb;
    }
    k_matvec_finish<<<nrb, 256, 0, st>>>(part, nc, n, bin, yout, nrm);
    note_launch();
    O3G_CUDA_TRY(cudaGetLastError());
    if (norm2) {
      O3G_CUDA_TRY(cudaMemcpyAsync(hn.data(), nrm, (size_t)nrb * 8, cudaMemcpyDeviceToHost, st));
      O3G_CUDA_TRY(cudaStreamSynchronize(st));
      double s2 = 0.0;
      for (int k = 0; k < nrb; ++k) s2 += hn[k];
      *norm2 = s2;
    }
    return O3G_OK;
  };
  double bb = 0.0;
  O3G_TRY(matvec(nullptr, bd, V, &bb));           // V0 = b, ||b||^2
  const double bnorm = std::sqrt(bb);
  int total = 0;
  double rel = 0.0;
  KernelTimer& tm = thread_timer();
  tm.begin(st);
  if (bnorm > 0.0) {
    std::vector<double> H((size_t)(m + 1) * m, 0.0), cs(m), sn(m), g(m + 1), y(m), hc(2 * (size_t)(m + 1));
    auto Hat = [&](int i, int k) -> double& { return H[(size_t)k * (m + 1) + i]; };
    for (;;) {
      double rr = 0.0;
      O3G_TRY(matvec(total > 0 ? xd : nullptr, bd, V, &rr));   // V0 = r = b - A x
      rel = std::sqrt(rr) / bnorm;
      if (rel <= tol || total >= max_iter) break;
      const double beta = std::sqrt(rr);
      k_kry_scale<<<nrb, 256, 0, st>>>(V, n, 1.0 / beta);
      note_launch();
      std::fill(g.begin(), g.end(), 0.0);
      g[0] = beta;
      int k = 0;
      for (; k < m && total < max_iter;) {
        double* vk = V + (size_t)k * n;
        double* w = V + (size_t)(k + 1) * n;
        if (pre) {
          // right preconditioning: w = A M^-1 v_k, so the residual stays the system's own
          block_apply(Minv, npb, bs, vk, zd, 0, st);
          O3G_TRY(matvec(zd, nullptr, w, nullptr));
        } else {
          O3G_TRY(matvec(vk, nullptr, w, nullptr));
        }
        // classical Gram-Schmidt, twice
        for (int pass = 0; pass < 2; ++pass) gs_pass(V, n, k + 1, w, hd + (size_t)pass * (m + 1), kpart, st);
        norm_partials(w, n, npart, st);
        O3G_CUDA_TRY(cudaMemcpyAsync(hc.data(), hd, 2 * (size_t)(m + 1) * 8, cudaMemcpyDeviceToHost, st));
        O3G_CUDA_TRY(cudaMemcpyAsync(hnp.data(), npart, (size_t)nkb * 8, cudaMemcpyDeviceToHost, st));
        O3G_CUDA_TRY(cudaStreamSynchronize(st));
        const double wn = std::sqrt(host_sum(hnp));
        for (int i = 0; i <= k; ++i) Hat(i, k) = hc[i] + hc[(size_t)(m + 1) + i];
        Hat(k + 1, k) = wn;
        if (wn > 0.0) {
          k_kry_scale<<<nrb, 256, 0, st>>>(w, n, 1.0 / wn);
          note_launch();
        }
        // previous rotations, then a new one that zeroes H(k+1, k)
        for (int i = 0; i < k; ++i) {
          const double a = Hat(i, k), c = Hat(i + 1, k);
          Hat(i, k) = cs[i] * a + sn[i] * c;
          Hat(i + 1, k) = -sn[i] * a + cs[i] * c;
        }
        const double dd = std::hypot(Hat(k, k), Hat(k + 1, k));
        cs[k] = dd > 0.0 ? Hat(k, k) / dd : 1.0;
        sn[k] = dd > 0.0 ? Hat(k + 1, k) / dd : 0.0;
        Hat(k, k) = dd;
        Hat(k + 1, k) = 0.0;
        g[k + 1] = -sn[k] * g[k];
        g[k] = cs[k] * g[k];
        ++k;
        ++total;
        if (std::fabs(g[k]) <= 0.5 * tol * bnorm || wn == 0.0) break;
      }
      // x += V y with H(0:k, 0:k) y = g(0:k)
      for (int i = k - 1; i >= 0; --i) {
        double sacc = g[i];
        for (int j = i + 1; j < k; ++j) sacc -= Hat(i, j) * y[j];
        y[i] = Hat(i, i) != 0.0 ? sacc / Hat(i, i) : 0.0;
      }
      O3G_CUDA_TRY(cudaMemcpyAsync(hd, y.data(), (size_t)k * 8, cudaMemcpyHostToDevice, st));
      if (pre) {
        // x += M^-1 (V y)
        O3G_CUDA_TRY(cudaMemsetAsync(zd, 0, (size_t)n * 8, st));
        k_kry_update<<<nrb, 256, 0, st>>>(V, n, k, hd, 1.0, zd);
        note_launch();
        block_apply(Minv, npb, bs, zd, xd, 1, st);
      } else {
        k_kry_update<<<nrb, 256, 0, st>>>(V, n, k, hd, 1.0, xd);
        note_launch();
      }
    }
  }
  tm.end(st);
  k_d2f<<<nrb, 256, 0, st>>>(xd, xf, n);
  note_launch();
  if (x)
    O3G_CUDA_TRY(cudaMemcpyAsync(x, xf, (size_t)n * 4, mem == O3G_MEM_HOST ? cudaMemcpyDeviceToHost
                                                                            : cudaMemcpyDeviceToDevice, st));
  if (x64)
    O3G_CUDA_TRY(cudaMemcpyAsync(x64, xd, (size_t)n * 8, mem == O3G_MEM_HOST ? cudaMemcpyDeviceToHost
                                                                              : cudaMemcpyDeviceToDevice, st));
  O3G_CUDA_TRY(cudaStreamSynchronize(st));
  if (iters) *iters = total;
  if (relres) *relres = rel;
  if (!(rel <= tol)) {
    char msg[160];
    std::snprintf(msg, sizeof(msg), "o3g_bem_solve_gmres: relative residual %.3e after %d iterations (tol %.1e)", rel,
                  total, tol);
    set_error(msg);
    return O3G_ERR_NOT_CONVERGED;
  }
  return O3G_OK;
}

// =====================================================================================
// Several right-hand sides per pass over the matrix.  Each refinement sweep and each
// GMRES iteration of one right-hand side streams the n^2 FP32 matrix once (6.7 GB at
// n = 40,960): the products, the triangular solves and the Krylov steps below serve up to
// kMaxRhs right-hand sides with that one pass.  BEM::solve takes one b (BEM.h:200-203); the
// reference solves again per RK stage (Convection.h:197) and per diffusion step
// (Diffusion.h:184-187), and these entry points let a caller hand all of them over at once.
namespace o3g {

constexpr int kMaxRhs = 8;
constexpr int kMvChunkM = 512;   // columns per block of the multi-vector product

struct DIn { const double* p[kMaxRhs]; };
struct DOut { double* p[kMaxRhs]; };

// xh/xl[c][.] = the float split of src.p[c] (K vectors of n)
__global__ void k_split_f64_multi(DIn src, float* xh, float* xl, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
  if (i >= n) return;
  const double v = src.p[c][i];
  const float h = (float)v;
  xh[(size_t)c * n + i] = h;
  xl[(size_t)c * n + i] = (float)(v - (double)h);
}

// part[cb][c][i] = sum over the columns of chunk cb of A[i, j] x_c[j], double-single as in
// k_matvec_ds: every matrix element is loaded once for the K vectors.  With K vectors the
// sums cost K times the FP32 instructions of one, so they run in packed FP32 (FFMA2,
// FADD2, FMUL2; each lane rounds like the scalar instruction): columns j and j + 1 of the
// chunk ride in the two lanes, each lane carrying its own double-single sum, added in
// double at the end.  Differences are formed as fused multiply-adds with -1 (exact
// negation), so the two-sum needs no negated operands: shared memory holds x_h, -x_h and
// x_l of each column pair.
__device__ __forceinline__ void ds_add_product2(float2 a, float2 h, float2 hn, float2 l, float2& hi, float2& lo) {
  const float2 m1 = make_float2(-1.f, -1.f);
  const float2 pn = __fmul2_rn(a, hn);                      // -p, p = a h rounded
  const float2 e = __ffma2_rn(a, h, pn);                    // a h - p, exact
  const float2 sum = __ffma2_rn(pn, m1, hi);                // hi + p
  const float2 bb = __ffma2_rn(hi, m1, sum);                // sum - hi
  const float2 t2 = __ffma2_rn(__ffma2_rn(bb, m1, sum), m1, hi);   // hi - (sum - bb)
  const float2 t = __ffma2_rn(__fadd2_rn(pn, bb), m1, t2);  // t2 + (p - bb)
  hi = sum;
  lo = __ffma2_rn(a, l, __fadd2_rn(lo, __fadd2_rn(t, e)));
}

template <int K>
__global__ void __launch_bounds__(256) k_matvec_ds_multi(const float* __restrict__ A, long long ld, int n,
                                                         const float* __restrict__ xh, const float* __restrict__ xl,
                                                         double* __restrict__ part) {
  constexpr int M2 = kMvChunkM / 2;
  __shared__ float2 sh[K][M2], shn[K][M2], sl[K][M2];   // column pairs (x_h, -x_h, x_l)
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int cb = blockIdx.y;
  const int j0 = cb * kMvChunkM, m = min(n - j0, kMvChunkM);
#pragma unroll
  for (int c = 0; c < K; ++c)
    for (int k = threadIdx.x; k < M2; k += blockDim.x) {
      // a column beyond the chunk gets x = 0 (and its matrix element 0 below)
      const float h0 = 2 * k < m ? xh[(size_t)c * n + j0 + 2 * k] : 0.f;
      const float h1 = 2 * k + 1 < m ? xh[(size_t)c * n + j0 + 2 * k + 1] : 0.f;
      const float l0 = 2 * k < m ? xl[(size_t)c * n + j0 + 2 * k] : 0.f;
      const float l1 = 2 * k + 1 < m ? xl[(size_t)c * n + j0 + 2 * k + 1] : 0.f;
      sh[c][k] = make_float2(h0, h1);
      shn[c][k] = make_float2(-h0, -h1);
      sl[c][k] = make_float2(l0, l1);
    }
  __syncthreads();
  if (i >= n) return;
  const float* a = A + (size_t)j0 * ld + i;
  float2 hi[K], lo[K];
#pragma unroll
  for (int c = 0; c < K; ++c) { hi[c] = make_float2(0.f, 0.f); lo[c] = make_float2(0.f, 0.f); }
  const float2 m1 = make_float2(-1.f, -1.f);
  int k = 0;
  for (; k + 8 <= m; k += 8) {
    float2 av[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      av[q] = make_float2(__ldg(a + (size_t)(k + 2 * q) * ld), __ldg(a + (size_t)(k + 2 * q + 1) * ld));
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < K; ++c)
        ds_add_product2(av[q], sh[c][k / 2 + q], shn[c][k / 2 + q], sl[c][k / 2 + q], hi[c], lo[c]);
    // renormalise: move the bulk of lo into hi (Dekker's fast two-sum, |hi| >= |lo|)
#pragma unroll
    for (int c = 0; c < K; ++c) {
      const float2 s2 = __fadd2_rn(hi[c], lo[c]);
      lo[c] = __ffma2_rn(__ffma2_rn(hi[c], m1, s2), m1, lo[c]);
      hi[c] = s2;
    }
  }
  for (; k < m; k += 2) {   // the chunk's last columns (m is even except at the matrix edge)
    const float2 av = make_float2(__ldg(a + (size_t)k * ld), k + 1 < m ? __ldg(a + (size_t)(k + 1) * ld) : 0.f);
#pragma unroll
    for (int c = 0; c < K; ++c) ds_add_product2(av, sh[c][k / 2], shn[c][k / 2], sl[c][k / 2], hi[c], lo[c]);
  }
#pragma unroll
  for (int c = 0; c < K; ++c)
    part[((size_t)cb * K + c) * n + i] = ((double)hi[c].x + (double)lo[c].x) + ((double)hi[c].y + (double)lo[c].y);
}

// y_c = b_c - sum_cb part (b given) or y_c = sum_cb part, c = blockIdx.y < K; per-block sums
// of y_c^2 into nrm[c][blockIdx.x]
__global__ void k_matvec_finish_multi(const double* __restrict__ part, int ncb, int K, int n, DIn b, DOut y,
                                      double* __restrict__ nrm) {
  __shared__ double s1[8];
  const int i = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
  double yy = 0.0;
  if (i < n) {
    double s = 0.0;
    for (int k = 0; k < ncb; ++k) s += part[((size_t)k * K + c) * n + i];
    const double v = b.p[c] ? b.p[c][i] - s : s;
    y.p[c][i] = v;
    yy = v * v;
  }
  for (int o = 16; o > 0; o >>= 1) yy += __shfl_xor_sync(0xffffffffu, yy, o);
  if ((threadIdx.x & 31) == 0) s1[threadIdx.x >> 5] = yy;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a1 = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) a1 += s1[w];
    nrm[(size_t)c * gridDim.x + blockIdx.x] = a1;
  }
}

// y[c][i] = r[c][perm[i]] for the columns in `mask`, 0 for the others (no correction)
__global__ void k_permute_to_float_multi(const double* r, const int* perm, float* y, int n, unsigned mask) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
  if (i < n) y[(size_t)c * n + i] = ((mask >> c) & 1u) ? (float)r[(size_t)c * n + perm[i]] : 0.f;
}

// the products b_c - A x_c (b given) or A x_c for K vectors in one pass over A, with the
// squared norms of the results on the host (synchronises) when norm2 is given
static int32_t matvec_multi(o3g_bem_t* h, int K, const DIn& x, const DIn& b, const DOut& y, float* xh, float* xl,
                            double* part, double* nrm, std::vector<double>* norm2, cudaStream_t st) {
  const int n = h->n;
  const int nrb = (n + 255) / 256;
  const int ncb = (n + kMvChunkM - 1) / kMvChunkM;
  int nc = 0;
  if (x.p[0] && K == 1) {
    // one vector: the single-vector product (HBM-bound already, 1024-column chunks)
    k_split_f64_multi<<<dim3(nrb, 1), 256, 0, st>>>(x, xh, xl, n);
    const int ncb1 = (n + kMvChunk - 1) / kMvChunk;
    k_matvec_ds<<<dim3(nrb, ncb1), 256, 0, st>>>(h->A, h->ld, n, xh, xl, part);
    note_launch(2);
    nc = ncb1;
  } else if (x.p[0]) {
    k_split_f64_multi<<<dim3(nrb, K), 256, 0, st>>>(x, xh, xl, n);
    const dim3 g(nrb, ncb);
    switch (K) {
      case 2: k_matvec_ds_multi<2><<<g, 256, 0, st>>>(h->A, h->ld, n, xh, xl, part); break;
      case 3: k_matvec_ds_multi<3><<<g, 256, 0, st>>>(h->A, h->ld, n, xh, xl, part); break;
      case 4: k_matvec_ds_multi<4><<<g, 256, 0, st>>>(h->A, h->ld, n, xh, xl, part); break;
      case 5: k_matvec_ds_multi<5><<<g, 256, 0, st>>>(h->A, h->ld, n, xh, xl, part); break;
      case 6: k_matvec_ds_multi<6><<<g, 256, 0, st>>>(h->A, h->ld, n, xh, xl, part); break;
      case 7: k_matvec_ds_multi<7><<<g, 256, 0, st>>>(h->A, h->ld, n, xh, xl, part); break;
      default: k_matvec_ds_multi<8><<<g, 256, 0, st>>>(h->A, h->ld, n, xh, xl, part); break;
    }
    note_launch(2);
    nc = ncb;
  }
  k_matvec_finish_multi<<<dim3(nrb, K), 256, 0, st>>>(part, nc, K, n, b, y, nrm);
  note_launch();
  O3G_CUDA_TRY(cudaGetLastError());
  if (norm2) {
    std::vector<double> hn((size_t)K * nrb);
    O3G_CUDA_TRY(cudaMemcpyAsync(hn.data(), nrm, hn.size() * 8, cudaMemcpyDeviceToHost, st));
    O3G_CUDA_TRY(cudaStreamSynchronize(st));
    norm2->assign(K, 0.0);
    for (int c = 0; c < K; ++c)
      for (int k = 0; k < nrb; ++k) (*norm2)[c] += hn[(size_t)c * nrb + k];
  }
  return O3G_OK;
}

}  // namespace o3g

static int32_t many_args(o3g_bem_t* h, int32_t nrhs, const float* B, int32_t mem, double tol, int32_t max_iter,
                         const char* who) {
  O3G_TRY(bem_check(h));
  if (nrhs < 0 || (nrhs > 0 && !B) || (mem != O3G_MEM_HOST && mem != O3G_MEM_DEVICE) || max_iter < 1 ||
      !(tol >= 0.0)) {
    char msg[160];
    std::snprintf(msg, sizeof(msg), "%s: bad arguments (nrhs >= 0, B given, mem HOST or DEVICE, max_iter >= 1, tol >= 0)",
                  who);
    set_error(msg);
    return O3G_ERR_INVALID_ARG;
  }
  return O3G_OK;
}

extern "C" int32_t o3g_bem_solve_many(o3g_bem_t* h, int32_t nrhs, const float* B, float* X, double* X64, int32_t mem,
                                      double tol, int32_t max_iter, int32_t* iters, double* relres, void* stream) {
  O3G_TRY(many_args(h, nrhs, B, mem, tol, max_iter, "o3g_bem_solve_many"));
  if (!h->factored) {
    set_error("o3g_bem_solve_many: factor the matrix first (o3g_bem_factor)");
    return O3G_ERR_STATE;
  }
  if (nrhs == 0) return O3G_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int n = h->n;
  const long long ld = h->ld;
  DeviceFacts df;
  O3G_TRY(device_facts(&df));
  const int KM = std::min(nrhs, kMaxRhs);
  const int ncb = (n + kMvChunkM - 1) / kMvChunkM;
  const int nrb = (n + 255) / 256;
  const size_t kn = (size_t)KM * n;
  const size_t need = 3 * align_up(kn * 8) + 5 * align_up(kn * 4) + align_up((size_t)ncb * kn * 8) +
                      align_up((size_t)KM * nrb * 8);
  O3G_TRY(bem_scratch(h, need));
  Carve cv(h->scratch);
  double* bd = cv.take<double>(kn);
  double* xd = cv.take<double>(kn);
  double* rd = cv.take<double>(kn);
  float* bf = cv.take<float>(kn);
  float* y = cv.take<float>(kn);
  float* w = cv.take<float>(kn);
  float* xh = cv.take<float>(kn);
  float* xl = cv.take<float>(kn);
  double* part = cv.take<double>((size_t)ncb * kn);
  double* nrm = cv.take<double>((size_t)KM * nrb);
  const cudaMemcpyKind h2d = mem == O3G_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  const cudaMemcpyKind d2h = mem == O3G_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  bool timed_out = false, all_converged = true;
  KernelTimer& tm = thread_timer();
  tm.begin(st);
  for (int g0 = 0; g0 < nrhs; g0 += kMaxRhs) {
    const int K = std::min(kMaxRhs, nrhs - g0);
    const size_t knn = (size_t)K * n;
    O3G_CUDA_TRY(cudaMemcpyAsync(bf, B + (size_t)g0 * n, knn * 4, h2d, st));
    k_f2d<<<(unsigned)((knn + 255) / 256), 256, 0, st>>>(bf, bd, (int)knn);
    note_launch();
    O3G_CUDA_TRY(cudaMemsetAsync(xd, 0, knn * 8, st));
    O3G_CUDA_TRY(cudaMemsetAsync(h->flags, 0, 4 * sizeof(int), st));
    DIn xin{}, bin{};
    DOut rout{};
    for (int c = 0; c < K; ++c) {
      xin.p[c] = xd + (size_t)c * n;
      bin.p[c] = bd + (size_t)c * n;
      rout.p[c] = rd + (size_t)c * n;
    }
    DIn none{};
    const int G = trsv_grid(df.num_sms);
    TrsvArgs lo, up;
    lo.LU = h->LU; lo.dinv = h->dinv; lo.ld = ld; lo.n = n; lo.y = y; lo.out = w;
    lo.bar = make_barrier(h->flags);
    up = lo;
    up.y = w; up.out = y;
    std::vector<double> rr, bnorm(K, 0.0), rel(K, 1.0);
    unsigned todo = (1u << K) - 1u;   // the columns of this pass
    std::vector<int> it_of(K, max_iter);
    for (int pass = 0; pass < refine_passes(n) && todo; ++pass) {
      unsigned active = todo;
      const bool last = pass + 1 == refine_passes(n);
      bool finite = true;
      for (int c = 0; c < K && pass > 0; ++c)
        if ((todo >> c) & 1u) O3G_CUDA_TRY(cudaMemsetAsync(xd + (size_t)c * n, 0, (size_t)n * 8, st));
      for (int it = 0; it <= max_iter; ++it) {
        O3G_TRY(matvec_multi(h, K, it > 0 || pass > 0 ? xin : none, bin, rout, xh, xl, part, nrm, &rr, st));
        for (int c = 0; c < K; ++c) {
          if (it == 0 && pass == 0) bnorm[c] = std::sqrt(rr[c]);
          if (!((active >> c) & 1u)) continue;
          rel[c] = bnorm[c] > 0.0 ? std::sqrt(rr[c]) / bnorm[c] : std::sqrt(rr[c]);
          if (!std::isfinite(rel[c])) finite = false;
          if (rel[c] <= tol || it == max_iter || (!std::isfinite(rel[c]) && !last)) {
            active &= ~(1u << c);
            it_of[c] = it;
          }
        }
        if (!active) break;
        k_permute_to_float_multi<<<dim3(nrb, K), 256, 0, st>>>(rd, h->perm, y, n, active);
        note_launch();
        O3G_TRY(trsv(K, refine_step(pass), lo, up, G, st));
        k_axpy_f2d<<<(unsigned)((knn + 255) / 256), 256, 0, st>>>(xd, y, (int)knn);
        note_launch();
      }
      // (an infinite inverse spoils the finished columns too: 0 inf)
      if (finite)
        for (int c = 0; c < K; ++c)
          if (rel[c] <= tol) todo &= ~(1u << c);
    }
    int fl = 0;
    O3G_CUDA_TRY(cudaMemcpyAsync(&fl, h->flags, sizeof(int), cudaMemcpyDeviceToHost, st));
    k_d2f<<<(unsigned)((knn + 255) / 256), 256, 0, st>>>(xd, bf, (int)knn);
    note_launch();
    if (X) O3G_CUDA_TRY(cudaMemcpyAsync(X + (size_t)g0 * n, bf, knn * 4, d2h, st));
    if (X64) O3G_CUDA_TRY(cudaMemcpyAsync(X64 + (size_t)g0 * n, xd, knn * 8, d2h, st));
    O3G_CUDA_TRY(cudaStreamSynchronize(st));
    for (int c = 0; c < K; ++c) {
      if (iters) iters[g0 + c] = it_of[c];
      if (relres) relres[g0 + c] = rel[c];
      if (!(rel[c] <= tol)) all_converged = false;
    }
    if (fl) {
      timed_out = true;
      break;
    }
  }
  tm.end(st);
  if (timed_out) {
    set_error("o3g_bem_solve_many: a grid barrier timed out");
    return O3G_ERR_TIMEOUT;
  }
  if (!all_converged) {
    set_error("o3g_bem_solve_many: some right-hand sides did not reach the tolerance (see relres)");
    return O3G_ERR_NOT_CONVERGED;
  }
  return O3G_OK;
}

// GMRES(restart) for several right-hand sides in lockstep: each keeps its own Krylov basis,
// Hessenberg matrix and restarts (the single-vector algorithm of o3g_bem_solve_gmres), and
// every iteration applies A to all of their current vectors in one pass over the matrix.
extern "C" int32_t o3g_bem_solve_gmres_many(o3g_bem_t* h, int32_t nrhs, const float* B, float* X, double* X64,
                                            int32_t mem, double tol, int32_t max_iter, int32_t restart,
                                            int32_t* iters, double* relres, void* stream) {
  O3G_TRY(many_args(h, nrhs, B, mem, tol, max_iter, "o3g_bem_solve_gmres_many"));
  if (restart < 1 || restart > 500) {
    set_error("o3g_bem_solve_gmres_many: restart must be 1..500");
    return O3G_ERR_INVALID_ARG;
  }
  if (nrhs == 0) return O3G_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int n = h->n;
  const int m = std::min(restart, max_iter);
  const int KM = std::min(nrhs, kMaxRhs);
  const int ncb = (n + kMvChunkM - 1) / kMvChunkM;
  const int nrb = (n + 255) / 256;
  const size_t kn = (size_t)KM * n;
  const int nkb = (n + kKrylovRows - 1) / kKrylovRows;
  const int bs = h->bs, npb = n / bs;
  const bool pre = bs > 1;   // right-preconditioned by the diagonal blocks, as o3g_bem_solve_gmres
  const size_t need = align_up(kn * (m + 1) * 8) + 2 * align_up(kn * 8) + 3 * align_up(kn * 4) +
                      align_up((size_t)ncb * kn * 8) + align_up((size_t)KM * nrb * 8) +
                      align_up((size_t)KM * 2 * (m + 1) * 8) + 2 * align_up((size_t)nkb * (m + 1) * 8) +
                      align_up((size_t)n * bs * 8) + align_up(kn * 8);
  O3G_TRY(bem_scratch(h, need));
  Carve cv(h->scratch);
  double* V = cv.take<double>(kn * (m + 1));     // basis of column c at V + c (m+1) n
  double* bd = cv.take<double>(kn);
  double* xd = cv.take<double>(kn);
  float* bf = cv.take<float>(kn);
  float* xh = cv.take<float>(kn);
  float* xl = cv.take<float>(kn);
  double* part = cv.take<double>((size_t)ncb * kn);
  double* nrm = cv.take<double>((size_t)KM * nrb);
  double* hd = cv.take<double>((size_t)KM * 2 * (m + 1));
  double* kpart = cv.take<double>((size_t)nkb * (m + 1));
  double* npart = cv.take<double>((size_t)nkb * (m + 1));
  double* Minv = cv.take<double>((size_t)n * bs);
  double* zb = cv.take<double>(kn);   // per column: M^-1 v, and V y before M^-1
  std::vector<double> hnp((size_t)nkb);
  if (pre) block_inv(h->A, h->ld, npb, bs, Minv, st);
  const cudaMemcpyKind h2d = mem == O3G_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  const cudaMemcpyKind d2h = mem == O3G_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  bool all_converged = true;
  KernelTimer& tm = thread_timer();
  tm.begin(st);
  struct Rhs {
    std::vector<double> H, cs, sn, g, y;
    double bnorm = 0.0, rel = 1.0;
    int k = 0, total = 0;
    bool done = false, fresh = true;   // fresh: a cycle starts (residual, basis reset) next
  };
  for (int g0 = 0; g0 < nrhs; g0 += kMaxRhs) {
    const int K = std::min(kMaxRhs, nrhs - g0);
    const size_t knn = (size_t)K * n;
    O3G_CUDA_TRY(cudaMemcpyAsync(bf, B + (size_t)g0 * n, knn * 4, h2d, st));
    k_f2d<<<(unsigned)((knn + 255) / 256), 256, 0, st>>>(bf, bd, (int)knn);
    note_launch();
    O3G_CUDA_TRY(cudaMemsetAsync(xd, 0, knn * 8, st));
    std::vector<Rhs> R(K);
    auto Vc = [&](int c, int k) { return V + ((size_t)c * (m + 1) + k) * n; };
    for (int c = 0; c < K; ++c) {
      R[c].H.assign((size_t)(m + 1) * m, 0.0);
      R[c].cs.assign(m, 0.0);
      R[c].sn.assign(m, 0.0);
      R[c].g.assign(m + 1, 0.0);
      R[c].y.assign(m, 0.0);
    }
    // ||b_c||
    {
      DIn none{}, bin{};
      DOut vout{};
      for (int c = 0; c < K; ++c) {
        bin.p[c] = bd + (size_t)c * n;
        vout.p[c] = Vc(c, 0);
      }
      std::vector<double> bb;
      O3G_TRY(matvec_multi(h, K, none, bin, vout, xh, xl, part, nrm, &bb, st));
      for (int c = 0; c < K; ++c) {
        R[c].bnorm = std::sqrt(bb[c]);
        if (R[c].bnorm == 0.0) { R[c].done = true; R[c].rel = 0.0; }
      }
    }
    for (;;) {
      // columns starting a cycle: r = b - A x into their V_0, in one pass (x = 0 on the
      // first cycle: r = b, no product)
      std::vector<int> fr;
      for (int c = 0; c < K; ++c)
        if (!R[c].done && R[c].fresh) fr.push_back(c);
      if (!fr.empty()) {
        DIn xin{}, bin{};
        DOut vout{};
        bool any_x = false;
        for (int q = 0; q < (int)fr.size(); ++q) {
          const int c = fr[q];
          xin.p[q] = xd + (size_t)c * n;
          bin.p[q] = bd + (size_t)c * n;
          vout.p[q] = Vc(c, 0);
          any_x = any_x || R[c].total > 0;
        }
        if (!any_x) xin = DIn{};
        std::vector<double> rr;
        O3G_TRY(matvec_multi(h, (int)fr.size(), xin, bin, vout, xh, xl, part, nrm, &rr, st));
        for (int q = 0; q < (int)fr.size(); ++q) {
          Rhs& s = R[fr[q]];
          s.rel = std::sqrt(rr[q]) / s.bnorm;
          if (s.rel <= tol || s.total >= max_iter) {
            s.done = true;
            continue;
          }
          const double beta = std::sqrt(rr[q]);
          k_kry_scale<<<nrb, 256, 0, st>>>(Vc(fr[q], 0), n, 1.0 / beta);
          note_launch();
          std::fill(s.g.begin(), s.g.end(), 0.0);
          s.g[0] = beta;
          s.k = 0;
          s.fresh = false;
        }
      }
      std::vector<int> act;
      for (int c = 0; c < K; ++c)
        if (!R[c].done) act.push_back(c);
      if (act.empty()) break;
      // w_c = A v_{c,k} for every active column, one pass
      {
        DIn xin{}, none{};
        DOut wout{};
        for (int q = 0; q < (int)act.size(); ++q) {
          xin.p[q] = Vc(act[q], R[act[q]].k);
          wout.p[q] = Vc(act[q], R[act[q]].k + 1);
          if (pre) {
            block_apply(Minv, npb, bs, xin.p[q], zb + (size_t)q * n, 0, st);
            xin.p[q] = zb + (size_t)q * n;
          }
        }
        O3G_TRY(matvec_multi(h, (int)act.size(), xin, none, wout, xh, xl, part, nrm, nullptr, st));
      }
      for (int c : act) {
        Rhs& s = R[c];
        const int k = s.k;
        double* Vb = Vc(c, 0);
        double* w = Vc(c, k + 1);
        double* hc_d = hd + (size_t)c * 2 * (m + 1);
        for (int pass = 0; pass < 2; ++pass) gs_pass(Vb, n, k + 1, w, hc_d + (size_t)pass * (m + 1), kpart, st);
        norm_partials(w, n, npart, st);
        std::vector<double> hc(2 * (size_t)(m + 1));
        O3G_CUDA_TRY(cudaMemcpyAsync(hc.data(), hc_d, hc.size() * 8, cudaMemcpyDeviceToHost, st));
        O3G_CUDA_TRY(cudaMemcpyAsync(hnp.data(), npart, (size_t)nkb * 8, cudaMemcpyDeviceToHost, st));
        O3G_CUDA_TRY(cudaStreamSynchronize(st));
        const double wn = std::sqrt(host_sum(hnp));
        auto Hat = [&](int i, int kk) -> double& { return s.H[(size_t)kk * (m + 1) + i]; };
        for (int i = 0; i <= k; ++i) Hat(i, k) = hc[i] + hc[(size_t)(m + 1) + i];
        Hat(k + 1, k) = wn;
        if (wn > 0.0) {
          k_kry_scale<<<nrb, 256, 0, st>>>(w, n, 1.0 / wn);
          note_launch();
        }
        for (int i = 0; i < k; ++i) {
          const double a = Hat(i, k), cc = Hat(i + 1, k);
          Hat(i, k) = s.cs[i] * a + s.sn[i] * cc;
          Hat(i + 1, k) = -s.sn[i] * a + s.cs[i] * cc;
        }
        const double dd = std::hypot(Hat(k, k), Hat(k + 1, k));
        s.cs[k] = dd > 0.0 ? Hat(k, k) / dd : 1.0;
        s.sn[k] = dd > 0.0 ? Hat(k + 1, k) / dd : 0.0;
        Hat(k, k) = dd;
        Hat(k + 1, k) = 0.0;
        s.g[k + 1] = -s.sn[k] * s.g[k];
        s.g[k] = s.cs[k] * s.g[k];
        s.k = k + 1;
        ++s.total;
        if (s.k == m || s.total >= max_iter || std::fabs(s.g[s.k]) <= 0.5 * tol * s.bnorm || wn == 0.0) {
          // end of the cycle: x += V y with H(0:k, 0:k) y = g(0:k)
          const int kk = s.k;
          for (int i = kk - 1; i >= 0; --i) {
            double sacc = s.g[i];
            for (int j = i + 1; j < kk; ++j) sacc -= Hat(i, j) * s.y[j];
            s.y[i] = Hat(i, i) != 0.0 ? sacc / Hat(i, i) : 0.0;
          }
          O3G_CUDA_TRY(cudaMemcpyAsync(hc_d, s.y.data(), (size_t)kk * 8, cudaMemcpyHostToDevice, st));
          if (pre) {
            double* z = zb + (size_t)c * n;
            O3G_CUDA_TRY(cudaMemsetAsync(z, 0, (size_t)n * 8, st));
            k_kry_update<<<nrb, 256, 0, st>>>(Vb, n, kk, hc_d, 1.0, z);
            note_launch();
            block_apply(Minv, npb, bs, z, xd + (size_t)c * n, 1, st);
          } else {
            k_kry_update<<<nrb, 256, 0, st>>>(Vb, n, kk, hc_d, 1.0, xd + (size_t)c * n);
            note_launch();
          }
          s.fresh = true;
        }
      }
    }
    k_d2f<<<(unsigned)((knn + 255) / 256), 256, 0, st>>>(xd, bf, (int)knn);
    note_launch();
    if (X) O3G_CUDA_TRY(cudaMemcpyAsync(X + (size_t)g0 * n, bf, knn * 4, d2h, st));
    if (X64) O3G_CUDA_TRY(cudaMemcpyAsync(X64 + (size_t)g0 * n, xd, knn * 8, d2h, st));
    O3G_CUDA_TRY(cudaStreamSynchronize(st));
    for (int c = 0; c < K; ++c) {
      if (iters) iters[g0 + c] = R[c].total;
      if (relres) relres[g0 + c] = R[c].rel;
      if (!(R[c].rel <= tol)) all_converged = false;
    }
  }
  tm.end(st);
  if (!all_converged) {
    set_error("o3g_bem_solve_gmres_many: some right-hand sides did not reach the tolerance (see relres)");
    return O3G_ERR_NOT_CONVERGED;
  }
  return O3G_OK;
}
