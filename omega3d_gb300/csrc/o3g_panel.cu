// o3g_panel.cu -- adaptive panel kernels: panels_affect_points (Influence.h:557-1099,
// rkernel_2vs_0pg / rkernel_2vs_0p, Kernels.h:1028-1211) and points_affect_panels
// (Influence.h:1107-1221, the same kernel used backwards for the BEM right-hand side).
//
// Subdivision follows the reference per pair: a (sub)triangle is evaluated as one
// singular vortex+source point at its centroid when dist(target, centroid) >
// 4*sqrt(area) or its level reached maxlev, otherwise it splits into the four children
// {0,1,3},{1,2,4},{1,4,3},{3,4,5} of its corner/midpoint list (Kernels.h:1085-1092),
// each with a quarter of the strength and area, visited depth first in that order.
// The well-separation test is computed with the reference's operation order and no
// fused multiply-adds (__fmul_rn/__fadd_rn), so every split decision is the reference's.
// With the source core radius 0 every core of CoreFunc.h reduces to the singular kernel,
// so the leaves here use 1/d^3 for all cores.
//
// Two kinds of work, kept apart because they suit different mappings:
//   * far pairs (nearly all): packed FP32 over pairs of panels (or particles), as the
//     particle kernels; a pair counts as far here when its squared distance passes the
//     squared threshold by 2^-18, so that the reference's rounded test surely agrees.  The
//     others' contributions are masked to zero and
//   * the pairs left go to a queue of nodes per warp: (owner, panel or particle, sub-triangle
//     path).  32 nodes are taken at a time, one per lane, whoever owns them; each takes the
//     reference's exact test and becomes a leaf or four child nodes.  Every lane has one
//     sub-triangle to do, while a thread that subdivides its own pairs holds up its warp: few
//     lanes have a close panel at the same time, and their trees have 4 to 64 leaves.
// The owner adds its nodes' sums in queue order: results do not depend on scheduling.
// Measured (one GB300), 5,120 panels on 262,144 points with gradients, compensated: 4.32 ->
// 2.28 ms; 100,000 particles on 20,480 panels: 3.05 -> 1.33 ms (1.41 with six rows a tile); 20 panels on
// 20,000 points, nearly all close, compensated with gradients: 0.63 -> 0.67 ms.
//
#include "o3g_pair_impl.cuh"

#include <algorithm>

namespace o3g {

constexpr int kPW = 32;           // threads per block (one warp) / panels (or particles) per tile
constexpr int kMaxLev = 6;        // deepest subdivision accepted by the C-ABI
constexpr int kFoldTiles = 4;     // tiles between two folds of the compensated sums (128 elements)
// A node queue is popped from its end, 32 at a time, and grows by at most 4 children each: below 32
// nodes before a sweep step adds up to 64 TPT, then the children pushed by one batch, at most 128, of
// which at most 96 are left while others lie behind them; the lowest level among those is one deeper than
// among these, so there are at most maxlev such groups
__host__ __device__ constexpr int queue_cap(int tpt, int maxlev) {
  return 31 + 64 * tpt + 96 * (maxlev > 1 ? maxlev - 1 : 0) + 128;
}
constexpr int kRows = 4;          // float4 rows of a staged tile

// A tile of kPW panels or particles, as pairs, component-major (kRows rows of kPW / 2 float4):
//   0: (-x0, -x1, -y0, -y1)   1: (-z0, -z1, t0, t1)   2: (sx0, sx1, sy0, sy1)
//   3: (sz0, sz1, q0, q1)
// position (a panel's centroid), squared far threshold, strength, source strength.
__device__ __forceinline__ void store_row(float4* tiles, int j, float x, float y, float z, float t, float sx, float sy,
                                          float sz, float q) {
  float* b = reinterpret_cast<float*>(tiles + (size_t)(j / kPW) * (kRows * kPW / 2) + (j % kPW) / 2) + (j & 1);
  constexpr int R = 4 * (kPW / 2);
  b[0] = -x;          b[2] = -y;
  b[R] = -z;          b[R + 2] = t;
  b[2 * R] = sx;      b[2 * R + 2] = sy;
  b[3 * R] = sz;      b[3 * R + 2] = q;
}

struct PanelNear {
  float4 a;   // x0 y0 z0 x1
  float4 b;   // y1 z1 x2 y2
  float4 d;   // z2, area, -, -
  float4 s;   // absolute strength x, y, z (sheet * area); source strength * area
};

struct Tri {
  float x0, y0, z0, x1, y1, z1, x2, y2, z2;
};

// centroid and well-separation test in the reference's order (Kernels.h:1141-1158)
__device__ __forceinline__ void centroid(const Tri& t, float& cx, float& cy, float& cz) {
  cx = div3_rn(__fadd_rn(__fadd_rn(t.x0, t.x1), t.x2));
  cy = div3_rn(__fadd_rn(__fadd_rn(t.y0, t.y1), t.y2));
  cz = div3_rn(__fadd_rn(__fadd_rn(t.z0, t.z1), t.z2));
}
__device__ __forceinline__ float dist_rn(float tx, float ty, float tz, float cx, float cy, float cz) {
  const float dx = __fsub_rn(tx, cx), dy = __fsub_rn(ty, cy), dz = __fsub_rn(tz, cz);
  return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
}
// the squared distance beyond which the rounded test above surely says far: the packed sum of
// squares differs from the rounded one by less than 2^-21 relative, and so do the roundings of
// the root and of this product.  maxlev 0: every pair is far.
__device__ __forceinline__ float sure_far2(float thr, int maxlev) {
  return maxlev == 0 ? -1.0f : __fmul_rn(__fmul_rn(thr, thr), 1.000003814697265625f);   // 1 + 2^-18
}

// child c of a triangle: corner/midpoint list {v0, m01, v1, m02, m12, v2}, children {0,1,3},
// {1,2,4},{1,4,3},{3,4,5} (Kernels.h:1085)
__device__ __forceinline__ Tri child(const Tri& t, int c) {
  const float mx01 = 0.5f * (t.x0 + t.x1), my01 = 0.5f * (t.y0 + t.y1), mz01 = 0.5f * (t.z0 + t.z1);
  const float mx02 = 0.5f * (t.x0 + t.x2), my02 = 0.5f * (t.y0 + t.y2), mz02 = 0.5f * (t.z0 + t.z2);
  const float mx12 = 0.5f * (t.x1 + t.x2), my12 = 0.5f * (t.y1 + t.y2), mz12 = 0.5f * (t.z1 + t.z2);
  Tri o;
  o.x0 = c == 0 ? t.x0 : (c == 3 ? mx02 : mx01);
  o.y0 = c == 0 ? t.y0 : (c == 3 ? my02 : my01);
  o.z0 = c == 0 ? t.z0 : (c == 3 ? mz02 : mz01);
  o.x1 = c == 0 ? mx01 : (c == 1 ? t.x1 : mx12);
  o.y1 = c == 0 ? my01 : (c == 1 ? t.y1 : my12);
  o.z1 = c == 0 ? mz01 : (c == 1 ? t.z1 : mz12);
  o.x2 = c == 1 ? mx12 : (c == 3 ? t.x2 : mx02);
  o.y2 = c == 1 ? my12 : (c == 3 ? t.y2 : my02);
  o.z2 = c == 1 ? mz12 : (c == 3 ? t.z2 : mz02);
  return o;
}

// Sums of a thread's target: a[0..2] velocity, a[3..11] b3 d (x) c (c = s x d + q d),
// a[12..14] r3 s, a[15] r3 q; kernel_0vs_0pg with sr = 0 (Kernels.h:294-345).
template <bool GRADS, bool SRC> struct PanelSums { static constexpr int n = GRADS ? (SRC ? 16 : 15) : 3; };

// the pair of panels (particles) of rows q0..q2, (wz, qs) on one target tt = (x,x), (y,y), (z,z); `t2` the
// far thresholds; nx, ny: the pairs that are left out.  The warp votes first: almost always no
// lane has a near pair and nothing is selected.
template <bool GRADS, bool SRC, bool ACC>
__device__ __forceinline__ void far_pair(const float2* tt, const float4& q0, const float4& q1, const float4& q2,
                                         const float2& wz, const float2& qs, const float2& t2,
                                         float2* a, bool& nx, bool& ny, bool& any) {
  const float2 dx = __fadd2_rn(tt[0], f2lo(q0));
  const float2 dy = __fadd2_rn(tt[1], f2hi(q0));
  const float2 dz = __fadd2_rn(tt[2], f2lo(q1));
  const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
  float2 s2, r3;
  rsq2<ACC>(r2, s2, r3);
  nx = !(r2.x > t2.x);
  ny = !(r2.y > t2.y);
  if (__any_sync(0xffffffffu, nx || ny)) {
    // (a coincident point's s2 and r3 are infinite)
    r3 = make_float2(nx ? 0.f : r3.x, ny ? 0.f : r3.y);
    s2 = make_float2(nx ? 0.f : s2.x, ny ? 0.f : s2.y);
    any = true;
  }
  // signs on register operands, as pair2
  const float2 wx = f2lo(q2), wy = f2hi(q2);
  const float2 ndx = ACC ? dx : neg2(dx), ndy = ACC ? dy : neg2(dy), ndz = ACC ? dz : neg2(dz);
  const float2 nwx = ACC ? neg2(wx) : wx, nwy = ACC ? neg2(wy) : wy, nwz = ACC ? neg2(wz) : wz;
  float2 cx = __fmul2_rn(ndy, nwz), cy = __fmul2_rn(dx, wz), cz = __fmul2_rn(ndx, nwy);
  if (SRC) {
    cx = __ffma2_rn(dx, qs, cx);
    cy = __ffma2_rn(dy, qs, cy);
    cz = __ffma2_rn(dz, qs, cz);
  }
  cx = __ffma2_rn(dz, wy, cx);     // dz wy - dy wz
  cy = __ffma2_rn(ndz, nwx, cy);   // dx wz - dz wx
  cz = __ffma2_rn(dy, wx, cz);     // dy wx - dx wy
  a[0] = __ffma2_rn(r3, cx, a[0]);
  a[1] = __ffma2_rn(r3, cy, a[1]);
  a[2] = __ffma2_rn(r3, cz, a[2]);
  if (GRADS) {
    a[12] = __ffma2_rn(r3, wx, a[12]);
    a[13] = __ffma2_rn(r3, wy, a[13]);
    a[14] = __ffma2_rn(r3, wz, a[14]);
    if (SRC) a[15] = __ffma2_rn(r3, qs, a[15]);
    const float2 b3 = __fmul2_rn(r3, s2);
    cx = __fmul2_rn(cx, b3);
    cy = __fmul2_rn(cy, b3);
    cz = __fmul2_rn(cz, b3);
    a[3] = __ffma2_rn(dx, cx, a[3]);
    a[4] = __ffma2_rn(dx, cy, a[4]);
    a[5] = __ffma2_rn(dx, cz, a[5]);
    a[8] = __ffma2_rn(dy, cz, a[8]);
    a[7] = __ffma2_rn(dy, cy, a[7]);
    a[6] = __ffma2_rn(dy, cx, a[6]);
    a[9] = __ffma2_rn(dz, cx, a[9]);
    a[10] = __ffma2_rn(dz, cy, a[10]);
    a[11] = __ffma2_rn(dz, cz, a[11]);
  }
}

// one leaf: the same sums of a single point c on the target t, into v[0..n).  The leaves are few
// and the largest terms: they take the corrected reciprocal square root in every precision.
template <bool GRADS, bool SRC>
__device__ __forceinline__ void leaf(float dx, float dy, float dz, float sx, float sy, float sz, float q, float* v) {
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  float2 s2, r3;
  rsq2<true>(make_float2(r2, r2), s2, r3);
  float cx = dz * sy - dy * sz, cy = dx * sz - dz * sx, cz = dy * sx - dx * sy;
  if (SRC) {
    cx = fmaf(dx, q, cx);
    cy = fmaf(dy, q, cy);
    cz = fmaf(dz, q, cz);
  }
  v[0] = r3.x * cx;
  v[1] = r3.x * cy;
  v[2] = r3.x * cz;
  if (GRADS) {
    v[12] = r3.x * sx;
    v[13] = r3.x * sy;
    v[14] = r3.x * sz;
    if (SRC) v[15] = r3.x * q;
    const float b3 = r3.x * s2.x;
    cx *= b3; cy *= b3; cz *= b3;
    v[3] = dx * cx; v[4] = dx * cy; v[5] = dx * cz;
    v[6] = dy * cx; v[7] = dy * cy; v[8] = dy * cz;
    v[9] = dz * cx; v[10] = dz * cy; v[11] = dz * cz;
  }
}

// the 3 or 12 results from a thread's sums
template <bool GRADS, bool SRC>
__device__ __forceinline__ void panel_fold(float* a) {
  if (!GRADS) return;
  fold_grads<CORE_SING>(a);
  if (SRC) {
    a[3] += a[15];
    a[7] += a[15];
    a[11] += a[15];
  }
}

// error-free a + b = s + e (Knuth's two-sum)
__device__ __forceinline__ void two_sum_f(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// compensated mode: fold the plain partial sums of one tile into (hi, lo)
template <int NC>
__device__ __forceinline__ void fold_tile(float* a, float* hi, float* lo) {
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    float sum, err;
    two_sum_f(hi[c], a[c], sum, err);
    hi[c] = sum;
    lo[c] += err;
  }
}

// The node queue of one warp.  A node: x = panel or particle index, y = owner lane | target k
// << 5 | level << 8 | path << 11 (2 bits per level, level 1 in the low ones).
template <bool GRADS, bool SRC, bool ACC> struct NodeSums {
  // compensated: a node's finished results, added to (hi, lo) one by one (the close nodes are
  // the largest terms, and their sums' parts cancel); plain: its sums
  static constexpr int n = ACC ? (GRADS ? 12 : 3) : PanelSums<GRADS, SRC>::n;
};
// In dynamic shared memory: two staged tiles, then the nodes' sums, the owners' masks and the
// nodes.
template <int NV, int TPT> struct WarpShared {
  float4 buf[2][kRows][kPW / 2];
  float sums[NV][32];      // the nodes' sums, by the lane that computed them
  unsigned mine[TPT][32];  // per owner: the lanes whose sums are its own
  uint2 node[1];           // queue_cap(TPT, maxlev) of them
  static size_t bytes(int maxlev) { return sizeof(WarpShared) + (queue_cap(TPT, maxlev) - 1) * sizeof(uint2); }
};

// Takes the last min(32, cnt) nodes.  fetch(node, tri, area, px, py, pz, sx, sy, sz, q) gives a
// node's panel, its evaluation point (relative sign SGN: d = SGN (point - centroid)) and strength;
// it is called by every lane (it may shuffle).
template <bool GRADS, bool SRC, bool ACC, int TPT, int SGN, class Shared, class Fetch>
__device__ __forceinline__ void take_nodes(Shared& q, int& cnt, int maxlev,
                                           float2 (*a)[PanelSums<GRADS, SRC>::n], float (*hi)[GRADS ? 12 : 3],
                                           float (*lo)[GRADS ? 12 : 3], const Fetch& fetch) {
  constexpr int NV = NodeSums<GRADS, SRC, ACC>::n;
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int take = min(32, cnt);
  const int base = cnt - take;
  const bool act = lane < take;
  const uint2 nd = act ? q.node[base + lane] : make_uint2(0u, 0u);
#pragma unroll
  for (int k = 0; k < TPT; ++k) q.mine[k][lane] = 0u;
  Tri t;
  float area, px, py, pz, sx, sy, sz, qs;
  fetch(nd, act, t, area, px, py, pz, sx, sy, sz, qs);
  const int lev = (int)((nd.y >> 8) & 7u);
  for (int l = 0; l < lev; ++l) t = child(t, (int)((nd.y >> (11 + 2 * l)) & 3u));
  float cx, cy, cz;
  centroid(t, cx, cy, cz);
  // 4 sqrt(area 0.25^lev) = 4 sqrt(area) 0.5^lev, exactly
  const float thr = __fmul_rn(__fmul_rn(__fsqrt_rn(area), 4.0f), __int_as_float((127 - lev) << 23));
  const bool split = act && lev < maxlev && !(dist_rn(px, py, pz, cx, cy, cz) > thr);
  __syncwarp();
  if (act && !split) {
    // 0.25^lev, exact powers of two (the reference scales by 0.25 per split, Kernels.h:1072-1075)
    const float f = __int_as_float((127 - 2 * lev) << 23);
    float v[16];
    leaf<GRADS, SRC>(SGN * (px - cx), SGN * (py - cy), SGN * (pz - cz), sx * f, sy * f, sz * f, qs * f, v);
    if (ACC) panel_fold<GRADS, SRC>(v);
#pragma unroll
    for (int c = 0; c < NV; ++c) q.sums[c][lane] = v[c];
    atomicOr(&q.mine[(nd.y >> 5) & 7u][nd.y & 31u], 1u << lane);
  }
  const unsigned m = __ballot_sync(full, split);
  if (split) {
    const int at = base + __popc(m & ((1u << lane) - 1u)), ns = __popc(m);
    const unsigned y = (nd.y & 0xffu) | ((unsigned)(lev + 1) << 8) | (nd.y & ~0x7ffu);
    // child 0 of all last: it is taken first.  Child by child, so that the next 32 nodes belong to as many
    // owners as these: an owner adds its nodes one after the other (20 panels on 20,000 points, nearly all
    // close, compensated: 1.09 -> 0.67 ms; parent by parent was slower than a thread per point there).
#pragma unroll
    for (int c = 0; c < 4; ++c) q.node[at + c * ns] = make_uint2(nd.x, y | ((unsigned)(3 - c) << (11 + 2 * lev)));
  }
  cnt = base + 4 * __popc(m);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    for (unsigned bits = q.mine[k][lane]; bits; bits &= bits - 1u) {
      const int e = __ffs(bits) - 1;
#pragma unroll
      for (int c = 0; c < NV; ++c) {
        if constexpr (ACC) {
          float sum, err;
          two_sum_f(hi[k][c], q.sums[c][e], sum, err);
          hi[k][c] = sum;
          lo[k][c] += err;
        } else {
          a[k][c].x += q.sums[c][e];
        }
      }
    }
  }
  __syncwarp();
}

// Sweeps tiles [t0, t1) for the TPT targets of each thread (live: the thread's target exists),
// near pairs through the warp's queue; folds every kFoldTiles tiles into (hi, lo) when ACC.
// OWN_T: the far threshold belongs to the thread's target (own2) instead of the swept element.
// A warp stages its own tiles (cp.async, the next one while it sweeps this one) and meets no
// other warp at a barrier: the queues' work differs from warp to warp, and with four warps
// sharing tiles each waited for the slowest (1.9 stalls per issue at the barrier).
template <bool GRADS, bool SRC, bool ACC, int TPT, int SGN, bool OWN_T, class Shared, class Fetch>
__device__ __forceinline__ void sweep_panels(const float4* __restrict__ tiles, int t0, int t1, int maxlev, Shared& q,
                                             const float2 (*tt)[3], const float* own2, const bool* live,
                                             float2 (*a)[PanelSums<GRADS, SRC>::n], float (*hi)[GRADS ? 12 : 3],
                                             float (*lo)[GRADS ? 12 : 3], const Fetch& fetch) {
  constexpr int NS = PanelSums<GRADS, SRC>::n;
  constexpr int NC = GRADS ? 12 : 3;
  constexpr int HALF = kPW / 2;
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x;
  int cnt = 0;
  auto stage = [&](int tile, int b) {
    const float4* g = tiles + (size_t)tile * (kRows * HALF);
    const unsigned d = (unsigned)__cvta_generic_to_shared(&q.buf[b][0][0]);
#pragma unroll
    for (int e = 0; e < kRows * HALF; e += kPW)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16u * (e + lane)), "l"(g + e + lane) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (t0 < t1) stage(t0, 0);
  for (int tile = t0; tile < t1; ++tile) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();   // this tile is staged for every lane; no lane still reads the other buffer
    const int cur = (tile - t0) & 1;
    if (tile + 1 < t1) stage(tile + 1, cur ^ 1);
    const float4 (*Q)[HALF] = q.buf[cur];
#pragma unroll 1
    for (int p = 0; p < HALF; ++p) {
      const float4 q0 = Q[0][p], q1 = Q[1][p], q2 = Q[2][p];
      float2 wz, qs = f2(0.f);
      if (SRC) {
        const float4 q3 = Q[3][p];
        wz = f2lo(q3);
        qs = f2hi(q3);
      } else {
        wz = *reinterpret_cast<const float2*>(&Q[3][p]);
      }
      bool nx[TPT], ny[TPT];
      const bool last = tile + 1 == t1 && p + 1 == HALF;
      bool any = last && cnt > 0;
#pragma unroll
      for (int k = 0; k < TPT; ++k)
        far_pair<GRADS, SRC, ACC>(tt[k], q0, q1, q2, wz, qs, OWN_T ? f2(own2[k]) : f2hi(q1), a[k], nx[k], ny[k],
                                  any);
      if (any) {
#pragma unroll
        for (int k = 0; k < TPT; ++k)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const bool nr = live[k] && (h ? ny[k] : nx[k]);
            const unsigned m = __ballot_sync(full, nr);
            if (nr)
              q.node[cnt + __popc(m & ((1u << lane) - 1u))] =
                  make_uint2((unsigned)(tile * kPW + 2 * p + h), (unsigned)lane | ((unsigned)k << 5));
            cnt += __popc(m);
          }
        __syncwarp();
        while (cnt >= 32 || (last && cnt > 0)) take_nodes<GRADS, SRC, ACC, TPT, SGN>(q, cnt, maxlev, a, hi, lo, fetch);
      }
    }
    if (ACC && ((tile - t0) % kFoldTiles == kFoldTiles - 1 || tile + 1 == t1)) {
#pragma unroll
      for (int k = 0; k < TPT; ++k) {
        float v[NS];
#pragma unroll
        for (int c = 0; c < NS; ++c) {
          v[c] = a[k][c].x + a[k][c].y;
          a[k][c] = f2(0.f);
        }
        panel_fold<GRADS, SRC>(v);
        fold_tile<NC>(v, hi[k], lo[k]);
      }
    }
  }
}

// panels as swept elements (tiles) and / or as owners (cen: centroid and squared far
// threshold), with their near records
__global__ void k_pack_panels(int np, const float* __restrict__ nx, const float* __restrict__ ny,
                              const float* __restrict__ nz, const uint32_t* __restrict__ idx,
                              const float* __restrict__ area, const float* __restrict__ tsx,
                              const float* __restrict__ tsy, const float* __restrict__ tsz,
                              const float* __restrict__ sss, int np_pad, int maxlev, float4* tiles, float4* cen,
                              PanelNear* nearr) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= np_pad) return;
  PanelNear n;
  float cx, cy, cz, t2;
  if (j < np) {
    const uint32_t p0 = idx[3 * (size_t)j], p1 = idx[3 * (size_t)j + 1], p2 = idx[3 * (size_t)j + 2];
    const Tri t{nx[p0], ny[p0], nz[p0], nx[p1], ny[p1], nz[p1], nx[p2], ny[p2], nz[p2]};
    centroid(t, cx, cy, cz);
    const float sa = area[j];
    float sx = 0.f, sy = 0.f, sz = 0.f;
    if (tsx) {
      // sheet strength = ts / area (Influence.h:958), absolute again at level 0 (Kernels.h:1040-1046)
      sx = __fmul_rn(__fdiv_rn(tsx[j], sa), sa);
      sy = __fmul_rn(__fdiv_rn(tsy[j], sa), sa);
      sz = __fmul_rn(__fdiv_rn(tsz[j], sa), sa);
    }
    const float s3 = sss ? __fmul_rn(sss[j], sa) : 0.f;
    t2 = sure_far2(__fmul_rn(__fsqrt_rn(sa), 4.0f), maxlev);
    n.a = make_float4(t.x0, t.y0, t.z0, t.x1);
    n.b = make_float4(t.y1, t.z1, t.x2, t.y2);
    n.d = make_float4(t.z2, sa, 0.f, 0.f);
    n.s = make_float4(sx, sy, sz, s3);
  } else {
    // a padding panel with zero strength far away contributes exactly zero
    cx = cy = cz = 1.0e18f;
    t2 = -1.0f;
    n.a = make_float4(1.0e18f, 1.0e18f, 1.0e18f, 1.0e18f);
    n.b = make_float4(1.0e18f, 1.0e18f, 1.0e18f, 1.0e18f);
    n.d = make_float4(1.0e18f, 1.0f, 0.f, 0.f);
    n.s = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (tiles) store_row(tiles, j, cx, cy, cz, t2, n.s.x, n.s.y, n.s.z, n.s.w);
  if (cen) cen[j] = make_float4(cx, cy, cz, t2);
  nearr[j] = n;
}

__device__ __forceinline__ void near_tri(const PanelNear& n, Tri& t, float& area) {
  t = Tri{n.a.x, n.a.y, n.a.z, n.a.w, n.b.x, n.b.y, n.b.z, n.b.w, n.d.x};
  area = n.d.y;
}

// partial sums of one split, or the sums into the outputs; SIGN: the sums are added
template <int NC, bool ACC, int TPT>
__device__ __forceinline__ void panel_store(const float (*v)[NC], const float (*hi)[NC], const float (*lo)[NC],
                                            int i0, int n, float* partial, int n_pad, const OutPtrs<float>& out) {
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    const int i = i0 + 32 * k;
    if (partial) {
      float* base = partial + (size_t)blockIdx.y * (ACC ? 2 : 1) * NC * n_pad;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        base[(size_t)c * n_pad + i] = ACC ? hi[k][c] : v[k][c];
        if (ACC) base[(size_t)(NC + c) * n_pad + i] = lo[k][c];
      }
    } else if (i < n) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (ACC) out.p[c][i] = (float)((double)out.p[c][i] + ((double)hi[k][c] + (double)lo[k][c]));
        else     out.p[c][i] += v[k][c];
      }
    }
  }
}

// panels_affect_points: TPT targets per thread, sweeping panel tiles
template <bool GRADS, bool SRC, bool ACC, int TPT>
__global__ void __launch_bounds__(kPW) k_panpt(const float4* __restrict__ tiles, const PanelNear* __restrict__ nearr,
                                               int ntiles, int tiles_per_split, int maxlev, int nt,
                                               const float* __restrict__ tx, const float* __restrict__ ty,
                                               const float* __restrict__ tz, float* partial, int nt_pad,
                                               OutPtrs<float> out) {
  constexpr int NC = GRADS ? 12 : 3;
  constexpr int NS = PanelSums<GRADS, SRC>::n;
  using Shared = WarpShared<NodeSums<GRADS, SRC, ACC>::n, TPT>;
  extern __shared__ __align__(16) char smem[];
  Shared& sh = *reinterpret_cast<Shared*>(smem);
  const int i0 = blockIdx.x * (kPW * TPT) + threadIdx.x;
  float px[TPT][3];
  float2 tt[TPT][3];
  bool live[TPT];
  float2 a[TPT][NS];
  float hi[TPT][NC], lo[TPT][NC];
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    const int i = i0 + 32 * k;
    live[k] = i < nt;
    px[k][0] = live[k] ? tx[i] : 0.f;
    px[k][1] = live[k] ? ty[i] : 0.f;
    px[k][2] = live[k] ? tz[i] : 0.f;
#pragma unroll
    for (int d = 0; d < 3; ++d) tt[k][d] = f2(px[k][d]);
#pragma unroll
    for (int c = 0; c < NS; ++c) a[k][c] = f2(0.f);
#pragma unroll
    for (int c = 0; c < NC; ++c) { hi[k][c] = 0.f; lo[k][c] = 0.f; }
  }
  // a node's point is its owner's target, its panel and strength are the swept ones
  auto fetch = [&](const uint2& nd, bool act, Tri& t, float& area, float& x, float& y, float& z, float& sx, float& sy,
                   float& sz, float& q) {
    const int o = (int)(nd.y & 31u), ko = (int)((nd.y >> 5) & 7u);
    x = y = z = 0.f;
#pragma unroll
    for (int k = 0; k < TPT; ++k) {
      const float vx = __shfl_sync(0xffffffffu, px[k][0], o), vy = __shfl_sync(0xffffffffu, px[k][1], o),
                  vz = __shfl_sync(0xffffffffu, px[k][2], o);
      if (k == ko) { x = vx; y = vy; z = vz; }
    }
    const PanelNear n = nearr[act ? nd.x : 0u];
    near_tri(n, t, area);
    sx = n.s.x; sy = n.s.y; sz = n.s.z; q = n.s.w;
  };
  const int t0 = blockIdx.y * tiles_per_split;
  const int t1 = min(ntiles, t0 + tiles_per_split);
  sweep_panels<GRADS, SRC, ACC, TPT, 1, false>(tiles, t0, t1, maxlev, sh, tt, nullptr, live, a, hi, lo, fetch);
  float v[TPT][NC];
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    float w[NS];
#pragma unroll
    for (int c = 0; c < NS; ++c) w[c] = a[k][c].x + a[k][c].y;
    panel_fold<GRADS, SRC>(w);
#pragma unroll
    for (int c = 0; c < NC; ++c) v[k][c] = w[c];
  }
  panel_store<NC, ACC, TPT>(v, hi, lo, i0, nt, partial, nt_pad, out);
}

// points_affect_panels: TPT target panels per thread, sweeping particle tiles; the panel is the
// subdivided "source" with the particle's strength, evaluated at the particle and subtracted
// (Influence.h:1209-1212): with d = centroid - particle the sum has that sign already.
template <bool ACC, int TPT>
__global__ void __launch_bounds__(kPW) k_ptpan(const float4* __restrict__ cen, const PanelNear* __restrict__ nearr,
                                               int np, const float4* __restrict__ tiles, int ntiles,
                                               int tiles_per_split, int maxlev, float* partial, int np_pad,
                                               OutPtrs<float> out) {
  using Shared = WarpShared<3, TPT>;
  extern __shared__ __align__(16) char smem[];
  Shared& sh = *reinterpret_cast<Shared*>(smem);
  const int w0 = blockIdx.x * (kPW * TPT);
  const int i0 = w0 + threadIdx.x;
  float2 tt[TPT][3], a[TPT][3];
  float own2[TPT], hi[TPT][3], lo[TPT][3], v[TPT][3];
  bool live[TPT];
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    const int i = i0 + 32 * k;
    live[k] = i < np;
    const float4 c = cen[i];
    tt[k][0] = f2(c.x); tt[k][1] = f2(c.y); tt[k][2] = f2(c.z);
    own2[k] = c.w;
#pragma unroll
    for (int d = 0; d < 3; ++d) { a[k][d] = f2(0.f); hi[k][d] = 0.f; lo[k][d] = 0.f; }
  }
  // a node's panel is its owner's, its point and strength are the swept particle's
  auto fetch = [&](const uint2& nd, bool act, Tri& t, float& area, float& x, float& y, float& z, float& sx, float& sy,
                   float& sz, float& q) {
    const PanelNear n = nearr[w0 + 32 * (int)((nd.y >> 5) & 7u) + (int)(nd.y & 31u)];
    near_tri(n, t, area);
    const unsigned j = act ? nd.x : 0u;
    const float* b = reinterpret_cast<const float*>(tiles + (size_t)(j / kPW) * (kRows * kPW / 2) + (j % kPW) / 2) + (j & 1u);
    constexpr int R = 4 * (kPW / 2);
    x = -b[0]; y = -b[2]; z = -b[R];
    sx = b[2 * R]; sy = b[2 * R + 2]; sz = b[3 * R];
    q = 0.f;
  };
  const int t0 = blockIdx.y * tiles_per_split;
  const int t1 = min(ntiles, t0 + tiles_per_split);
  sweep_panels<false, false, ACC, TPT, -1, true>(tiles, t0, t1, maxlev, sh, tt, own2, live, a, hi, lo, fetch);
#pragma unroll
  for (int k = 0; k < TPT; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) v[k][c] = a[k][c].x + a[k][c].y;
  panel_store<3, ACC, TPT>(v, hi, lo, i0, np, partial, np_pad, out);
}

__global__ void k_pack_particles(int n, int n_pad, const float* __restrict__ x, const float* __restrict__ y,
                                 const float* __restrict__ z, const float* __restrict__ sx,
                                 const float* __restrict__ sy, const float* __restrict__ sz, float4* tiles) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_pad) return;
  if (j < n) store_row(tiles, j, x[j], y[j], z[j], 0.f, sx[j], sy[j], sz[j], 0.f);
  else       store_row(tiles, j, 1.0e18f, 1.0e18f, 1.0e18f, 0.f, 0.f, 0.f, 0.f, 0.f);
}

template <bool GRADS, bool SRC, bool ACC, int TPT>
static void panpt_kernel_of(int maxlev, const void** k, size_t* smem) {
  *k = (const void*)&k_panpt<GRADS, SRC, ACC, TPT>;
  *smem = WarpShared<NodeSums<GRADS, SRC, ACC>::n, TPT>::bytes(maxlev);
}
template <bool SRC, bool ACC>
static void panpt_kernel(bool grads, int tpt, int maxlev, const void** k, size_t* smem) {
  if (grads)         panpt_kernel_of<true, SRC, ACC, 1>(maxlev, k, smem);
  else if (tpt == 2) panpt_kernel_of<false, SRC, ACC, 2>(maxlev, k, smem);
  else               panpt_kernel_of<false, SRC, ACC, 1>(maxlev, k, smem);
}
template <int TPT>
static void ptpan_kernel(bool comp, int maxlev, const void** k, size_t* smem) {
  *k = comp ? (const void*)&k_ptpan<true, TPT> : (const void*)&k_ptpan<false, TPT>;
  *smem = WarpShared<3, TPT>::bytes(maxlev);
}

// Splits the swept tiles over blockIdx.y: up to 4 waves of resident blocks (their near work
// differs), whole waves when a split would fall below 8 tiles (256 elements: shorter ones spend
// their time on the queues' last, partly filled batches and on the partial sums), and shorter
// ones down to single tiles where the GPU would not be filled otherwise.
static void plan_split(int nunits_outer, int ninner_tiles, int slots, int* nsplit, int* tps) {
  int least = 8;
  while (least > 1 && (long)nunits_outer * (ninner_tiles / least) < slots) least /= 2;
  const long cap = std::max(1, ninner_tiles / least);
  long ns = (4L * slots + nunits_outer - 1) / nunits_outer;
  if (ns > cap) {
    const long waves = std::max(1L, nunits_outer * cap / slots);
    ns = std::max(1L, std::min(cap, waves * slots / nunits_outer));
  }
  *tps = (int)((ninner_tiles + ns - 1) / ns);
  *nsplit = (ninner_tiles + *tps - 1) / *tps;
}
// Targets (panels) per thread: two for velocities, whose sums leave the registers for it,
// unless one is needed to fill the GPU (about 20 resident blocks per SM) with 8-tile splits
static int targets_per_thread(bool grads, int n, int ntiles, int num_sms) {
  if (grads) return 1;
  return (long)((n + 2 * kPW - 1) / (2 * kPW)) * (ntiles / 8) >= 20L * num_sms ? 2 : 1;
}

}  // namespace o3g

using namespace o3g;

extern "C" int32_t o3g_panels_affect_points(int32_t prec, int32_t mem, int32_t maxlev, int32_t nn, const float* nx,
                                            const float* ny, const float* nz, int32_t np, const uint32_t* idx,
                                            const float* area, const float* tsx, const float* tsy, const float* tsz,
                                            const float* sss, int32_t nt, const float* tx, const float* ty,
                                            const float* tz, float* tu, float* tv, float* tw, float* const* tug,
                                            void* stream) {
  if ((mem != O3G_MEM_HOST && mem != O3G_MEM_DEVICE) || maxlev < 0 || maxlev > kMaxLev || nn < 0 || np < 0 ||
      nt < 0 || (prec != O3G_PREC_PLAIN && prec != O3G_PREC_COMPENSATED)) {
    set_error("panels_affect_points: bad precision (PLAIN or COMPENSATED), mem, maxlev (0..6) or negative count");
    return O3G_ERR_INVALID_ARG;
  }
  const bool comp = prec == O3G_PREC_COMPENSATED;
  if (np > 0 && (!nx || !ny || !nz || !idx || !area || !tsx || !tsy || !tsz)) {
    set_error("panels_affect_points: null panel array");
    return O3G_ERR_INVALID_ARG;
  }
  if (nt > 0 && (!tx || !ty || !tz || !tu || !tv || !tw)) {
    set_error("panels_affect_points: null target array");
    return O3G_ERR_INVALID_ARG;
  }
  const bool grads = tug != nullptr;
  if (grads && nt > 0)
    for (int k = 0; k < 9; ++k)
      if (!tug[k]) { set_error("panels_affect_points: null gradient component"); return O3G_ERR_INVALID_ARG; }
  if (np == 0 || nt == 0) return O3G_OK;
  if (mem == O3G_MEM_HOST) {
    for (int j = 0; j < 3 * np; ++j)
      if (idx[j] >= (uint32_t)nn) { set_error("panels_affect_points: panel index out of range"); return O3G_ERR_INVALID_ARG; }
  }
  DeviceFacts df;
  O3G_TRY(device_facts(&df));
  cudaStream_t st = (cudaStream_t)stream;
  const int NC = grads ? 12 : 3;
  const int ntiles = (np + kPW - 1) / kPW, np_pad = ntiles * kPW;
  const int tpt = targets_per_thread(grads, nt, ntiles, df.num_sms);
  const int tb = (nt + kPW * tpt - 1) / (kPW * tpt), nt_pad = tb * kPW * tpt;
  int nb = 0;
  const void* kp;
  size_t smem;
  if (sss) comp ? panpt_kernel<true, true>(grads, tpt, maxlev, &kp, &smem) : panpt_kernel<true, false>(grads, tpt, maxlev, &kp, &smem);
  else     comp ? panpt_kernel<false, true>(grads, tpt, maxlev, &kp, &smem) : panpt_kernel<false, false>(grads, tpt, maxlev, &kp, &smem);
  O3G_TRY(occupancy_blocks(kp, kPW, &nb, smem));
  const int PC = comp ? 2 * NC : NC;   // partial components per split
  int nsplit = 1, tps = ntiles;
  plan_split(tb, ntiles, nb * df.num_sms, &nsplit, &tps);

  const size_t tile_f4 = (size_t)ntiles * (kRows * kPW / 2);
  size_t bytes = align_up(tile_f4 * sizeof(float4)) + align_up((size_t)np_pad * sizeof(PanelNear));
  if (nsplit > 1) bytes += align_up((size_t)nsplit * PC * nt_pad * sizeof(float));
  size_t staging = 0;
  if (mem == O3G_MEM_HOST)
    staging = 3 * align_up((size_t)nn * 4) + align_up((size_t)np * 12) + 4 * align_up((size_t)np * 4) +
              (sss ? align_up((size_t)np * 4) : 0) + 3 * align_up((size_t)nt * 4) + NC * align_up((size_t)nt * 4);
  Workspace* ws = nullptr;
  O3G_TRY(workspace_get(st, staging + bytes, &ws));
  Carve cv(ws->base);
  const float *dnx = nx, *dny = ny, *dnz = nz, *dar = area, *dtsx = tsx, *dtsy = tsy, *dtsz = tsz, *dsss = sss;
  const float *dtx = tx, *dty = ty, *dtz = tz;
  const uint32_t* didx = idx;
  OutPtrs<float> out;
  out.p[0] = tu; out.p[1] = tv; out.p[2] = tw;
  for (int k = 0; k < 9; ++k) out.p[3 + k] = grads ? tug[k] : nullptr;
  OutPtrs<float> hout = out;
  if (mem == O3G_MEM_HOST) {
    auto up = [&](const float* h, size_t n) -> const float* {
      float* d = cv.take<float>(n);
      cudaMemcpyAsync(d, h, n * 4, cudaMemcpyHostToDevice, st);
      return d;
    };
    dnx = up(nx, nn); dny = up(ny, nn); dnz = up(nz, nn);
    uint32_t* di = cv.take<uint32_t>((size_t)3 * np);
    O3G_CUDA_TRY(cudaMemcpyAsync(di, idx, (size_t)np * 12, cudaMemcpyHostToDevice, st));
    didx = di;
    dar = up(area, np); dtsx = up(tsx, np); dtsy = up(tsy, np); dtsz = up(tsz, np);
    if (sss) dsss = up(sss, np);
    dtx = up(tx, nt); dty = up(ty, nt); dtz = up(tz, nt);
    for (int c = 0; c < NC; ++c) out.p[c] = const_cast<float*>(up(hout.p[c], nt));
    O3G_CUDA_TRY(cudaGetLastError());
  }
  Carve cw(ws->base + staging);
  float4* tiles = cw.take<float4>(tile_f4);
  PanelNear* nearr = cw.take<PanelNear>(np_pad);
  float* partial = nsplit > 1 ? cw.take<float>((size_t)nsplit * PC * nt_pad) : nullptr;
  k_pack_panels<<<(np_pad + 255) / 256, 256, 0, st>>>(np, dnx, dny, dnz, didx, dar, dtsx, dtsy, dtsz, dsss, np_pad,
                                                     maxlev, tiles, nullptr, nearr);
  note_launch();
  dim3 grid(tb, nsplit);
  KernelTimer& tm = thread_timer();
  tm.begin(st);
  {
    int ntl = ntiles, mxl = maxlev, ntt = nt, ntp = nt_pad;
    void* args[] = {&tiles, &nearr, &ntl, &tps, &mxl, &ntt, &dtx, &dty, &dtz, &partial, &ntp, &out};
    O3G_CUDA_TRY(cudaLaunchKernel(kp, grid, dim3(kPW), args, smem, st));
  }
  note_launch();
  tm.end(st);
  if (nsplit > 1) {
    if (comp) {
      if (grads) launch_reduce<12, true, float, float>(partial, nsplit, nt, nt_pad, out, nullptr, st);
      else       launch_reduce<3, true, float, float>(partial, nsplit, nt, nt_pad, out, nullptr, st);
    } else {
      if (grads) launch_reduce<12, false, float, float>(partial, nsplit, nt, nt_pad, out, nullptr, st);
      else       launch_reduce<3, false, float, float>(partial, nsplit, nt, nt_pad, out, nullptr, st);
    }
  }
  O3G_CUDA_TRY(cudaGetLastError());
  if (mem == O3G_MEM_HOST) {
    for (int c = 0; c < NC; ++c)
      O3G_CUDA_TRY(cudaMemcpyAsync(hout.p[c], out.p[c], (size_t)nt * 4, cudaMemcpyDeviceToHost, st));
    O3G_CUDA_TRY(cudaStreamSynchronize(st));
  }
  return O3G_OK;
}

extern "C" int32_t o3g_points_affect_panels(int32_t prec, int32_t mem, int32_t maxlev, int32_t ns, const float* sx,
                                            const float* sy, const float* sz, const float* ssx, const float* ssy,
                                            const float* ssz, int32_t nn, const float* nx, const float* ny,
                                            const float* nz, int32_t np, const uint32_t* idx, const float* area,
                                            float* pu, float* pv, float* pw, void* stream) {
  if ((mem != O3G_MEM_HOST && mem != O3G_MEM_DEVICE) || maxlev < 0 || maxlev > kMaxLev || nn < 0 || np < 0 ||
      ns < 0 || (prec != O3G_PREC_PLAIN && prec != O3G_PREC_COMPENSATED)) {
    set_error("points_affect_panels: bad precision (PLAIN or COMPENSATED), mem, maxlev (0..6) or negative count");
    return O3G_ERR_INVALID_ARG;
  }
  const bool comp = prec == O3G_PREC_COMPENSATED;
  if (ns > 0 && (!sx || !sy || !sz || !ssx || !ssy || !ssz)) {
    set_error("points_affect_panels: null particle array");
    return O3G_ERR_INVALID_ARG;
  }
  if (np > 0 && (!nx || !ny || !nz || !idx || !area || !pu || !pv || !pw)) {
    set_error("points_affect_panels: null panel array");
    return O3G_ERR_INVALID_ARG;
  }
  if (np == 0 || ns == 0) return O3G_OK;
  if (mem == O3G_MEM_HOST) {
    for (int j = 0; j < 3 * np; ++j)
      if (idx[j] >= (uint32_t)nn) { set_error("points_affect_panels: panel index out of range"); return O3G_ERR_INVALID_ARG; }
  }
  DeviceFacts df;
  O3G_TRY(device_facts(&df));
  cudaStream_t st = (cudaStream_t)stream;
  const int ptiles = (ns + kPW - 1) / kPW, ns_pad = ptiles * kPW;
  const int tpt = targets_per_thread(false, np, ptiles, df.num_sms);
  const int tb = (np + kPW * tpt - 1) / (kPW * tpt), np_pad = tb * kPW * tpt;
  int nb = 0;
  const void* kp;
  size_t smem;
  if (tpt == 2) ptpan_kernel<2>(comp, maxlev, &kp, &smem);
  else          ptpan_kernel<1>(comp, maxlev, &kp, &smem);
  O3G_TRY(occupancy_blocks(kp, kPW, &nb, smem));
  int nsplit = 1, tps = ptiles;
  plan_split(tb, ptiles, nb * df.num_sms, &nsplit, &tps);
  const int PC = comp ? 6 : 3;
  const size_t tile_f4 = (size_t)ptiles * (kRows * kPW / 2);
  size_t bytes = align_up((size_t)np_pad * sizeof(float4)) + align_up((size_t)np_pad * sizeof(PanelNear)) +
                 align_up(tile_f4 * sizeof(float4));
  if (nsplit > 1) bytes += align_up((size_t)nsplit * PC * np_pad * sizeof(float));
  size_t staging = 0;
  if (mem == O3G_MEM_HOST)
    staging = 3 * align_up((size_t)nn * 4) + align_up((size_t)np * 12) + align_up((size_t)np * 4) +
              6 * align_up((size_t)ns * 4) + 3 * align_up((size_t)np * 4);
  Workspace* ws = nullptr;
  O3G_TRY(workspace_get(st, staging + bytes, &ws));
  Carve cv(ws->base);
  const float *dnx = nx, *dny = ny, *dnz = nz, *dar = area;
  const float *dsx = sx, *dsy = sy, *dsz = sz, *dssx = ssx, *dssy = ssy, *dssz = ssz;
  const uint32_t* didx = idx;
  OutPtrs<float> out;
  out.p[0] = pu; out.p[1] = pv; out.p[2] = pw;
  OutPtrs<float> hout = out;
  if (mem == O3G_MEM_HOST) {
    auto up = [&](const float* h, size_t n) -> const float* {
      float* d = cv.take<float>(n);
      cudaMemcpyAsync(d, h, n * 4, cudaMemcpyHostToDevice, st);
      return d;
    };
    dnx = up(nx, nn); dny = up(ny, nn); dnz = up(nz, nn);
    uint32_t* di = cv.take<uint32_t>((size_t)3 * np);
    O3G_CUDA_TRY(cudaMemcpyAsync(di, idx, (size_t)np * 12, cudaMemcpyHostToDevice, st));
    didx = di;
    dar = up(area, np);
    dsx = up(sx, ns); dsy = up(sy, ns); dsz = up(sz, ns);
    dssx = up(ssx, ns); dssy = up(ssy, ns); dssz = up(ssz, ns);
    for (int c = 0; c < 3; ++c) out.p[c] = const_cast<float*>(up(hout.p[c], np));
    O3G_CUDA_TRY(cudaGetLastError());
  }
  Carve cw(ws->base + staging);
  float4* cen = cw.take<float4>(np_pad);
  PanelNear* nearr = cw.take<PanelNear>(np_pad);
  float4* tiles = cw.take<float4>(tile_f4);
  float* partial = nsplit > 1 ? cw.take<float>((size_t)nsplit * PC * np_pad) : nullptr;
  k_pack_panels<<<(np_pad + 255) / 256, 256, 0, st>>>(np, dnx, dny, dnz, didx, dar, nullptr, nullptr, nullptr, nullptr,
                                                     np_pad, maxlev, nullptr, cen, nearr);
  k_pack_particles<<<(ns_pad + 255) / 256, 256, 0, st>>>(ns, ns_pad, dsx, dsy, dsz, dssx, dssy, dssz, tiles);
  note_launch(2);
  KernelTimer& tm = thread_timer();
  tm.begin(st);
  {
    int npa = np, ptl = ptiles, mxl = maxlev, npp = np_pad;
    void* args[] = {&cen, &nearr, &npa, &tiles, &ptl, &tps, &mxl, &partial, &npp, &out};
    O3G_CUDA_TRY(cudaLaunchKernel(kp, dim3(tb, nsplit), dim3(kPW), args, smem, st));
  }
  note_launch();
  tm.end(st);
  if (nsplit > 1) {
    if (comp) launch_reduce<3, true, float, float>(partial, nsplit, np, np_pad, out, nullptr, st);
    else      launch_reduce<3, false, float, float>(partial, nsplit, np, np_pad, out, nullptr, st);
  }
  O3G_CUDA_TRY(cudaGetLastError());
  if (mem == O3G_MEM_HOST) {
    for (int c = 0; c < 3; ++c)
      O3G_CUDA_TRY(cudaMemcpyAsync(hout.p[c], out.p[c], (size_t)np * 4, cudaMemcpyDeviceToHost, st));
    O3G_CUDA_TRY(cudaStreamSynchronize(st));
  }
  return O3G_OK;
}
