// pm_vanka_patch.cu — cell-Vanka sweeps of one-block Q2 hexahedral levels
// from a per-cell packed copy of the velocity rows.
//
// One colour of a sweep (CellVanka, src/FE/NSE_MGLevel4.C:1653-2087, in the
// colour-block order of CellVanka_GPU, src/FE/NSE_CellVanka.cu:1748-2555) is
// one launch of persistent CTAs: local residual r = f - K u on
// the cell's 85 DOFs, block elimination (pm_vanka_schur.cu) and the update.
//
// Why a packed copy.  The rows of a cell couple to the 343 nodes of the cell
// and its 26 neighbours: 2,197 A entries and 500 x 3 BT entries.  Walking the
// CSR rows with one warp (pm_vanka.cu) costs a column index per entry, seven
// serial row steps of dependent loads and one gather per entry through L1; a
// colour launch took 20-30 us however few cells the level had, and
// 0.255 + 0.047 ms at 64^3.  Here eight lanes own each row, all 27 rows at
// once (seven warps); the values lie in the order in which the lanes use them
// (coalesced, no column indices), the patch's nodes are gathered once into
// shared memory, and nothing but that gather depends on the previous colour,
// so every other load is issued before the launch waits for its predecessor
// (programmatic dependent launch).
//
// Order of operations.  A row's sums run over the lanes and entries in the
// order of k_vanka_residual_rows<float,1,1,8,27,true,true> (entry j of a row
// belongs to lane j % 8; eight A entries, the BT entries, the other A
// entries; a butterfly over the lanes), and the block solve in the order of
// k_schur_apply, so FP32 sweeps are equal to theirs bit for bit.
//
// Patch.  Each cell keeps the sorted list of its patch's nodes; where the
// nodes lie in shared memory and where entry j of row r finds its node is a
// pattern that cells with the same neighbourhood and numbering order share
// (one for all inner cells of a uniform mesh).  The places are chosen at
// set-up (patch_places) so that the eight lanes of a row read eight different
// 16-byte bank groups: in list order a row's runs of five nodes collided
// pairwise.  Meshes whose cells have more than one
// neighbour beyond a face, edge or vertex, or whose rows do not fit the lanes
// (128 / 80 / 48 columns on vertex / edge / other rows) keep the CSR kernels.
//
// Current values.  Cells of one colour share no node, but a cell's patch
// reaches nodes that other cells of its colour update.  Every node that lies
// in more than one cell therefore has two copies: an update reads one and
// writes the other, and which copy is current at the turn of a colour follows
// from the colours of the node's cells alone (bit 0 of the patch entry).  A
// node in an odd number > 1 of cells changes sides every sweep (bit 1); a
// node or pressure of one cell is read by no other cell of its colour and is
// updated in place.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <climits>
#include <cstdint>
#include <vector>

#include "pm_bulk.cuh"
#include "pm_chain.cuh"
#include "pm_kernels.h"

namespace pm {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kPatchThreads = 256;  // warps 0-1 vertex rows, 2-4 edges, 5-6 the rest, 7 block solve
constexpr int kRowLanes = 224;
constexpr int kZeroSlot = kPatchNodes;  // a node that is zero: padding entries point to it
constexpr int kZeroP = 27 * NP_LOC;
// offsets of the packed values of a cell (see PatchPos)
constexpr int kOffE = 64 * 16, kOffE2 = kOffE + 96 * 8, kOffR = kOffE + 96 * 10,
              kOffR2 = kOffR + 64 * 4, kOffTV = kOffR + 64 * 6, kOffTE = kOffTV + 64 * 12,
              kOffTR = kOffTE + 96 * 6;
static_assert(kOffTR + 64 * 3 == kPatchValues, "packed values of a cell");

// rows in the order of their stencil size (8 vertices, 12 edges, 6 faces, centre)
__constant__ unsigned char c_rows[28] = {0,  2,  6,  8,  18, 20, 24, 26, 1,  3,  5,  7,  9, 11,
                                         15, 17, 19, 21, 23, 25, 4,  10, 12, 14, 16, 22, 13, 13};

// entries per lane of the row with index k (in c_rows order)
__device__ __forceinline__ int row_cap(int k) { return k < 8 ? 16 : (k < 20 ? 10 : 6); }
__device__ __forceinline__ int bt_cap(int k) { return k < 8 ? 4 : (k < 20 ? 2 : 1); }

// position of A entry q of lane li (0..223: row li / 8, lane li % 8)
__device__ __forceinline__ int a_pos(int li, int q) {
  if (li < 64) return ((q >> 2) * 64 + li) * 4 + (q & 3);
  if (li < 160) return q < 8 ? kOffE + ((q >> 2) * 96 + li - 64) * 4 + (q & 3)
                             : kOffE2 + (li - 64) * 2 + (q & 1);
  return q < 4 ? kOffR + (li - 160) * 4 + q : kOffR2 + (li - 160) * 2 + (q & 1);
}
// position of component c of BT entry q of lane li
__device__ __forceinline__ int bt_pos(int li, int q, int c) {
  if (li < 64) return kOffTV + (c * 64 + li) * 4 + q;
  if (li < 160) return kOffTE + (c * 96 + li - 64) * 2 + q;
  return kOffTR + c * 64 + li - 160;
}

}  // namespace

// Where the entries of a cell's rows find their nodes, pressures and B values.
struct PatchPattern {
  uint16_t slot[kRowLanes][16];  // A entry: 16 x place of its node in shared memory
  uint8_t bt[kRowLanes][4];      // BT entry: 4 * neighbour + mode
  uint8_t bj[32][4];             // B row lane / 8, entry lane % 8 + 8 q: own node
  uint16_t own[32];              // own node: 16 x its place
  uint16_t place[kPatchIds - 48];  // patch list entry: its place
};
static_assert(sizeof(PatchPattern) == kPatchPatternBytes, "pattern size");

namespace {

// Current values of a node: three components (and a pad) on 16- or 32-byte
// boundaries.  Reads go to L2: the previous launch of the chain may still
// have been writing when this one started.
template <typename T>
struct Node;
template <>
struct Node<float> {
  float4 v;
  static __device__ __forceinline__ Node load(const void *p, size_t i) {
    return Node{__ldcg(reinterpret_cast<const float4 *>(p) + i)};
  }
  __device__ __forceinline__ void store(void *p, size_t i) const {
    reinterpret_cast<float4 *>(p)[i] = v;
  }
};
template <>
struct Node<double> {
  double2 a, b;
  static __device__ __forceinline__ Node load(const void *p, size_t i) {
    const double2 *q = reinterpret_cast<const double2 *>(p) + 2 * i;
    return Node{__ldcg(q), __ldcg(q + 1)};
  }
  __device__ __forceinline__ void store(void *p, size_t i) const {
    double2 *q = reinterpret_cast<double2 *>(p) + 2 * i;
    q[0] = a;
    q[1] = b;
  }
};
__device__ __forceinline__ Node<float> make_node(float x, float y, float z) {
  return Node<float>{make_float4(x, y, z, 0.f)};
}
__device__ __forceinline__ Node<double> make_node(double x, double y, double z) {
  return Node<double>{make_double2(x, y), make_double2(z, 0.0)};
}
__device__ __forceinline__ void comps(const Node<float> &n, float &x, float &y, float &z) {
  x = n.v.x;
  y = n.v.y;
  z = n.v.z;
}
__device__ __forceinline__ void comps(const Node<double> &n, double &x, double &y, double &z) {
  x = n.a.x;
  y = n.a.y;
  z = n.b.x;
}

// triples in shared memory: one 16-byte load in FP32, 16 + 8 bytes in FP64
template <typename T, int N>
struct Tri;
template <int N>
struct Tri<float, N> {
  float4 v[N];
  __device__ __forceinline__ void get(int i, float &x, float &y, float &z) const {
    const float4 q = v[i];
    x = q.x;
    y = q.y;
    z = q.z;
  }
  __device__ __forceinline__ void at(unsigned off, float &x, float &y, float &z) const {
    const float4 q = *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(v) + off);
    x = q.x;
    y = q.y;
    z = q.z;
  }
  __device__ __forceinline__ float &ref(int i, int c) {
    return reinterpret_cast<float *>(v)[4 * i + c];
  }
  __device__ __forceinline__ void set(int i, float x, float y, float z) {
    v[i] = make_float4(x, y, z, 0.f);
  }
};
template <int N>
struct Tri<double, N> {
  double2 v[N];
  double w[N];
  __device__ __forceinline__ void get(int i, double &x, double &y, double &z) const {
    const double2 q = v[i];
    x = q.x;
    y = q.y;
    z = w[i];
  }
  __device__ __forceinline__ void at(unsigned off, double &x, double &y, double &z) const {
    const double2 q = *reinterpret_cast<const double2 *>(reinterpret_cast<const char *>(v) + off);
    x = q.x;
    y = q.y;
    z = *reinterpret_cast<const double *>(reinterpret_cast<const char *>(w) + (off >> 1));
  }
  __device__ __forceinline__ double &ref(int i, int c) {
    return c < 2 ? reinterpret_cast<double *>(v)[2 * i + c] : w[i];
  }
  __device__ __forceinline__ void set(int i, double x, double y, double z) {
    v[i] = make_double2(x, y);
    w[i] = z;
  }
};

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// named barriers of a CTA
enum { kBarRows = 1, kBarFull = 2, kBarFree = 4 };  // kBarFull, kBarFree: two each
__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("barrier.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// a0 b0 + a1 b1 + a2 b2, contracted in FP32 as the compiler does in
// k_schur_apply and in the pressure rows of the row-group kernel
template <typename T>
__device__ __forceinline__ T dot3(T a0, T b0, T a1, T b1, T a2, T b2) {
  if constexpr (sizeof(T) == 4)
    return __fmaf_rn(a2, b2, __fmaf_rn(a0, b0, __fmul_rn(a1, b1)));
  else
    return a0 * b0 + a1 * b1 + a2 * b2;
}

template <typename T>
__device__ __forceinline__ void lds4(const T *p, T (&o)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  } else {
    const double2 a = reinterpret_cast<const double2 *>(p)[0],
                  b = reinterpret_cast<const double2 *>(p)[1];
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
  }
}
template <typename T>
__device__ __forceinline__ void lds2(const T *p, T &x, T &y) {
  if constexpr (sizeof(T) == 4) {
    const float2 v = *reinterpret_cast<const float2 *>(p);
    x = v.x;
    y = v.y;
  } else {
    const double2 v = *reinterpret_cast<const double2 *>(p);
    x = v.x;
    y = v.y;
  }
}

// Sum of one row's entries for one lane of its eight: entries q of lane li in
// the order of the row-group kernel.  VAL: the cell's packed values; u, p: the
// patch; s0, s1, bts: places of the lane's nodes and pressures.
template <typename T, typename U>
__device__ __forceinline__ void row_sum(int group, int li, const T *V, const U &u, const T *p,
                                        const uint4 &s0, const uint4 &s1, unsigned bts, T &c0,
                                        T &c1, T &c2) {
  c0 = c1 = c2 = T(0);
  auto a_entry = [&](unsigned off, T v) {
    T x, y, z;
    u.at(off, x, y, z);
    c0 += v * x;
    c1 += v * y;
    c2 += v * z;
  };
  auto a_four = [&](unsigned lo, unsigned hi, const T *q) {
    T v[4];
    lds4(q, v);
    a_entry(lo & 0xffff, v[0]);
    a_entry(lo >> 16, v[1]);
    a_entry(hi & 0xffff, v[2]);
    a_entry(hi >> 16, v[3]);
  };
  auto a_two = [&](unsigned o, const T *q) {
    T v0, v1;
    lds2(q, v0, v1);
    a_entry(o & 0xffff, v0);
    a_entry(o >> 16, v1);
  };
  auto bt_entry = [&](int q, T v0, T v1, T v2) {
    const T pc = p[(bts >> (8 * q)) & 0xff];
    c0 += v0 * pc;
    c1 += v1 * pc;
    c2 += v2 * pc;
  };
  if (group < 2) {  // vertex rows
    V += 4 * li;
    a_four(s0.x, s0.y, V);
    a_four(s0.z, s0.w, V + 256);
    T g0[4], g1[4], g2[4];
    lds4(V + kOffTV, g0);
    lds4(V + kOffTV + 256, g1);
    lds4(V + kOffTV + 512, g2);
#pragma unroll
    for (int q = 0; q < 4; ++q) bt_entry(q, g0[q], g1[q], g2[q]);
    a_four(s1.x, s1.y, V + 512);
    a_four(s1.z, s1.w, V + 768);
  } else if (group < 5) {  // edge rows
    li -= 64;
    a_four(s0.x, s0.y, V + kOffE + 4 * li);
    a_four(s0.z, s0.w, V + kOffE + 4 * (96 + li));
    T g0[2], g1[2], g2[2];
    lds2(V + kOffTE + 2 * li, g0[0], g0[1]);
    lds2(V + kOffTE + 2 * li + 192, g1[0], g1[1]);
    lds2(V + kOffTE + 2 * li + 384, g2[0], g2[1]);
    bt_entry(0, g0[0], g1[0], g2[0]);
    bt_entry(1, g0[1], g1[1], g2[1]);
    a_two(s1.x, V + kOffE2 + 2 * li);
  } else {  // face rows and the centre
    li -= 160;
    a_four(s0.x, s0.y, V + kOffR + 4 * li);
    a_two(s0.z, V + kOffR2 + 2 * li);
    bt_entry(0, V[kOffTR + li], V[kOffTR + 64 + li], V[kOffTR + 128 + li]);
  }
}

// Pressure rows of a cell: lanes 8 k .. 8 k + 7 return the sum of row k; bj,
// o01, o23: the row's own nodes and their places (D in the order of the CSR
// row)
template <typename T, typename U>
__device__ __forceinline__ T pressure_sum(int sub, const T *fac, const U &u, unsigned bj,
                                          unsigned o01, unsigned o23) {
  T c = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int jn = (bj >> (8 * q)) & 0xff;
    const bool live = jn < NU_LOC;
    const T *D = fac + Schur<1>::offD + sub * 3 * NU_LOC + (live ? jn : 0);
    T g0, g1, g2;
    u.at(((q < 2 ? o01 : o23) >> (16 * (q & 1))) & 0xffff, g0, g1, g2);
    const T d0 = live ? D[0] : T(0), d1 = live ? D[NU_LOC] : T(0),
            d2 = live ? D[2 * NU_LOC] : T(0);
    c += dot3(d0, g0, d1, g1, d2, g2);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
  return c;
}
template <typename P>
__device__ __forceinline__ void pressure_pattern(const P &pat, int lane, unsigned &bj,
                                                 unsigned &o01, unsigned &o23) {
  bj = __ldg(reinterpret_cast<const unsigned *>(pat.bj[lane]));
  unsigned o[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) o[q] = __ldg(&pat.own[(bj >> (8 * q)) & 0xff]);
  o01 = o[0] | (o[1] << 16);
  o23 = o[2] | (o[3] << 16);
}

// copy of a patch entry's node that is current at this colour's turn
__device__ __forceinline__ size_t node_at(int e, int odd, int nu) {
  return (size_t)((e ^ ((e >> 1) & odd)) & 1) * nu + (e >> 2);
}

// 16 bytes global -> shared, asynchronous, through L2
__device__ __forceinline__ void async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// bounded wait for a copy after a wait for it ran out
__device__ __forceinline__ void drain(uint64_t *bar, int phase) {
  for (int it = 0; it < kMaxPolls; ++it)
    if (mbar_test_wait(bar, phase & 1)) break;
}

// ------------------------------------------------------------------ FP32 ---
struct Smem32 {
  float values[2][kPatchValues];        // packed rows of this cell and the next
  float fac[2][Schur<1>::stride];       // factors of this cell and the next
  int ids[4][kPatchIds];                // patch lists, up to three cells ahead
  Tri<float, kPatchNodes + 1> u[3];     // current values of a patch, then a zero
  float4 p[3][28];                      // pressures of a cell and its neighbours, then zeros
  float4 f[3][28];                      // right-hand side: own nodes, then the pressure part
  Tri<float, NU_LOC> r[2];              // velocity part of the local residual
  float rp[2][NP_LOC];
  uint64_t vbar[2], fbar[2], ibar[4];
};
constexpr int kCtas32 = 3;  // resident CTAs per SM (67 KB of shared memory each)

// Persistent CTAs, each walking the colour's cells with a stride.  Warps 0..6
// form a cell's local residual; warp 7 solves the cell before it, writes its
// update and starts the bulk copies: packed rows (15.6 KB) and factors
// (5.6 KB) two cells ahead, patch lists four ahead.  The gathers of current
// values, which no cell of this colour changes, are 16-byte asynchronous
// copies into shared memory two cells ahead: one cell ahead (in registers or
// in a second buffer) left their latency exposed.
// Bound by HBM and by shared-memory wavefronts on large levels, by the chain
// gather -> sums -> solve -> update on small ones.  LIMITED: polls of a wait as
// the caller says; with the number in a register instead of a constant a solve
// at 8^3 took 3.42 instead of 3.38 ms.
template <bool LIMITED>
__global__ void __launch_bounds__(kPatchThreads, kCtas32) k_patch_sweep32(
    PatchLevel<float> L, const int *__restrict__ list, int n, const float *__restrict__ factors,
    float damp, int odd, int *err, int limit) {
  using S1 = Schur<1>;
  extern __shared__ __align__(16) unsigned char raw[];
  Smem32 &sm = *reinterpret_cast<Smem32 *>(raw);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, sub = lane >> 3, sl = lane & 7;
  const int nu = L.nu, G = gridDim.x, first = blockIdx.x;
  const int count = (n - first + G - 1) / G;
  start_next();
  if (t == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.vbar[b], 1);
      mbar_init(&sm.fbar[b], 1);
    }
    for (int b = 0; b < 4; ++b) mbar_init(&sm.ibar[b], 1);
    fence_mbar_init();
    for (int b = 0; b < 3; ++b) {
      sm.u[b].set(kZeroSlot, 0.f, 0.f, 0.f);
      sm.p[b][27] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  __syncthreads();
  // a wait that runs out marks the launch as failed; the warp goes on without
  // touching global memory through a patch list that did not arrive
  int polls = LIMITED ? limit : kMaxPolls;
  auto arrived = [&](uint64_t *bar, int phase) {
    if (mbar_wait(bar, phase & 1, polls)) return true;
    polls = 1;
    if (lane == 0) atomicOr(err, PM_ERR_BULK_TIMEOUT);
    return false;
  };

  if (warp == 7) {
    // ------------------------------------------------ copies and block solve
    int nv = 0, nf = 0, ni = 0;  // lane 0: copies started of each kind
    auto cell_of = [&](int c) { return __ldg(list + first + (size_t)c * G); };
    auto bring_values = [&](int c, int cell) {
      bulk_load(sm.values[c & 1], L.values + (size_t)cell * kPatchValues, sizeof(sm.values[0]),
                &sm.vbar[c & 1]);
      nv = c + 1;
    };
    auto bring_fac = [&](int c, int cell) {
      bulk_load(sm.fac[c & 1], factors + (size_t)cell * S1::stride, sizeof(sm.fac[0]),
                &sm.fbar[c & 1]);
      nf = c + 1;
    };
    auto bring_ids = [&](int c, int cell) {
      bulk_load(sm.ids[c & 3], L.ids + (size_t)cell * kPatchIds, sizeof(sm.ids[0]),
                &sm.ibar[c & 3]);
      ni = c + 1;
    };
    int a2 = 0, a3 = 0, a4 = 0;  // cells j + 2, j + 3 and j + 4
    if (lane == 0) {
      const int c0 = cell_of(0);
      bring_ids(0, c0);
      bring_values(0, c0);
      bring_fac(0, c0);
      if (count > 1) {
        const int c1 = cell_of(1);
        bring_ids(1, c1);
        bring_values(1, c1);
        bring_fac(1, c1);
      }
      if (count > 2) bring_ids(2, a2 = cell_of(2));
      if (count > 3) bring_ids(3, a3 = cell_of(3));
      if (count > 4) a4 = cell_of(4);
    }
    const bool in = lane < NU_LOC;
    bool alive = true;
    wait_previous();
    for (int j = 0; j < count; ++j) {
      const int b = j & 1;
      const int *ids = sm.ids[j & 3];
      alive = arrived(&sm.ibar[j & 3], j >> 2) && alive;
      Node<float> old = {};
      float pold = 0.f;
      size_t where = 0;
      if (alive) {
        const int me = ids[kPatchOwn + (in ? lane : 0)];
        old = Node<float>::load(L.u, node_at(me, odd, nu));
        // into the other copy, unless the node belongs to this cell alone
        const bool single = ((unsigned)ids[kPatchSingle] >> lane) & 1;
        where = node_at(single ? me : me ^ 1, odd, nu);
        if (lane < NP_LOC) pold = __ldcg(L.p + ids[kPatchBase] + lane);
      }
      alive = arrived(&sm.fbar[b], j >> 1) && alive;
      const float *F = sm.fac[b] + (in ? lane : 0);
      bar_sync(kBarFull + b, kPatchThreads);  // the residual is there
      // the row warps have waited for the values of this cell
      if (alive && lane == 0 && j + 2 < count) bring_values(j + 2, a2);
      // y_c = A^{-1} r_c
      float y0 = 0, y1 = 0, y2 = 0;
#pragma unroll
      for (int q = 0; q < NU_LOC; ++q) {
        float x, y, z;
        sm.r[b].get(q, x, y, z);
        const float a = F[q * NU_LOC];
        y0 += a * x;
        y1 += a * y;
        y2 += a * z;
      }
      if (!in) y0 = y1 = y2 = 0.f;
      // t = r_p - D y, p = S^{-1} t, x = y - W p
      float s[NP_LOC], p[NP_LOC];
#pragma unroll
      for (int k = 0; k < NP_LOC; ++k) {
        const float *D = F + S1::offD + 3 * NU_LOC * k;
        s[k] = dot3(in ? D[0] : 0.f, y0, in ? D[NU_LOC] : 0.f, y1, in ? D[2 * NU_LOC] : 0.f, y2);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NP_LOC; ++k) s[k] += __shfl_xor_sync(kFull, s[k], o);
#pragma unroll
      for (int k = 0; k < NP_LOC; ++k) {
        s[k] = sm.rp[b][k] - s[k];
        p[k] = 0.f;
      }
#pragma unroll
      for (int m = 0; m < NP_LOC; ++m)
#pragma unroll
        for (int k = 0; k < NP_LOC; ++k) p[k] += sm.fac[b][S1::offS + m * NP_LOC + k] * s[m];
#pragma unroll
      for (int k = 0; k < NP_LOC; ++k) {
        const float *W = F + S1::offW + 3 * NU_LOC * k;
        y0 -= W[0] * p[k];
        y1 -= W[NU_LOC] * p[k];
        y2 -= W[2 * NU_LOC] * p[k];
      }
      if (alive) {
        if (in) {
          float x, y, z;
          comps(old, x, y, z);
          x += damp * y0;
          y += damp * y1;
          z += damp * y2;
          make_node(x, y, z).store(L.u, where);
        }
        if (lane < NP_LOC) {
          const float pl = lane == 0 ? p[0] : (lane == 1 ? p[1] : (lane == 2 ? p[2] : p[3]));
          pold += damp * pl;
          L.p[ids[kPatchBase] + lane] = pold;
        }
      }
      __syncwarp();  // factors and patch list have been read
      if (alive && lane == 0) {
        if (j + 2 < count) bring_fac(j + 2, a2);
        if (j + 4 < count) bring_ids(j + 4, a4);
        a2 = a3;
        a3 = a4;
        if (j + 5 < count) a4 = cell_of(j + 5);
      }
      if (j + 2 < count) bar_arrive(kBarFree + b, kPatchThreads);
    }
    if (!alive && lane == 0) {  // copies still in flight
      for (int c = nv > 2 ? nv - 2 : 0; c < nv; ++c) drain(&sm.vbar[c & 1], c >> 1);
      for (int c = nf > 2 ? nf - 2 : 0; c < nf; ++c) drain(&sm.fbar[c & 1], c >> 1);
      for (int c = ni > 4 ? ni - 4 : 0; c < ni; ++c) drain(&sm.ibar[c & 3], c >> 2);
    }
    return;
  }

  // ------------------------------------------------------------ residuals
  const bool last = warp == 6;
  const int k = warp * 4 + sub;  // row in c_rows order; the spare group of warp 6 repeats the centre
  const int row = c_rows[k];
  bool alive = true;
  int pid = -1;
  uint4 s0 = {0, 0, 0, 0}, s1 = {0, 0, 0, 0};
  unsigned bts = 0, bj = 0, o01 = 0, o23 = 0;
  auto pattern = [&](int id) {  // where the lane's entries lie in the patch
    if (id == pid) return;      // most cells of a level share one
    pid = id;
    const PatchPattern &pat = L.patterns[id];
    s0 = __ldg(reinterpret_cast<const uint4 *>(pat.slot[t]));
    bts = __ldg(reinterpret_cast<const unsigned *>(pat.bt[t]));
    if (warp < 5) s1 = __ldg(reinterpret_cast<const uint4 *>(pat.slot[t]) + 1);
    if (last) pressure_pattern(pat, lane, bj, o01, o23);
  };
  // start the gathers of cell c (one group of copies a cell, empty or not)
  int gpid = -1;  // pattern of the places below
  unsigned pl = 0;
  auto gather = [&](int c) {
    if (c < count) {
      alive = arrived(&sm.ibar[c & 3], c >> 2) && alive;
      if (alive) {
        const int *ids = sm.ids[c & 3];
        const int g = c % 3;
        if (ids[kPatchPattern] != gpid) {
          gpid = ids[kPatchPattern];
          const PatchPattern &pat = L.patterns[gpid];
          pl = __ldg(&pat.place[t]);
          if (t + kRowLanes < kPatchNodes) pl |= (unsigned)__ldg(&pat.place[t + kRowLanes]) << 16;
        }
        const float4 *u4 = static_cast<const float4 *>(L.u);
        async16(&sm.u[g].v[pl & 0xffff], u4 + node_at(ids[t], odd, nu));
        if (t + kRowLanes < kPatchNodes)
          async16(&sm.u[g].v[pl >> 16], u4 + node_at(ids[t + kRowLanes], odd, nu));
        if (t < 27)
          async16(&sm.p[g][t], L.p + ids[kPatchBase + t]);
        else if (t < 55)  // own nodes of the right-hand side, then its pressures
          async16(&sm.f[g][t - 27],
                  t < 54 ? static_cast<const float4 *>(L.f) + (ids[kPatchOwn + t - 27] >> 2)
                         : reinterpret_cast<const float4 *>(L.fp + ids[kPatchBase]));
      }
    }
    async_commit();
  };
  if (arrived(&sm.ibar[0], 0)) pattern(sm.ids[0][kPatchPattern]);
  // everything up to here does not depend on the previous launch
  wait_previous();
  gather(0);
  gather(1);
  for (int j = 0; j < count; ++j) {
    const int b = j & 1, g = j % 3;
    async_wait<1>();                  // this thread's copies of cell j
    bar_sync(kBarRows, kRowLanes);    // everybody's; and cell j - 1 has been read
    gather(j + 2);
    if (alive) pattern(sm.ids[j & 3][kPatchPattern]);
    if (!arrived(&sm.vbar[b], j >> 1)) {
      // warp 7, which fills the stage again, does not wait for it itself
      drain(&sm.vbar[b], j >> 1);
      alive = false;
    }
    float c0, c1, c2;
    row_sum(warp, t, sm.values[b], sm.u[g], &sm.p[g][0].x, s0, s1, bts, c0, c1, c2);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      c0 += __shfl_xor_sync(kFull, c0, o);
      c1 += __shfl_xor_sync(kFull, c1, o);
      c2 += __shfl_xor_sync(kFull, c2, o);
    }
    float cp = 0.f;
    if (last) {
      alive = arrived(&sm.fbar[b], j >> 1) && alive;
      cp = pressure_sum(sub, sm.fac[b], sm.u[g], bj, o01, o23);
    }
    if (j >= 2) bar_sync(kBarFree + b, kPatchThreads);  // this buffer's cell before is solved
    if (k < NU_LOC && sl < 3)
      sm.r[b].ref(row, sl) =
          reinterpret_cast<const float *>(&sm.f[g][row])[sl] - (sl == 0 ? c0 : (sl == 1 ? c1 : c2));
    if (last && sl == 0) sm.rp[b][sub] = reinterpret_cast<const float *>(&sm.f[g][27])[sub] - cp;
    bar_arrive(kBarFull + b, kPatchThreads);
  }
}

// ------------------------------------------------------------------ FP64 ---
template <int ST>
struct Smem64 {
  double values[ST][kPatchValues];
  double fac[ST][Schur<1>::stride];
  int ids[3][kPatchIds];
  Tri<double, kPatchNodes + 1> u;
  __align__(16) double p[28][NP_LOC];
  Tri<double, 28> r;
  double yp[3][7 * NU_LOC];  // partial A^{-1} r
  double y[3][32];
  double rp[NP_LOC], t[NP_LOC];
  uint64_t vbar[ST], fbar[ST], ibar[3];
};
// resident CTAs per SM: 63 KB of shared memory with one stage, 106 KB with two
__host__ __device__ constexpr int ctas64(int stages) { return stages == 1 ? 3 : 2; }

// FP64: the pipe takes half a lane per cycle in each quarter of the SM, so a
// warp's FMA occupies its quarter for 64 cycles and every phase is spread
// over the quarters (warp % 4): vertex rows on quarters 0 and 1, edges on 2,
// 3 and 2, the other rows on 0 and 3, pressure rows on 1; the block solve on
// all warps instead of one.  With one stage (ST = 1) of packed rows and factors
// the next cell's rows arrive during the block solve, and the other two CTAs of
// the SM use the pipe meanwhile (83 % busy at 32^3; 72 % with ST = 2).  Rows and
// factors from DRAM at 64^3, one colour: 979 us (1.47 TB/s; the CSR kernels
// take 1,046), 32^3 134 (162), 16^3 29 (69), 8^3 12.6 (52).
template <int ST, bool LIMITED>
__global__ void __launch_bounds__(kPatchThreads, ctas64(ST)) k_patch_sweep64(
    PatchLevel<double> L, const int *__restrict__ list, int n, const double *__restrict__ factors,
    double damp, int odd, int *err, int limit) {
  using S1 = Schur<1>;
  extern __shared__ __align__(16) unsigned char raw[];
  Smem64<ST> &sm = *reinterpret_cast<Smem64<ST> *>(raw);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, sub = lane >> 3, sl = lane & 7;
  const int nu = L.nu, G = gridDim.x, first = blockIdx.x;
  const int count = (n - first + G - 1) / G;
  start_next();
  if (t == 0) {
    for (int b = 0; b < ST; ++b) {
      mbar_init(&sm.vbar[b], 1);
      mbar_init(&sm.fbar[b], 1);
    }
    for (int b = 0; b < 3; ++b) mbar_init(&sm.ibar[b], 1);
    fence_mbar_init();
    sm.u.set(kZeroSlot, 0.0, 0.0, 0.0);
    for (int m = 0; m < NP_LOC; ++m) sm.p[27][m] = 0.0;
    sm.r.set(27, 0.0, 0.0, 0.0);
  }
  __syncthreads();
  // as in the FP32 kernel; thread 0, which starts the copies, has waited for
  // the last one of a stage itself
  int polls = LIMITED ? limit : kMaxPolls;
  auto arrived = [&](uint64_t *bar, int phase) {
    if (mbar_wait(bar, phase & 1, polls)) return true;
    polls = 1;
    if (lane == 0) atomicOr(err, PM_ERR_BULK_TIMEOUT);
    return false;
  };
  auto cell_of = [&](int c) { return __ldg(list + first + (size_t)c * G); };
  // thread 0: rows, factors and patch list of one cell
  auto bring_values = [&](int c, int cell) {
    bulk_load(sm.values[c % ST], L.values + (size_t)cell * kPatchValues, sizeof(sm.values[0]),
              &sm.vbar[c % ST]);
  };
  auto bring_fac = [&](int c, int cell) {
    bulk_load(sm.fac[c % ST], factors + (size_t)cell * S1::stride, sizeof(sm.fac[0]),
              &sm.fbar[c % ST]);
  };
  auto bring_ids = [&](int c, int cell) {
    bulk_load(sm.ids[c % 3], L.ids + (size_t)cell * kPatchIds, sizeof(sm.ids[0]), &sm.ibar[c % 3]);
  };
  int a1 = 0, a2 = 0, a3 = 0, nv = 0, nf = 0, ni = 0;  // thread 0: next cells, copies started
  if (t == 0) {
    const int c0 = cell_of(0);
    bring_ids(0, c0);
    bring_values(0, c0);
    bring_fac(0, c0);
    nv = nf = 1;
    if (count > 1) bring_ids(1, a1 = cell_of(1));
    if (ST == 2 && count > 1) bring_values(1, a1), bring_fac(1, a1), nv = nf = 2;
    if (count > 2) bring_ids(2, a2 = cell_of(2));
    if (count > 3) a3 = cell_of(3);
    ni = count < 3 ? count : 3;
  }
  // row group of a warp: 0, 1 vertices, 2..4 edges, 5, 6 the rest, 7 pressure rows
  const int group = warp < 4 ? warp : (warp == 4 ? 5 : (warp == 5 ? 7 : (warp == 6 ? 4 : 6)));
  const int k = group * 4 + sub, li = 32 * group + lane;
  const int row = c_rows[k < 27 ? k : 27];
  const bool in = lane < NU_LOC;
  // current values and right-hand side of one cell, on their way
  Node<double> n0 = {}, n1 = {};
  double pv = 0.0, f = 0.0;
  auto gather_u = [&](const int *ids) {
    n0 = Node<double>::load(L.u, node_at(ids[t], odd, nu));
    if (t + kPatchThreads < kPatchNodes)
      n1 = Node<double>::load(L.u, node_at(ids[t + kPatchThreads], odd, nu));
    if (t < 27 * NP_LOC) pv = __ldcg(L.p + ids[kPatchBase + (t >> 2)] + (t & 3));
    if (k < NU_LOC && sl < 3)
      f = __ldcg(static_cast<const double *>(L.f) + 4 * (size_t)(ids[kPatchOwn + row] >> 2) + sl);
    if (group == 7 && sl == 0) f = __ldcg(L.fp + ids[kPatchBase] + sub);
  };
  uint4 s0 = {0, 0, 0, 0}, s1 = {0, 0, 0, 0};
  unsigned bts = 0, bj = 0, o01 = 0, o23 = 0, pl = 0, mine = 0;
  int pid = -1;
  auto pattern = [&](int id) {
    if (id == pid) return;
    pid = id;
    const PatchPattern &pat = L.patterns[id];
    if (group < 7) {
      s0 = __ldg(reinterpret_cast<const uint4 *>(pat.slot[li]));
      if (group < 5) s1 = __ldg(reinterpret_cast<const uint4 *>(pat.slot[li]) + 1);
      bts = __ldg(reinterpret_cast<const unsigned *>(pat.bt[li]));
    } else {
      pressure_pattern(pat, lane, bj, o01, o23);
    }
    pl = __ldg(&pat.place[t]);
    if (t + kPatchThreads < kPatchNodes)
      pl |= (unsigned)__ldg(&pat.place[t + kPatchThreads]) << 16;
    mine = __ldg(&pat.own[lane]);
  };
  bool alive = arrived(&sm.ibar[0], 0);
  if (alive) pattern(sm.ids[0][kPatchPattern]);
  wait_previous();
  if (alive) gather_u(sm.ids[0]);
  int ib = 0, ip = 0;
  for (int j = 0; j < count; ++j) {
    const int b = j % ST;
    const int *ids = sm.ids[ib];
    const int ibn = ib == 2 ? 0 : ib + 1, ipn = ib == 2 ? ip ^ 1 : ip;
    {
      double x, y, z;
      comps(n0, x, y, z);
      sm.u.set(pl & 0xffff, x, y, z);
      if (t + kPatchThreads < kPatchNodes) {
        comps(n1, x, y, z);
        sm.u.set(pl >> 16, x, y, z);
      }
      if (t < 27 * NP_LOC) (&sm.p[0][0])[t] = pv;
    }
    const double fi = f;
    __syncthreads();
    int next_pid = pid;
    if (j + 1 < count) {
      alive = arrived(&sm.ibar[ibn], ipn) && alive;
      if (alive) {
        gather_u(sm.ids[ibn]);
        next_pid = sm.ids[ibn][kPatchPattern];
      }
    }
    if (group < 7) {
      alive = arrived(&sm.vbar[b], j / ST) && alive;
      double c0, c1, c2;
      row_sum(group, li, sm.values[b], sm.u, &sm.p[0][0], s0, s1, bts, c0, c1, c2);
      // six FP64 additions instead of nine: lanes 0..3 go on with component
      // 1, lanes 4..7 with component 2
      c0 += __shfl_xor_sync(kFull, c0, 4);
      const double o12 = __shfl_xor_sync(kFull, (sl & 4) ? c1 : c2, 4);
      double d = ((sl & 4) ? c2 : c1) + o12;
      c0 += __shfl_xor_sync(kFull, c0, 2);
      d += __shfl_xor_sync(kFull, d, 2);
      c0 += __shfl_xor_sync(kFull, c0, 1);
      d += __shfl_xor_sync(kFull, d, 1);
      const double d2 = __shfl_xor_sync(kFull, d, 6);
      if (k < NU_LOC && sl < 3) sm.r.ref(row, sl) = fi - (sl == 0 ? c0 : (sl == 1 ? d : d2));
    } else {
      alive = arrived(&sm.fbar[b], j / ST) && alive;
      const double c = pressure_sum(sub, sm.fac[b], sm.u, bj, o01, o23);
      if (sl == 0) sm.rp[sub] = fi - c;
    }
    __syncthreads();
    if (alive && t == 0 && j + ST < count) {
      bring_values(j + ST, ST == 1 ? a1 : a2);
      nv = j + ST + 1;
    }
    alive = arrived(&sm.fbar[b], j / ST) && alive;
    const double *F = sm.fac[b];
    if (t >= 64 && t - 64 < 7 * NU_LOC) {  // y = A^{-1} r: four columns per thread
      const int q = t - 64, gq = q / NU_LOC, i = q - gq * NU_LOC;
      double c0 = 0, c1 = 0, c2 = 0;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int col = 4 * gq + m;
        double x, y, z;
        sm.r.get(col, x, y, z);
        const double a = col < NU_LOC ? F[col * NU_LOC + i] : 0.0;
        c0 += a * x;
        c1 += a * y;
        c2 += a * z;
      }
      sm.yp[0][q] = c0;
      sm.yp[1][q] = c1;
      sm.yp[2][q] = c2;
    }
    __syncthreads();
    double y = 0;
    if (warp < 3) {  // one component per warp
      if (in) {
#pragma unroll
        for (int q = 0; q < 7; ++q) y += sm.yp[warp][q * NU_LOC + lane];
      }
      sm.y[warp][lane] = y;
    }
    __syncthreads();
    if (warp >= 4) {  // t = r_p - D y, one pressure per warp
      const double *D = F + S1::offD + (warp - 4) * 3 * NU_LOC + (in ? lane : 0);
      const double s = warp_sum(in ? D[0] * sm.y[0][lane] + D[NU_LOC] * sm.y[1][lane] +
                                         D[2 * NU_LOC] * sm.y[2][lane]
                                   : 0.0);
      if (lane == 0) sm.t[warp - 4] = sm.rp[warp - 4] - s;
    }
    __syncthreads();
    if (warp < 3) {  // p = S^{-1} t, x = y - W p, update of one component
      double pk = 0;
      if (lane < NP_LOC) {
#pragma unroll
        for (int m = 0; m < NP_LOC; ++m) pk += F[S1::offS + m * NP_LOC + lane] * sm.t[m];
      }
      const double *W = F + S1::offW + warp * NU_LOC + (in ? lane : 0);
#pragma unroll
      for (int m = 0; m < NP_LOC; ++m) y -= W[m * 3 * NU_LOC] * __shfl_sync(kFull, pk, m);
      if (alive) {
        if (in) {
          const int me = ids[kPatchOwn + lane];
          // into the other copy, unless the node belongs to this cell alone
          const bool single = ((unsigned)ids[kPatchSingle] >> lane) & 1;
          double v = sm.u.ref(mine >> 4, warp);
          v += damp * y;
          static_cast<double *>(L.u)[4 * node_at(single ? me : me ^ 1, odd, nu) + warp] = v;
        }
        if (warp == 2 && lane < NP_LOC) {
          double v = sm.p[0][lane];
          v += damp * pk;
          L.p[ids[kPatchBase] + lane] = v;
        }
      }
    }
    __syncthreads();  // the stage and the gathered values have been read
    if (alive && t == 0) {
      if (j + ST < count) bring_fac(j + ST, ST == 1 ? a1 : a2), nf = j + ST + 1;
      if (j + 3 < count) bring_ids(j + 3, a3), ni = j + 4;
      a1 = a2;
      a2 = a3;
      if (j + 4 < count) a3 = cell_of(j + 4);
    }
    pattern(next_pid);
    ib = ibn;
    ip = ipn;
  }
  if (!alive && t == 0) {  // copies still in flight
    for (int c = nv > ST ? nv - ST : 0; c < nv; ++c) drain(&sm.vbar[c % ST], c / ST);
    for (int c = nf > ST ? nf - ST : 0; c < nf; ++c) drain(&sm.fbar[c % ST], c / ST);
    for (int c = ni > 3 ? ni - 3 : 0; c < ni; ++c)
      drain(&sm.ibar[c % 3], c / 3);
  }
}

// node i of a vector [v1|v2|v3], read from L2 (the kernel before updates u in
// place)
template <typename T>
__device__ __forceinline__ Node<T> node_of(const T *v, int i, int nu) {
  return make_node(__ldcg(v + i), __ldcg(v + (size_t)nu + i), __ldcg(v + (size_t)2 * nu + i));
}

// u -> the copies (both), u on the Dirichlet nodes taken from the right-hand
// side; p -> its copy; the right-hand side with its components side by side
// (u = nullptr: zero).  The first kernel of a run of sweeps lets the next one
// start only after it has waited itself: what the sweeps read before they
// wait (packed rows, factors, patch lists) was complete then.
template <typename T>
__global__ void k_patch_begin(PatchLevel<T> L, const T *__restrict__ u, const T *__restrict__ rhs,
                              int hb, int np) {
  const int nu = L.nu, n = nu > np ? nu : np;
  wait_previous();
  start_next();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (i < nu) {
      const Node<T> f = node_of(rhs, i, nu);
      Node<T> v = f;
      if (i < hb)
        v = u ? node_of(u, i, nu) : make_node(T(0), T(0), T(0));
      v.store(L.u, i);
      v.store(L.u, (size_t)nu + i);
      f.store(L.f, i);
    }
    if (i < np) {
      L.p[i] = u ? __ldcg(u + (size_t)3 * nu + i) : T(0);
      L.fp[i] = __ldcg(rhs + (size_t)3 * nu + i);
    }
  }
}

// the Dirichlet nodes of both copies between two sweeps
template <typename T>
__global__ void k_patch_dirichlet(PatchLevel<T> L, const T *__restrict__ rhs, int hb) {
  const int nu = L.nu;
  start_next();
  wait_previous();
  for (int i = hb + blockIdx.x * blockDim.x + threadIdx.x; i < nu; i += gridDim.x * blockDim.x) {
    const Node<T> v = make_node(rhs[i], rhs[(size_t)nu + i], rhs[(size_t)2 * nu + i]);
    v.store(L.u, i);
    v.store(L.u, (size_t)nu + i);
  }
}

// the current copies -> u (Dirichlet nodes from the right-hand side, or zero
// without one) and p
template <typename T>
__global__ void k_patch_end(PatchLevel<T> L, T *__restrict__ u, const T *__restrict__ rhs, int hb,
                            int np, int odd) {
  const int nu = L.nu, n = nu > np ? nu : np;
  start_next();
  wait_previous();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (i < nu) {
      T x, y, z;
      if (i < hb) {
        const int copy = odd & L.flips[i];
        comps(Node<T>::load(L.u, (size_t)copy * nu + i), x, y, z);
      } else {
        x = rhs ? rhs[i] : T(0);
        y = rhs ? rhs[(size_t)nu + i] : T(0);
        z = rhs ? rhs[(size_t)2 * nu + i] : T(0);
      }
      u[i] = x;
      u[(size_t)nu + i] = y;
      u[(size_t)2 * nu + i] = z;
    }
    if (i < np) u[(size_t)3 * nu + i] = __ldcg(L.p + i);
  }
}

// Packed values of a level from its CSR arrays: one CTA per cell, entry j of
// a row goes to lane j % 8, place j / 8; staged in shared memory and written
// out in one stream.
template <typename T>
__global__ void __launch_bounds__(256) k_patch_pack(PatchLevel<T> L, DevOp<T> op) {
  __shared__ __align__(16) T stage[kPatchValues];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, cell = blockIdx.x;
  const int *own = L.ids + (size_t)cell * kPatchIds + kPatchOwn;
  for (int i = t; i < kPatchValues; i += 256) stage[i] = T(0);
  __syncthreads();
  const T *A = op.a[0];
  for (int k = warp; k < NU_LOC; k += 8) {
    const int r = __ldg(own + c_rows[k]) >> 2;
    const int rs = __ldg(op.a_rowptr + r), n = __ldg(op.a_rowptr + r + 1) - rs;
    for (int j = lane; j < n; j += 32) stage[a_pos(8 * k + (j & 7), j >> 3)] = __ldg(A + rs + j);
    if (r < op.nact) {
      const int ts = __ldg(op.bt_rowptr + r), m = __ldg(op.bt_rowptr + r + 1) - ts;
      for (int j = lane; j < m; j += 32) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
          stage[bt_pos(8 * k + (j & 7), j >> 3, c)] = __ldg(op.bt[c] + ts + j);
      }
    }
  }
  __syncthreads();
  T *V = L.values_w + (size_t)cell * kPatchValues;
  constexpr int VW = 16 / sizeof(T);
  for (int i = t; i < kPatchValues / VW; i += 256)
    reinterpret_cast<float4 *>(V)[i] = reinterpret_cast<const float4 *>(stage)[i];
}

// B against the D blocks of the stored factors: one warp per pressure row
template <typename T>
__global__ void __launch_bounds__(32 * NP_LOC) k_patch_compare_b(PatchLevel<T> L, DevOp<T> op,
                                                                const T *__restrict__ factors,
                                                                int *differ) {
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31, cell = blockIdx.x;
  const int *ids = L.ids + (size_t)cell * kPatchIds;
  const PatchPattern &pat = L.patterns[ids[kPatchPattern]];
  const T *D = factors + (size_t)cell * Schur<1>::stride + Schur<1>::offD + k * 3 * NU_LOC;
  const int rs = op.b_rowptr[ids[kPatchBase] + k], n = op.b_rowptr[ids[kPatchBase] + k + 1] - rs;
  bool other = false;
  if (lane < n) {
    const int at = pat.bj[8 * k + (lane & 7)][lane >> 3];
    for (int c = 0; c < 3; ++c) other |= !(op.b[c][rs + lane] == D[c * NU_LOC + at]);
  }
  if (other) atomicOr(differ, 1);
}

// Cells of every velocity node (slots: the first eight, cnt: all) and the
// owner count of every pressure block; *bad when a node lies in more than
// eight cells or a cell's pressure DOFs are not one aligned block of its own.
__global__ void k_patch_incidence(int ncells, const int *udofs, const int *pdofs, int *cnt,
                                  int *slots, int *owners, int *bad) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ncells * NU_LOC;
       i += gridDim.x * blockDim.x) {
    const int c = i / NU_LOC, k = i - c * NU_LOC, id = udofs[i], at = atomicAdd(cnt + id, 1);
    bool wrong = at >= 8;
    if (!wrong) slots[8 * (size_t)id + at] = c;
    if (k < NP_LOC) {
      const int base = pdofs[NP_LOC * (size_t)c];
      wrong = wrong || base % NP_LOC || pdofs[NP_LOC * (size_t)c + k] != base + k;
      if (k == 0 && atomicAdd(owners + base / NP_LOC, 1)) wrong = true;
    }
    if (wrong) atomicOr(bad, 1);
  }
}

// Features of a Q2 cell, 6 faces, 12 edges, 8 vertices: the middle node, and
// the features that contain it (whose neighbours touch it too).
__host__ __device__ constexpr bool feature_coords(int f, int d[3]) {
  for (int fixed = 1; fixed <= 3; ++fixed)
    for (int c = 0; c < 27; ++c) {
      d[0] = c % 3 - 1;
      d[1] = (c / 3) % 3 - 1;
      d[2] = c / 9 - 1;
      if ((d[0] != 0) + (d[1] != 0) + (d[2] != 0) == fixed && f-- == 0) return true;
    }
  return false;
}
struct Features {
  int pivot[26], sup[26];
};
constexpr Features make_features() {
  Features F = {};
  for (int f = 0; f < 26; ++f) {
    int d[3] = {}, e[3] = {};
    feature_coords(f, d);
    F.pivot[f] = d[0] + 1 + 3 * (d[1] + 1) + 9 * (d[2] + 1);
    for (int g = 0; g < f; ++g) {
      feature_coords(g, e);
      bool in = true;
      for (int k = 0; k < 3; ++k) in = in && (e[k] == 0 || e[k] == d[k]);
      if (in) F.sup[f] |= 1 << g;
    }
  }
  return F;
}
__constant__ Features c_feat = make_features();

// Patch list of a cell, once per level at set-up: its neighbours by feature
// (faces, then edges, then vertices; *bad when more than one lies beyond a
// feature), their nodes sorted and made unique.  On the host (16 threads) the
// lists and their upload took 80 ms at 32^3, in a set-up of 119 ms now.
__global__ void __launch_bounds__(256) k_patch_list(int ncells, const int *udofs, const int *pdofs,
                                                    const int *cnt, const int *slots,
                                                    const int *colour, int *ids, int *bad) {
  __shared__ int key[1024], list[kPatchNodes], nb[26], part[8];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, c = blockIdx.x;
  const int *own = udofs + (size_t)c * NU_LOC;
  if (warp == 0) {
    const int f = lane < 26 ? lane : 25, pv = own[c_feat.pivot[f]], sup = c_feat.sup[f];
    const int rank = f < 6 ? 0 : (f < 18 ? 1 : 2), m = cnt[pv] < 8 ? cnt[pv] : 8;
    bool two = false;
    for (int r = 0; r < 3; ++r) {
      if (lane < 26 && rank == r) {
        int mine = -1;
        for (int e = 0; e < m; ++e) {
          const int o = slots[8 * (size_t)pv + e];
          bool known = o == c;
          for (int g = 0; g < 18; ++g) known = known || ((sup >> g & 1) && nb[g] == o);
          if (known) continue;
          two = two || (mine >= 0 && mine != o);
          mine = o;
        }
        nb[lane] = mine;
      }
      __syncwarp();
    }
    if (two) atomicOr(bad, 1);
  }
  __syncthreads();
  for (int i = t; i < 1024; i += 256) {
    const int q = i / NU_LOC, k = i - q * NU_LOC;
    int v = INT_MAX;
    if (q == 0)
      v = own[k];
    else if (q <= 26 && nb[q - 1] >= 0)
      v = udofs[(size_t)nb[q - 1] * NU_LOC + k];
    key[i] = v;
  }
  for (int size = 2; size <= 1024; size *= 2)
    for (int step = size / 2; step > 0; step /= 2) {
      __syncthreads();
      for (int i = t; i < 512; i += 256) {
        const int lo = 2 * i - (i & (step - 1)), hi = lo + step;
        const int a = key[lo], b = key[hi];
        if ((a > b) == ((lo & size) == 0)) {
          key[lo] = b;
          key[hi] = a;
        }
      }
    }
  __syncthreads();
  // the first of each run of equal nodes, in order
  bool first[4];
  int n = 0;
  for (int q = 0; q < 4; ++q) {
    const int i = 4 * t + q;
    first[q] = key[i] != INT_MAX && (i == 0 || key[i] != key[i - 1]);
    n += first[q];
  }
  int before = n;
  for (int o = 1; o < 32; o *= 2) {
    const int v = __shfl_up_sync(kFull, before, o);
    if (lane >= o) before += v;
  }
  if (lane == 31) part[warp] = before;
  __syncthreads();
  int total = 0;
  for (int w = 0; w < 8; ++w) {
    if (w == warp) before += total - n;
    total += part[w];
  }
  for (int q = 0; q < 4; ++q)
    if (first[q]) {
      if (before < kPatchNodes) list[before] = key[4 * t + q];
      ++before;
    }
  __syncthreads();
  if (total > kPatchNodes) {
    if (t == 0) atomicOr(bad, 1);
    return;
  }
  int *out = ids + (size_t)c * kPatchIds;
  const int col = colour[c];
  auto entry = [&](int id) {  // with the updates by earlier colours of a sweep
    const int m = cnt[id];
    int up = 0;
    for (int e = 0; e < m && e < 8; ++e) up += colour[slots[8 * (size_t)id + e]] < col;
    return (id << 2) | (m > 1 ? ((m & 1) << 1) | (up & 1) : 0);
  };
  for (int q = t; q < kPatchNodes; q += 256) out[q] = entry(list[q < total ? q : 0]);
  if (warp == 0) {
    const int id = own[lane < NU_LOC ? lane : 0];
    if (lane < NU_LOC) out[kPatchOwn + lane] = entry(id);
    const unsigned single = __ballot_sync(kFull, lane < NU_LOC && cnt[id] == 1);
    if (lane == 0) {
      out[kPatchCount] = total;
      out[kPatchSingle] = (int)single;
      out[kPatchPattern] = 0;
    }
    if (lane < 27) {
      const int o = lane == 0 || nb[lane - 1] < 0 ? c : nb[lane - 1];
      out[kPatchBase + lane] = pdofs[NP_LOC * (size_t)o];
    }
  }
}

// nodes that change copies from sweep to sweep: an odd number > 1 of updates
__global__ void k_patch_flips(int nu, const int *cnt, unsigned char *flips) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nu; i += gridDim.x * blockDim.x)
    flips[i] = cnt[i] > 1 && (cnt[i] & 1);
}

__global__ void k_patch_assign(int *ids, const int *pattern, int ncells) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < ncells) ids[(size_t)c * kPatchIds + kPatchPattern] = pattern[c];
}

// Pattern of a cell from the CSR patterns and its patch list (once per level,
// at set-up).  MODE 0: a hash of the pattern into hash[cell] (the words through
// the finaliser of splitmix64, Steele, Lea and Flood 2014, summed); 1: the
// pattern of cell which[blockIdx.x] into patterns[blockIdx.x]; 2: compare with
// the pattern that the cell was given.  Rows that do not fit set *bad.
template <int MODE>
__global__ void __launch_bounds__(256) k_patch_pattern(
    const int *ids_all, const int *a_rowptr, const int *a_col, const int *b_rowptr,
    const int *b_col, const int *bt_rowptr, const int *bt_col, int nact, const int *which,
    PatchPattern *patterns, unsigned long long *hash, int *bad) {
  __shared__ __align__(16) PatchPattern pt;
  __shared__ int node[kPatchNodes], own[NU_LOC], base[27];
  __shared__ unsigned long long h;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int cell = MODE == 1 ? which[blockIdx.x] : (int)blockIdx.x;
  const int *ids = ids_all + (size_t)cell * kPatchIds;
  const int n = ids[kPatchCount];
  for (int i = t; i < kPatchNodes; i += 256) node[i] = ids[i] >> 2;
  if (t < NU_LOC) {
    own[t] = ids[kPatchOwn + t] >> 2;
    base[t] = ids[kPatchBase + t];
  }
  if (t == 0) h = 0;
  for (int i = t; i < kRowLanes * 16; i += 256) (&pt.slot[0][0])[i] = (uint16_t)(16 * kZeroSlot);
  for (int i = t; i < kRowLanes * 4; i += 256) (&pt.bt[0][0])[i] = (uint8_t)kZeroP;
  if (t < 128) (&pt.bj[0][0])[t] = (uint8_t)NU_LOC;
  if (t < 32) pt.own[t] = (uint16_t)(16 * kZeroSlot);
  for (int i = t; i < kPatchIds - 48; i += 256) pt.place[i] = (uint16_t)i;
  __syncthreads();
  auto find = [&](int id) {
    int lo = 0, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (node[mid] < id)
        lo = mid + 1;
      else
        hi = mid;
    }
    return lo < n && node[lo] == id ? lo : -1;
  };
  bool miss = false;
  if (t < NU_LOC) {
    const int s = find(own[t]);
    if (s < 0)
      miss = true;
    else
      pt.own[t] = (uint16_t)(16 * s);
  }
  for (int k = warp; k < NU_LOC; k += 8) {
    const int r = own[c_rows[k]];
    const int rs = a_rowptr[r], m = a_rowptr[r + 1] - rs;
    if (m > 8 * row_cap(k)) miss = true;
    for (int j = lane; j < m && j < 8 * row_cap(k); j += 32) {
      const int s = find(a_col[rs + j]);
      if (s < 0)
        miss = true;
      else
        pt.slot[8 * k + (j & 7)][j >> 3] = (uint16_t)(16 * s);
    }
    if (r >= nact) continue;
    const int ts = bt_rowptr[r], mt = bt_rowptr[r + 1] - ts;
    if (mt > 8 * bt_cap(k)) miss = true;
    for (int j = lane; j < mt && j < 8 * bt_cap(k); j += 32) {
      const int c = bt_col[ts + j];
      int nb = -1;
      for (int q = 26; q >= 0; --q)
        if (base[q] == (c & ~3)) nb = q;
      if (nb < 0)
        miss = true;
      else
        pt.bt[8 * k + (j & 7)][j >> 3] = (uint8_t)(4 * nb + (c & 3));
    }
  }
  // the pressure rows couple to the cell's own nodes only (their values are
  // the D block of the stored factors), each once
  if (warp < NP_LOC) {
    const int rs = b_rowptr[base[0] + warp], m = b_rowptr[base[0] + warp + 1] - rs;
    if (m > NU_LOC) miss = true;
    for (int j = lane; j < m && j < NU_LOC; j += 32) {
      const int c = b_col[rs + j];
      int at = -1;
      for (int q = 0; q < NU_LOC; ++q)
        if (own[q] == c) at = q;
      if (at < 0 || (j > 0 && b_col[rs + j - 1] >= c))
        miss = true;
      else
        pt.bj[8 * warp + (j & 7)][j >> 3] = (uint8_t)at;
    }
  }
  if (miss) atomicOr(bad, 1);
  __syncthreads();
  constexpr int words = (int)(sizeof(PatchPattern) / 8);
  const unsigned long long *w = reinterpret_cast<const unsigned long long *>(&pt);
  if constexpr (MODE == 0) {
    unsigned long long s = 0;
    for (int i = t; i < words; i += 256) {
      unsigned long long x = w[i] + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);
      x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
      x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
      s += x ^ (x >> 31);
    }
    atomicAdd(&h, s);
    __syncthreads();
    if (t == 0) hash[cell] = h;
  } else if constexpr (MODE == 1) {
    for (int i = t; i < words; i += 256)
      reinterpret_cast<unsigned long long *>(patterns + blockIdx.x)[i] = w[i];
  } else {
    const unsigned long long *v =
        reinterpret_cast<const unsigned long long *>(patterns + ids[kPatchPattern]);
    bool differ = false;
    for (int i = t; i < words; i += 256) differ |= v[i] != w[i];
    if (differ) atomicOr(bad, 1);
  }
}

inline int ok() { return cudaPeekAtLastError() == cudaSuccess ? 1 : -1; }

int node_grid(int n) {
  const int g = (n + 255) / 256;
  return g < 1 ? 1 : (g > 8 * 152 ? 8 * 152 : g);
}

}  // namespace

template <typename T>
int launch_patch_pack(const PatchLevel<T> &L, const DevOp<T> &op, int ncells, cudaStream_t s) {
  if (ncells <= 0) return 0;
  if (!op.structured) return -1;
  k_patch_pack<T><<<ncells, 256, 0, s>>>(L, op);
  return ok();
}

template <typename T>
int launch_patch_compare_b(const PatchLevel<T> &L, const DevOp<T> &op, int ncells,
                           const T *factors, int *differ, cudaStream_t s) {
  if (ncells <= 0) return 0;
  k_patch_compare_b<T><<<ncells, 32 * NP_LOC, 0, s>>>(L, op, factors, differ);
  return ok();
}

template <typename T>
int launch_patch_pattern(int mode, const int *ids, const DevOp<T> &op, int n, const int *which,
                         void *patterns, unsigned long long *hash, int *bad, cudaStream_t s) {
  if (n <= 0) return 0;
  PatchPattern *p = static_cast<PatchPattern *>(patterns);
  auto run = [&](auto kernel) {
    kernel<<<n, 256, 0, s>>>(ids, op.a_rowptr, op.a_col, op.b_rowptr, op.b_col, op.bt_rowptr,
                             op.bt_col, op.nact, which, p, hash, bad);
  };
  if (mode == 0)
    run(k_patch_pattern<0>);
  else if (mode == 1)
    run(k_patch_pattern<1>);
  else
    run(k_patch_pattern<2>);
  return ok();
}

// Places of a pattern's nodes: greedy over the nodes in list order, each into
// the bank group (place % 8) where the fewest lanes of a row's octets meet,
// then a pass of improving exchanges (1.7 ms; 533 -> 394 wavefronts for the
// 288 octets of an inner cell, more passes 386); place kZeroSlot stays the zero's.
void patch_places(void *patterns, long long count) {
  PatchPattern *P = static_cast<PatchPattern *>(patterns);
#pragma omp parallel for schedule(dynamic)
  for (long long c = 0; c < count; ++c) {
    PatchPattern &pt = P[c];
    constexpr int N = kPatchNodes, OCT = 28 * 16;
    std::vector<std::vector<int>> octets(N);  // octets (row, entry number) that read a node
    for (int r = 0; r < 28; ++r)
      for (int q = 0; q < 16; ++q)
        for (int l = 0; l < 8; ++l) {
          const int node = pt.slot[8 * r + l][q] / 16;
          if (node < N) octets[node].push_back(16 * r + q);
        }
    std::vector<int> group(N, -1), used(8, 0);
    std::vector<std::array<uint8_t, 8>> cnt(OCT);
    for (auto &o : cnt) o.fill(0);
    const int room[8] = {43, 43, 43, 43, 43, 43, 43, 42};  // places of a group (343 in all)
    auto cost = [&](int node, int g) {
      int s = 0;
      for (int o : octets[node]) s += cnt[o][g];
      return s;
    };
    auto put = [&](int node, int g, int d) {
      for (int o : octets[node]) cnt[o][g] = (uint8_t)(cnt[o][g] + d);
      used[g] += d;
    };
    int at = 0;
    for (int n = 0; n < N; ++n) {
      int best = -1, bc = 0;
      for (int q = 0; q < 8; ++q) {
        const int g = (at + q) & 7;
        if (used[g] >= room[g]) continue;
        const int k = cost(n, g);
        if (best < 0 || k < bc) {
          best = g;
          bc = k;
        }
      }
      group[n] = best;
      put(n, best, 1);
      at = best + 1;
    }
    for (int n = 0; n < N; ++n) {
      const int g = group[n];
      put(n, g, -1);
      const int own = cost(n, g);
      int gain = 0, with = -1;
      for (int m = 0; own > 0 && m < N; ++m) {
        const int h = group[m];
        if (m == n || h == g) continue;
        put(m, h, -1);
        const int before = own + cost(m, h), after = cost(n, h) + cost(m, g);
        put(m, h, 1);
        if (before - after > gain) {
          gain = before - after;
          with = m;
        }
      }
      if (with >= 0) {
        put(with, group[with], -1);
        group[n] = group[with];
        group[with] = g;
        put(with, g, 1);
      }
      put(n, group[n], 1);
    }
    int next[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint16_t place[N + 1];
    for (int n = 0; n < N; ++n) place[n] = (uint16_t)(8 * next[group[n]]++ + group[n]);
    place[N] = (uint16_t)N;
    for (auto &lane : pt.slot)
      for (uint16_t &e : lane) e = (uint16_t)(16 * place[e / 16]);
    for (uint16_t &e : pt.own) e = (uint16_t)(16 * place[e / 16]);
    for (int n = 0; n <= N; ++n) pt.place[n] = place[n];
  }
}

size_t patch_list_scratch(int ncells, int nu, int np) {
  return sizeof(int) * (9 * (size_t)nu + (size_t)np / NP_LOC + (size_t)ncells);
}

int launch_patch_lists(const DevCells &cells, int nu, int np, const int *colour, int *ids,
                       unsigned char *flips, void *scratch, int *bad, cudaStream_t s) {
  if (cells.ncells <= 0) return 0;
  int *slots = static_cast<int *>(scratch), *cnt = slots + 8 * (size_t)nu, *owners = cnt + nu,
      *col = owners + np / NP_LOC;
  if (cudaMemsetAsync(cnt, 0, sizeof(int) * ((size_t)nu + np / NP_LOC), s) != cudaSuccess ||
      cudaMemcpyAsync(col, colour, sizeof(int) * (size_t)cells.ncells, cudaMemcpyHostToDevice,
                      s) != cudaSuccess)
    return -1;
  k_patch_incidence<<<node_grid(cells.ncells * NU_LOC), 256, 0, s>>>(
      cells.ncells, cells.udofs, cells.pdofs, cnt, slots, owners, bad);
  k_patch_list<<<cells.ncells, 256, 0, s>>>(cells.ncells, cells.udofs, cells.pdofs, cnt, slots, col,
                                            ids, bad);
  k_patch_flips<<<node_grid(nu), 256, 0, s>>>(nu, cnt, flips);
  return cudaPeekAtLastError() == cudaSuccess ? 3 : -1;
}

int launch_patch_assign(int *ids, const int *pattern, int ncells, cudaStream_t s) {
  if (ncells <= 0) return 0;
  k_patch_assign<<<(ncells + 255) / 256, 256, 0, s>>>(ids, pattern, ncells);
  return ok();
}

int launch_patch_init() {
  auto set = [](auto kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) ==
           cudaSuccess;
  };
  return set(k_patch_sweep32<false>, sizeof(Smem32)) &&
                 set(k_patch_sweep32<true>, sizeof(Smem32)) &&
                 set(k_patch_sweep64<1, false>, sizeof(Smem64<1>)) &&
                 set(k_patch_sweep64<1, true>, sizeof(Smem64<1>)) &&
                 set(k_patch_sweep64<2, false>, sizeof(Smem64<2>)) &&
                 set(k_patch_sweep64<2, true>, sizeof(Smem64<2>))
             ? 0
             : -1;
}

template <typename T>
int launch_patch_begin(const PatchLevel<T> &L, const T *u, const T *rhs, int hb, int np,
                       cudaStream_t s) {
  return launch_chained<PatchLevel<T>, const T *, const T *, int, int>(
      k_patch_begin<T>, node_grid(std::max(L.nu, np)), 256, 0, s, L, u, rhs, hb, np);
}

template <typename T>
int launch_patch_colour(const PatchLevel<T> &L, const int *list, int n, const T *factors, T damp,
                        int odd, int *err, int num_sms, int wait_limit, cudaStream_t s) {
  if (n <= 0) return 0;
  const int limit = wait_limit > 0 ? wait_limit : kMaxPolls;
  if constexpr (sizeof(T) == 4)
    return launch_chained<PatchLevel<T>, const int *, int, const T *, T, int, int *, int>(
        wait_limit > 0 ? k_patch_sweep32<true> : k_patch_sweep32<false>,
        std::min(n, kCtas32 * num_sms), kPatchThreads, sizeof(Smem32), s, L, list, n, factors,
        damp, odd, err, limit);
  else {
    // Two stages while they hold all the cells of a CTA: with rows that come
    // from DRAM, two sweeps at 16^3 take 492 us against 541 with one stage.
    // One stage and a third CTA above: colour at 32^3 134 against 153 us, at
    // 64^3 979 against 1112.
    const int two = ctas64(2) * num_sms;
    const bool all = n <= 2 * two;
    return launch_chained<PatchLevel<T>, const int *, int, const T *, T, int, int *, int>(
        wait_limit > 0 ? (all ? k_patch_sweep64<2, true> : k_patch_sweep64<1, true>)
                       : (all ? k_patch_sweep64<2, false> : k_patch_sweep64<1, false>),
        std::min(n, all ? two : ctas64(1) * num_sms), kPatchThreads,
        all ? sizeof(Smem64<2>) : sizeof(Smem64<1>), s, L, list, n, factors, damp, odd, err, limit);
  }
}

template <typename T>
int launch_patch_between(const PatchLevel<T> &L, const T *rhs, int hb, cudaStream_t s) {
  if (hb >= L.nu) return 0;
  return launch_chained<PatchLevel<T>, const T *, int>(k_patch_dirichlet<T>, node_grid(L.nu - hb),
                                                       256, 0, s, L, rhs, hb);
}

template <typename T>
int launch_patch_end(const PatchLevel<T> &L, T *u, const T *rhs, int hb, int np, int odd,
                     cudaStream_t s) {
  return launch_chained<PatchLevel<T>, T *, const T *, int, int, int>(
      k_patch_end<T>, node_grid(std::max(L.nu, np)), 256, 0, s, L, u, rhs, hb, np, odd);
}

#define PM_PINST(T)                                                                               \
  template int launch_patch_pack<T>(const PatchLevel<T> &, const DevOp<T> &, int, cudaStream_t);  \
  template int launch_patch_compare_b<T>(const PatchLevel<T> &, const DevOp<T> &, int, const T *, \
                                         int *, cudaStream_t);                                    \
  template int launch_patch_pattern<T>(int, const int *, const DevOp<T> &, int, const int *,      \
                                       void *, unsigned long long *, int *, cudaStream_t);        \
  template int launch_patch_begin<T>(const PatchLevel<T> &, const T *, const T *, int, int,       \
                                     cudaStream_t);                                               \
  template int launch_patch_colour<T>(const PatchLevel<T> &, const int *, int, const T *,         \
                                      T, int, int *, int, int, cudaStream_t);                     \
  template int launch_patch_between<T>(const PatchLevel<T> &, const T *, int, cudaStream_t);      \
  template int launch_patch_end<T>(const PatchLevel<T> &, T *, const T *, int, int, int,          \
                                   cudaStream_t);
PM_PINST(double)
PM_PINST(float)
#undef PM_PINST

}  // namespace pm
