// pm_vanka_patch.cu — cell-Vanka sweeps of one-block Q2 hexahedral levels
// from a per-cell packed copy of the velocity rows.
//
// One colour of a sweep (CellVanka, src/FE/NSE_MGLevel4.C:1653-2087, in the
// colour-block order of CellVanka_GPU, src/FE/NSE_CellVanka.cu:1748-2555) is
// one launch, one CTA of 192 threads per cell: local residual r = f - K u on
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
// Patch.  Each cell keeps the sorted list of its patch's nodes; where entry j
// of row r finds its node in that list is a pattern of 16-bit positions that
// cells with the same neighbourhood and numbering order share (one for all
// inner cells of a uniform mesh).  Meshes whose cells have more than one
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
#include <cstdint>

#include "pm_kernels.h"

namespace pm {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kPatchThreads = 256;  // warps 0-1 vertex rows, 2-4 edges, 5-6 the rest, 7 pressure
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
  uint16_t slot[kRowLanes][16];  // A entry: position in the patch list
  uint8_t bt[kRowLanes][4];      // BT entry: 4 * neighbour + mode
  uint8_t bj[32][4];             // B row lane / 8, entry lane % 8 + 8 q: own node
  uint16_t own[32];              // own node: position in the patch list
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
  static __device__ __forceinline__ float *component(void *p, size_t i) {
    return reinterpret_cast<float *>(p) + 4 * i;
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
  static __device__ __forceinline__ double *component(void *p, size_t i) {
    return reinterpret_cast<double *>(p) + 4 * i;
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
  __device__ __forceinline__ float get(int i, int c) const {
    return reinterpret_cast<const float *>(v)[4 * i + c];
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
  __device__ __forceinline__ double get(int i, int c) const {
    return c < 2 ? reinterpret_cast<const double *>(v)[2 * i + c] : w[i];
  }
  __device__ __forceinline__ void set(int i, double x, double y, double z) {
    v[i] = make_double2(x, y);
    w[i] = z;
  }
};

// four (two) consecutive values, read once
__device__ __forceinline__ void ld4(const float *p, float &x, float &y, float &z, float &w) {
  const float4 v = __ldcs(reinterpret_cast<const float4 *>(p));
  x = v.x;
  y = v.y;
  z = v.z;
  w = v.w;
}
__device__ __forceinline__ void ld4(const double *p, double &x, double &y, double &z, double &w) {
  const double2 a = __ldcs(reinterpret_cast<const double2 *>(p)),
                b = __ldcs(reinterpret_cast<const double2 *>(p) + 1);
  x = a.x;
  y = a.y;
  z = b.x;
  w = b.y;
}
__device__ __forceinline__ void ld2(const float *p, float &x, float &y) {
  const float2 v = __ldcs(reinterpret_cast<const float2 *>(p));
  x = v.x;
  y = v.y;
}
__device__ __forceinline__ void ld2(const double *p, double &x, double &y) {
  const double2 v = __ldcs(reinterpret_cast<const double2 *>(p));
  x = v.x;
  y = v.y;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// the previous kernel of the stream has finished and its writes are visible
__device__ __forceinline__ void wait_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// the next kernel of the stream may start (it waits before it reads results)
__device__ __forceinline__ void start_next() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename T>
struct PatchSmem {
  Tri<T, kPatchNodes + 1> u;
  __align__(16) T r[3][28];  // local residual by component
  T p[28][NP_LOC];           // pressures of the cell and its neighbours, then zeros
  T y[3][32];
  T rp[NP_LOC], t[NP_LOC];
};

// FP32: bound by the packed values from HBM on large levels, by the chain
// gather -> sums -> solve -> update on small ones.  FP64: by the FP64 pipe.
template <typename T>
__global__ void __launch_bounds__(kPatchThreads, sizeof(T) == 4 ? 3 : 2) k_patch_sweep(
    PatchLevel<T> L, const int *__restrict__ list, const T *__restrict__ factors,
    const T *__restrict__ rhs, T damp, int odd) {
  using S1 = Schur<1>;
  __shared__ PatchSmem<T> sm;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, sub = lane >> 3, sl = lane & 7;
  const int nu = L.nu;
  start_next();
  const int cell = __ldg(list + blockIdx.x);

  // ---- everything that the previous colour does not change
  const int *ids = L.ids + (size_t)cell * kPatchIds;
  const PatchPattern &pat = L.patterns[__ldg(L.pattern + cell)];
  const int id0 = __ldg(ids + t);
  const int id1 = t + kPatchThreads < kPatchNodes ? __ldg(ids + t + kPatchThreads) : 0;
  const int pb = t < 27 ? __ldg(ids + kPatchBase + t) : 0;
  const T *V = L.values + (size_t)cell * kPatchValues;
  const T *F = factors + (size_t)cell * S1::stride;
  const bool vtx = warp < 2, edge = warp >= 2 && warp < 5, rest = warp == 5 || warp == 6;
  // Values a thread keeps, by the work of its warp (one array, so that the
  // warps' different lists share registers):
  //   vertex, edge rows: A entries 0..15, BT entries 16 + 4 c + q, D 28..30
  //   other rows:        A entries 0..5, BT entries 6 + c
  //   pressure rows:     B entries 4 c + q
  //   warps 5..7:        A^{-1} row 12..38, W 39..42, S^{-1} row 43..46
  T R[47];
  uint4 s0 = {0, 0, 0, 0}, s1 = {0, 0, 0, 0};
  unsigned bts = 0;
  if (vtx) {
    const T *p = V + 4 * t;
#pragma unroll
    for (int q = 0; q < 4; ++q) ld4(p + q * 256, R[4 * q], R[4 * q + 1], R[4 * q + 2], R[4 * q + 3]);
#pragma unroll
    for (int c = 0; c < 3; ++c)
      ld4(p + kOffTV + c * 256, R[16 + 4 * c], R[17 + 4 * c], R[18 + 4 * c], R[19 + 4 * c]);
  } else if (edge) {
    const int li = t - 64;
#pragma unroll
    for (int q = 0; q < 2; ++q)
      ld4(V + kOffE + (q * 96 + li) * 4, R[4 * q], R[4 * q + 1], R[4 * q + 2], R[4 * q + 3]);
    ld2(V + kOffE2 + li * 2, R[8], R[9]);
#pragma unroll
    for (int c = 0; c < 3; ++c) ld2(V + kOffTE + (c * 96 + li) * 2, R[16 + 4 * c], R[17 + 4 * c]);
  } else if (rest) {
    const int li = t - 160;
    ld4(V + kOffR + li * 4, R[0], R[1], R[2], R[3]);
    ld2(V + kOffR2 + li * 2, R[4], R[5]);
#pragma unroll
    for (int c = 0; c < 3; ++c) R[6 + c] = __ldcs(V + kOffTR + c * 64 + li);
  }
  if (warp < 7) {
    s0 = __ldg(reinterpret_cast<const uint4 *>(pat.slot[t]));
    if (warp < 5) s1 = __ldg(reinterpret_cast<const uint4 *>(pat.slot[t]) + 1);
    bts = __ldg(reinterpret_cast<const unsigned *>(pat.bt[t]));
  } else {  // B rows: the D block of the factors in the order of the CSR row
    bts = __ldg(reinterpret_cast<const unsigned *>(pat.bj[lane]));
    unsigned o[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = (bts >> (8 * q)) & 0xff;
      o[q] = __ldg(&pat.own[j]);
#pragma unroll
      for (int c = 0; c < 3; ++c)
        R[4 * c + q] = j < NU_LOC ? __ldg(F + S1::offD + (sub * 3 + c) * NU_LOC + j) : T(0);
    }
    s0.x = o[0] | (o[1] << 16);
    s0.y = o[2] | (o[3] << 16);
  }
  // right-hand side: lane 0..2 of a row its component, lane 0 of a B row
  const int k = warp * 4 + sub;  // row in c_rows order
  const int row = c_rows[k < 27 ? k : 27];
  T f = T(0);
  if (k < NU_LOC && sl < 3) f = __ldcg(rhs + (size_t)sl * nu + (__ldg(ids + kPatchOwn + row) >> 2));
  if (warp == 7 && sl == 0) f = __ldcg(rhs + (size_t)3 * nu + __ldg(ids + kPatchBase) + sub);
  // block solve: warps 5..7 one component each, warps 0..3 one row of D each
  const bool solver = warp >= 5;
  const int comp = warp - 5;
  const bool in = lane < NU_LOC;
  if (solver) {
#pragma unroll
    for (int j = 0; j < NU_LOC; ++j) R[12 + j] = in ? __ldcs(F + j * NU_LOC + lane) : T(0);
#pragma unroll
    for (int m = 0; m < NP_LOC; ++m) {
      R[39 + m] = in ? __ldcs(F + S1::offW + (m * 3 + comp) * NU_LOC + lane) : T(0);
      R[43 + m] = lane < NP_LOC ? __ldg(F + S1::offS + m * NP_LOC + lane) : T(0);  // S^{-1}[lane][m]
    }
  } else if (warp < NP_LOC) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
      R[28 + c] = in ? __ldcs(F + S1::offD + (warp * 3 + c) * NU_LOC + lane) : T(0);
  }

  // ---- current values of the patch
  wait_previous();
  {
    auto at = [&](int e) {  // the copy that holds node e >> 2 at this colour's turn
      return (size_t)((e ^ ((e >> 1) & odd)) & 1) * nu + (e >> 2);
    };
    T x, y, z;
    const Node<T> n0 = Node<T>::load(L.u, at(id0));
    if (t + kPatchThreads < kPatchNodes) {
      const Node<T> n1 = Node<T>::load(L.u, at(id1));
      comps(n1, x, y, z);
      sm.u.set(t + kPatchThreads, x, y, z);
    }
    if (t < 27) {
#pragma unroll
      for (int m = 0; m < NP_LOC; ++m) sm.p[t][m] = __ldcg(L.p + pb + m);
    }
    comps(n0, x, y, z);
    sm.u.set(t, x, y, z);
    if (t == kPatchThreads - 1) {
      sm.u.set(kZeroSlot, T(0), T(0), T(0));
#pragma unroll
      for (int m = 0; m < NP_LOC; ++m) sm.p[27][m] = T(0);
    }
  }
  __syncthreads();

  // ---- local residual
  {
    const unsigned sw[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    T c0 = 0, c1 = 0, c2 = 0;
    const T *ps = &sm.p[0][0];
    auto a_entry = [&](int q) {
      T x, y, z;
      sm.u.get((sw[q >> 1] >> (16 * (q & 1))) & 0xffff, x, y, z);
      c0 += R[q] * x;
      c1 += R[q] * y;
      c2 += R[q] * z;
    };
    auto bt_entry = [&](int q, int at, int stride) {
      const T pc = ps[(bts >> (8 * q)) & 0xff];
      c0 += R[at] * pc;
      c1 += R[at + stride] * pc;
      c2 += R[at + 2 * stride] * pc;
    };
    if (vtx) {
#pragma unroll
      for (int q = 0; q < 8; ++q) a_entry(q);
#pragma unroll
      for (int q = 0; q < 4; ++q) bt_entry(q, 16 + q, 4);
#pragma unroll
      for (int q = 8; q < 16; ++q) a_entry(q);
    } else if (edge) {
#pragma unroll
      for (int q = 0; q < 8; ++q) a_entry(q);
#pragma unroll
      for (int q = 0; q < 2; ++q) bt_entry(q, 16 + q, 4);
#pragma unroll
      for (int q = 8; q < 10; ++q) a_entry(q);
    } else if (rest) {
#pragma unroll
      for (int q = 0; q < 6; ++q) a_entry(q);
      bt_entry(0, 6, 1);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        T g0, g1, g2;
        sm.u.get((sw[q >> 1] >> (16 * (q & 1))) & 0xffff, g0, g1, g2);
        c0 += R[q] * g0 + R[4 + q] * g1 + R[8 + q] * g2;
      }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      c0 += __shfl_xor_sync(kFull, c0, o);
      if (warp < 7) {
        c1 += __shfl_xor_sync(kFull, c1, o);
        c2 += __shfl_xor_sync(kFull, c2, o);
      }
    }
    if (k < NU_LOC && sl < 3) sm.r[sl][row] = f - (sl == 0 ? c0 : (sl == 1 ? c1 : c2));
    if (warp == 7 && sl == 0) sm.rp[sub] = f - c0;
  }
  __syncthreads();

  // ---- y = A^{-1} r, one component per warp
  T y = 0;
  if (solver) {
#pragma unroll
    for (int j = 0; j < NU_LOC; ++j) y += R[12 + j] * sm.r[comp][j];
    sm.y[comp][lane] = y;
  }
  __syncthreads();

  // ---- t = r_p - D y, p = S^{-1} t, x = y - W p
  if (warp < NP_LOC) {
    const T s = warp_sum(R[28] * sm.y[0][lane] + R[29] * sm.y[1][lane] + R[30] * sm.y[2][lane]);
    if (lane == 0) sm.t[warp] = sm.rp[warp] - s;
  }
  __syncthreads();
  if (solver) {
    T pk = 0;
#pragma unroll
    for (int m = 0; m < NP_LOC; ++m) pk += R[43 + m] * sm.t[m];
#pragma unroll
    for (int m = 0; m < NP_LOC; ++m) y -= R[39 + m] * __shfl_sync(kFull, pk, m);
    if (in) {
      const int me = __ldg(ids + kPatchOwn + lane);
      const unsigned single = (unsigned)__ldg(ids + kPatchSingle);
      // into the other copy, unless the node belongs to this cell alone
      const int copy = (me ^ ((me >> 1) & odd)) & 1;
      const int w = ((single >> lane) & 1) ? copy : copy ^ 1;
      T v = sm.u.get(__ldg(&pat.own[lane]), comp);
      v += damp * y;
      Node<T>::component(L.u, (size_t)w * nu + (me >> 2))[comp] = v;
    }
    if (warp == 7 && lane < NP_LOC) {
      T v = sm.p[0][lane];
      v += damp * pk;
      L.p[__ldg(ids + kPatchBase) + lane] = v;
    }
  }
}

// u -> the copies (both), u on the Dirichlet nodes taken from the right-hand
// side; p -> its copy
template <typename T>
__global__ void k_patch_pack_u(PatchLevel<T> L, const T *__restrict__ u, const T *__restrict__ rhs,
                               int hb, int np) {
  const int nu = L.nu, n = nu > np ? nu : np;
  start_next();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (i < nu) {
      const T *s = i < hb ? u : rhs;
      const Node<T> v = make_node(s[i], s[(size_t)nu + i], s[(size_t)2 * nu + i]);
      v.store(L.u, i);
      v.store(L.u, (size_t)nu + i);
    }
    if (i < np) L.p[i] = u[(size_t)3 * nu + i];
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

// the current copies -> u (Dirichlet nodes from the right-hand side) and p
template <typename T>
__global__ void k_patch_unpack_u(PatchLevel<T> L, T *__restrict__ u, const T *__restrict__ rhs,
                                 int hb, int np, int odd) {
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
        x = rhs[i];
        y = rhs[(size_t)nu + i];
        z = rhs[(size_t)2 * nu + i];
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

// Pattern of a cell from the CSR patterns and its patch list (once per level,
// at set-up).  MODE 0: a hash of the pattern into hash[cell]; 1: the pattern
// of cell which[blockIdx.x] into patterns[blockIdx.x]; 2: compare with the
// pattern that the cell was given.  Rows that do not fit set *bad.
template <int MODE>
__global__ void __launch_bounds__(256) k_patch_pattern(
    const int *ids_all, const int *a_rowptr, const int *a_col, const int *b_rowptr,
    const int *b_col, const int *bt_rowptr, const int *bt_col, int nact, const int *which,
    PatchPattern *patterns, const int *pattern, unsigned long long *hash, int *bad) {
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
  for (int i = t; i < kRowLanes * 16; i += 256) (&pt.slot[0][0])[i] = (uint16_t)kZeroSlot;
  for (int i = t; i < kRowLanes * 4; i += 256) (&pt.bt[0][0])[i] = (uint8_t)kZeroP;
  if (t < 128) (&pt.bj[0][0])[t] = (uint8_t)NU_LOC;
  if (t < 32) pt.own[t] = (uint16_t)kZeroSlot;
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
      pt.own[t] = (uint16_t)s;
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
        pt.slot[8 * k + (j & 7)][j >> 3] = (uint16_t)s;
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
        reinterpret_cast<const unsigned long long *>(patterns + pattern[cell]);
    bool differ = false;
    for (int i = t; i < words; i += 256) differ |= v[i] != w[i];
    if (differ) atomicOr(bad, 1);
  }
}

inline int ok() { return cudaPeekAtLastError() == cudaSuccess ? 1 : -1; }

// launch that may start while the previous kernel of the stream still runs
// (the kernel waits for it with griddepcontrol.wait)
template <typename... Args>
int launch_chained(void (*kernel)(Args...), int grid, int block, cudaStream_t s,
                   const Args &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess ? 1 : -1;
}

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
int launch_patch_pattern(int mode, const int *ids, const DevOp<T> &op, int n, const int *which,
                         void *patterns, const int *pattern, unsigned long long *hash, int *bad,
                         cudaStream_t s) {
  if (n <= 0) return 0;
  PatchPattern *p = static_cast<PatchPattern *>(patterns);
  auto run = [&](auto kernel) {
    kernel<<<n, 256, 0, s>>>(ids, op.a_rowptr, op.a_col, op.b_rowptr, op.b_col, op.bt_rowptr,
                             op.bt_col, op.nact, which, p, pattern, hash, bad);
  };
  if (mode == 0)
    run(k_patch_pattern<0>);
  else if (mode == 1)
    run(k_patch_pattern<1>);
  else
    run(k_patch_pattern<2>);
  return ok();
}

template <typename T>
int launch_patch_begin(const PatchLevel<T> &L, const T *u, const T *rhs, int hb, int np,
                       cudaStream_t s) {
  k_patch_pack_u<T><<<node_grid(std::max(L.nu, np)), 256, 0, s>>>(L, u, rhs, hb, np);
  return ok();
}

template <typename T>
int launch_patch_colour(const PatchLevel<T> &L, const int *list, int n, const T *factors,
                        const T *rhs, T damp, int odd, cudaStream_t s) {
  if (n <= 0) return 0;
  return launch_chained<PatchLevel<T>, const int *, const T *, const T *, T, int>(
      k_patch_sweep<T>, n, kPatchThreads, s, L, list, factors, rhs, damp, odd);
}

template <typename T>
int launch_patch_between(const PatchLevel<T> &L, const T *rhs, int hb, cudaStream_t s) {
  if (hb >= L.nu) return 0;
  return launch_chained<PatchLevel<T>, const T *, int>(k_patch_dirichlet<T>, node_grid(L.nu - hb),
                                                       256, s, L, rhs, hb);
}

template <typename T>
int launch_patch_end(const PatchLevel<T> &L, T *u, const T *rhs, int hb, int np, int odd,
                     cudaStream_t s) {
  return launch_chained<PatchLevel<T>, T *, const T *, int, int, int>(
      k_patch_unpack_u<T>, node_grid(std::max(L.nu, np)), 256, s, L, u, rhs, hb, np, odd);
}

#define PM_PINST(T)                                                                               \
  template int launch_patch_pack<T>(const PatchLevel<T> &, const DevOp<T> &, int, cudaStream_t);  \
  template int launch_patch_pattern<T>(int, const int *, const DevOp<T> &, int, const int *,      \
                                       void *, const int *, unsigned long long *, int *,          \
                                       cudaStream_t);                                             \
  template int launch_patch_begin<T>(const PatchLevel<T> &, const T *, const T *, int, int,       \
                                     cudaStream_t);                                               \
  template int launch_patch_colour<T>(const PatchLevel<T> &, const int *, int, const T *,         \
                                      const T *, T, int, cudaStream_t);                           \
  template int launch_patch_between<T>(const PatchLevel<T> &, const T *, int, cudaStream_t);      \
  template int launch_patch_end<T>(const PatchLevel<T> &, T *, const T *, int, int, int,          \
                                   cudaStream_t);
PM_PINST(double)
PM_PINST(float)
#undef PM_PINST

}  // namespace pm
