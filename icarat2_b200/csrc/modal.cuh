// K u on the voxel grid through the modes of the box element (FP64 and FP32).
//
// The hexa8 box is symmetric under reflection in its three mid-planes.  In
// the basis of corner sums and differences per axis (a 2 x 2 x 2 Hadamard
// transform of the 8 corners, per displacement component) the 24 x 24 Ke0
// therefore falls apart into one 3 x 3 block per parity class, and those
// blocks into 45 non-zero coefficients: the three translations carry no
// stiffness, and parity leaves at most 2 x 2 coupling in six of the eight
// classes.  K u costs about 165 FP64 operations per element that way (xy
// transform of one new node layer 24, z sums and differences 21, blocks 45,
// back 18, scaling and the sum with the layer below 24, inverse transform 24,
// sum over the 4 elements of a node 9) against 588 for the products with
// Ke0's 3 x 3 blocks, which held the FP64 pipe at its limit.
//
// A block owns a tile of W x H element columns; the thread of element column
// (tx, ty) is also the thread of the node column at the element's lower
// corner.  The block marches along z: node layers arrive in a ring of shared
// tiles (cp.async, kModalAhead layers ahead, so loads hold no registers),
// every thread transforms its element's face, combines it with the face below,
// and keeps the upper face's forces for the next layer; the forces of a
// finished node layer are transformed back and passed to the three
// neighbouring nodes through shared memory.  The tile completes W - 1 node
// columns of its W (all W where its first node is on the box face), so tiles
// overlap by one element column and z chunks by one element layer; modal_plan
// picks W, H and the chunk for the least sum of both (27 x 7 tiles and 13
// layers at 129 x 65 x 65 nodes).
//
// Bound by latency (12 warps per SM, the loads and barriers of a layer; FP64
// pipe one third active).  Measured on a B200, cold caches, one K u, before
// (thread per node column, 3 x 3 blocks) and now: FP64 44.1 -> 24.6 us at
// 128 x 64 x 64 elements, 277 -> 128 us at 256 x 128 x 128; FP32 30.0 -> 19.0
// and 140 -> 78 us.
#pragma once
#include <map>
#include <mutex>
#include <set>
#include <tuple>
#include <utility>

#include "internal.cuh"

namespace icarat_b200
{

// Threads per block and resident blocks per SM.  FP64 needs 154 to 168
// registers (two faces, the carried forces, the epilogue's loads): 12 warps
// per SM.  At 16 warps (128 registers) it spills and takes 30.9 us instead of
// 24.6 at 129 x 65 x 65 nodes; one block of 384 threads takes 33.8, three of
// 128 threads 23.6 (but 129 against 128 us at 257 x 129 x 129).
template <typename T> struct ModalCfg
{
  static constexpr int threads = sizeof(T) == 8 ? 192 : 256;
  static constexpr int blocks = sizeof(T) == 8 ? 2 : 3;
  static constexpr int side = 32; // largest W and H
  // node tile (W + 1)(H + 1) for W H <= threads and W, H <= side
  static constexpr int nodes = threads + side + (threads + side - 1) / side + 1;
};
constexpr int kModalRing = 8;  // node layers in shared memory (a power of two)
constexpr int kModalAhead = 4; // layers a copy is started ahead

// Work items: ntx x nty tiles of W x H element columns times ceil(NZ / kc)
// chunks of kc node layers.
struct ModalPlan
{
  int W, H, ntx, nty, kc, items;
};

template <typename T> struct ModalShared
{
  T node[kModalRing][3][ModalCfg<T>::nodes];
  T force[2][9][ModalCfg<T>::threads];
};

// The plan for `slots` resident blocks on `sms` SMs.  Cost of a wave: its
// longest chunk, (kc + 1) element layers and about two layers of start-up,
// times the larger of one block's latency per layer and the SM's work for
// its blocks' warps, about 9 to 1 per warp.  Results do not depend on the plan.
inline ModalPlan modal_plan(const GridDev &g, int threads, int side, int slots, int sms)
{
  static std::mutex mu;
  static std::map<std::tuple<int, int, int, int, int, int>, ModalPlan> cache;
  const auto key = std::make_tuple(g.NX, g.NY, g.NZ, threads, slots, sms);
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if(it != cache.end())
    return it->second;
  ModalPlan best{0, 0, 0, 0, 0, 0};
  double best_cost = 0.0;
  int last_w = 0;
  // rows of fewer than 16 nodes waste most of the sectors they load (30 to 45
  // us at W 8 .. 12 against 26 at 17, 129 x 65 x 65 nodes)
  const int wmin = g.NX < 16 ? 2 : 16;
  for(int ntx = 1; ntx < g.NX; ntx++)
  {
    const int W = (g.NX - 1 + ntx - 1) / ntx + 1;
    if(W > side || W == last_w)
      continue;
    if(W < wmin && best.W)
      break;
    last_w = W;
    const int hmax = threads / W < side ? threads / W : side;
    const int nty = (g.NY - 1 + hmax - 2) / (hmax - 1);
    const int H = (g.NY - 1 + nty - 1) / nty + 1;
    const int tx = (g.NX - 1 + W - 2) / (W - 1);
    const long tiles = (long)tx * nty;
    const int warps = (W * H + 31) / 32;
    for(int kc = 1; kc <= g.NZ; kc++)
    {
      const long chunks = (g.NZ + kc - 1) / kc;
      if(kc > 1 && (g.NZ + kc - 2) / (kc - 1) == chunks)
        continue; // the same number of chunks, longer
      const long items = tiles * chunks;
      if(items > 2000000000L)
        continue;
      auto wave = [&](long blocks) {
        const long per_sm = (blocks + sms - 1) / sms;
        const double load = (double)(per_sm * warps);
        return (kc + 3.0) * (load > 9.0 ? load : 9.0);
      };
      const double cost =
          (double)(items / slots) * wave(slots) + (items % slots ? wave(items % slots) : 0.0);
      // narrow tiles load short rows: a tie goes to the wider one
      if(best.W == 0 || cost < best_cost)
      {
        best = ModalPlan{W, H, tx, nty, kc, (int)items};
        best_cost = cost;
      }
    }
  }
  if(cache.size() > 256)
    cache.clear();
  cache[key] = best;
  return best;
}

// plan, block count (capped) and dynamic shared memory of a launch of
// `kernel`; the shared-memory limit is raised once per kernel and device
template <typename T>
inline ModalPlan modal_launch(const GridDev &g, const void *kernel, int sms, int cap, int &blocks,
                              size_t &smem)
{
  static std::mutex mu;
  static std::set<std::pair<int, const void *>> ready;
  smem = sizeof(ModalShared<T>);
  {
    // (FP32: 46 KB, above the default limit with a kernel's static arrays)
    const auto key = std::make_pair(device_slot(), kernel);
    std::lock_guard<std::mutex> lock(mu);
    if(!ready.count(key))
    {
      ICK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      ready.insert(key);
    }
  }
  using C = ModalCfg<T>;
  const ModalPlan m = modal_plan(g, C::threads, C::side, C::blocks * sms, sms);
  blocks = m.items < cap ? m.items : cap;
  return m;
}

// the block's dynamic shared memory
template <typename T> __device__ __forceinline__ ModalShared<T> &modal_shared()
{
  extern __shared__ __align__(16) unsigned char modal_smem_raw[];
  return *reinterpret_cast<ModalShared<T> *>(modal_smem_raw);
}

// one value global -> shared without a register (0 where !valid)
template <typename T>
__device__ __forceinline__ void modal_copy(T *dst, const T *src, bool valid)
{
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = valid ? (int)sizeof(T) : 0;
  if(sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(n)
                 : "memory");
}

// what an epilogue r = b - K u needs of a node
template <typename T> struct ModalRhs
{
  unsigned fix;
  T b[3];
};
template <typename T>
__device__ __forceinline__ ModalRhs<T> modal_rhs(const GridDev &g, const uint8_t *fix, const T *b,
                                                 int n)
{
  return ModalRhs<T>{fix[n], {b[n], b[(long)g.numnp + n], b[2L * g.numnp + n]}};
}

// The march's input: a node vector (component-major), or an equation vector
// of the ABI (free components only, node by node: node n's are at base[n],
// in component order).  copy() starts the copies of node n for this thread's
// staging slot q; next() is told, a layer ahead, which node comes next there.
template <typename T> struct ModalNodes
{
  const T *u;
  int numnp;
  __device__ __forceinline__ void next(int, int, bool) {}
  __device__ __forceinline__ void copy(int, int n, bool v, T *d0, T *d1, T *d2)
  {
    const T *src = u + (v ? n : 0);
    modal_copy(d0, src, v);
    modal_copy(d1, src + numnp, v);
    modal_copy(d2, src + 2L * numnp, v);
  }
};
struct ModalEquations
{
  const double *u;
  const int *base;
  const uint8_t *fix;
  int at[2];
  unsigned f[2];
  __device__ __forceinline__ void next(int q, int n, bool v)
  {
    f[q] = v ? fix[n] : 7u;
    at[q] = v ? base[n] : 0;
  }
  __device__ __forceinline__ void copy(int q, int, bool, double *d0, double *d1, double *d2)
  {
    const unsigned g = ~f[q];
    const double *src = u + at[q];
    const int o1 = g & 1, o2 = o1 + ((g >> 1) & 1);
    modal_copy(d0, (g & 1) ? src : u, (g & 1) != 0);
    modal_copy(d1, (g & 2) ? src + o1 : u, (g & 2) != 0);
    modal_copy(d2, (g & 4) ? src + o2 : u, (g & 4) != 0);
  }
};

// x and y sums and differences of the element's four nodes on one layer:
// f[c][q], bit 0 of q the x difference, bit 1 the y difference
template <typename T>
__device__ __forceinline__ void modal_face(const T (&tile)[3][ModalCfg<T>::nodes], int at, int row,
                                           T (&f)[3][4])
{
#pragma unroll
  for(int c = 0; c < 3; c++)
  {
    const T a = tile[c][at], b = tile[c][at + 1];
    const T d = tile[c][at + row], e = tile[c][at + row + 1];
    const T s0 = a + b, d0 = b - a, s1 = d + e, d1 = e - d;
    f[c][0] = s0 + s1;
    f[c][1] = d0 + d1;
    f[c][2] = s1 - s0;
    f[c][3] = d1 - d0;
  }
}

// One element between the faces f0 (below) and f1 (above), modulus E: F = the
// lower face's total (this element's and, in carry, the one below), carry =
// this element's part of the upper face.  The xy parities make four groups of
// three face modes that never mix, so each is finished before the next.
template <typename T>
__device__ __forceinline__ void modal_element(const KhParam<T> &k, T E, const T (&f0)[3][4],
                                              const T (&f1)[3][4], T (&carry)[3][4],
                                              T (&F)[3][4])
{
  auto full = [](const T(&m)[6], T x, T y, T z, T &ox, T &oy, T &oz) {
    ox = fma(m[2], z, fma(m[1], y, m[0] * x));
    oy = fma(m[4], z, fma(m[3], y, m[1] * x));
    oz = fma(m[5], z, fma(m[4], y, m[2] * x));
  };
  auto pair = [](const T(&m)[3], T x, T y, T &ox, T &oy) {
    ox = fma(m[1], y, m[0] * x);
    oy = fma(m[2], y, m[1] * x);
  };
  auto sum = [&](int c, int q) { return f0[c][q] + f1[c][q]; };
  auto dif = [&](int c, int q) { return f1[c][q] - f0[c][q]; };
  auto both = [&](int c, int q, T gs, T gd) {
    F[c][q] = fma(E, gs - gd, carry[c][q]);
    carry[c][q] = E * (gs + gd);
  };
  auto only_dif = [&](int c, int q, T gd) { // the z sum is a translation
    F[c][q] = fma(-E, gd, carry[c][q]);
    carry[c][q] = E * gd;
  };
  T a, b, c, d, e, f;
  full(k.c0, sum(0, 1), sum(1, 2), dif(2, 0), a, b, c);
  pair(k.c4, dif(0, 1), dif(1, 2), d, e);
  both(0, 1, a, d);
  both(1, 2, b, e);
  only_dif(2, 0, c);
  pair(k.c1, sum(1, 3), dif(2, 1), a, b);
  pair(k.c5, dif(0, 0), sum(2, 1), c, d);
  both(1, 3, a, k.s5 * dif(1, 3));
  both(2, 1, d, b);
  only_dif(0, 0, c);
  pair(k.c2, sum(0, 3), dif(2, 2), a, b);
  pair(k.c6, dif(1, 0), sum(2, 2), c, d);
  both(0, 3, a, k.s6 * dif(0, 3));
  both(2, 2, d, b);
  only_dif(1, 0, c);
  pair(k.c3, sum(0, 2), sum(1, 1), a, b);
  full(k.c7, dif(0, 2), dif(1, 1), sum(2, 3), c, d, e);
  f = k.s3 * dif(2, 3);
  both(0, 2, a, c);
  both(1, 1, b, d);
  both(2, 3, e, f);
}

// K u of the plan's items of this block (blockIdx.x, + gridDim.x, ...).  Every
// thread of the block must call it.  In the thread of a node's column,
// load(n) returns what the epilogue needs of node n and emit(n, acc, uc, pre)
// receives the node's K u (unmasked), its own displacement and that.  One
// barrier per layer: the forces of a layer and the epilogue's loads cross it,
// and the layer is summed and emitted at the start of the next layer's turn
// (two force buffers).
template <typename T, typename S, typename L, typename F>
__device__ __forceinline__ void modal_march(const GridDev &g, const ModalPlan &m,
                                            const KhParam<T> &kh, const T *__restrict__ E, S src,
                                            ModalShared<T> &sh, L &&load, F &&emit)
{
  const int t = threadIdx.x;
  const int tx = t % m.W, ty = t / m.W;
  const int row = m.W + 1, tile_nodes = row * (m.H + 1);
  const bool active = t < m.W * m.H;
  const int at = active ? ty * row + tx : 0;
  const int plane = g.NX * g.NY, eplane = g.nx * g.ny;
  for(int item = blockIdx.x; item < m.items; item += gridDim.x)
  {
    const int bx = item % m.ntx, by = (item / m.ntx) % m.nty;
    const int k0 = item / (m.ntx * m.nty) * m.kc;
    const int k1 = min(k0 + m.kc, g.NZ);
    const int x0 = bx * (m.W - 1), y0 = by * (m.H - 1);
    const int i = x0 + tx, j = y0 + ty;
    const bool elem = active && i < g.nx && j < g.ny;
    const bool node = active && i < g.NX && j < g.NY && (tx > 0 || bx == 0) && (ty > 0 || by == 0);
    // staged node positions of this thread: in-plane offsets, -1 outside
    int off[2];
#pragma unroll
    for(int q = 0; q < 2; q++)
    {
      const int e = t + q * ModalCfg<T>::threads;
      const int x = x0 + e % row, y = y0 + e / row;
      off[q] = (e < tile_nodes && x < g.NX && y < g.NY) ? x + y * g.NX : -1;
    }
    auto stage = [&](int k) { // node layer k into its ring slot
      if(k <= k1)
      {
        const bool in = k >= 0 && k < g.NZ;
        T(&dst)[3][ModalCfg<T>::nodes] = sh.node[(k - k0 + 1) & (kModalRing - 1)];
#pragma unroll
        for(int q = 0; q < 2; q++)
        {
          const int e = t + q * ModalCfg<T>::threads;
          if(e < tile_nodes)
          {
            src.copy(q, off[q] + k * plane, in && off[q] >= 0, &dst[0][e], &dst[1][e], &dst[2][e]);
            src.next(q, off[q] + (k + 1) * plane, k + 1 >= 0 && k + 1 < g.NZ && off[q] >= 0);
          }
        }
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto modulus = [&](int e) {
      return elem && e >= 0 && e < g.nz ? __ldg(E + i + j * g.nx + e * eplane) : T(0);
    };
    T own[3];
    decltype(load(0)) pre;
    const int n0 = i + j * g.NX;
    auto finish = [&](int k) { // sum and emit node layer k
      if(node)
      {
        const T(&fb)[9][ModalCfg<T>::threads] = sh.force[k & 1];
        const T(&tile)[3][ModalCfg<T>::nodes] = sh.node[(k - k0 + 1) & (kModalRing - 1)];
        T un[3];
#pragma unroll
        for(int c = 0; c < 3; c++)
        {
          un[c] = tile[c][at];
          if(tx > 0)
            own[c] += fb[3 * c][t - 1];
          if(ty > 0)
            own[c] += fb[3 * c + 1][t - m.W];
          if(tx > 0 && ty > 0)
            own[c] += fb[3 * c + 2][t - m.W - 1];
        }
        emit(n0 + k * plane, own, un, pre);
      }
    };
    if(item != (int)blockIdx.x)
      __syncthreads(); // the previous item's last layer has been read
#pragma unroll
    for(int q = 0; q < 2; q++)
      src.next(q, off[q] + (k0 - 1) * plane, k0 >= 1 && off[q] >= 0);
#pragma unroll
    for(int q = 0; q <= kModalAhead; q++)
      stage(k0 - 1 + q);
    T Ee = modulus(k0 - 1);
    T f0[3][4], carry[3][4];
#pragma unroll
    for(int c = 0; c < 3; c++)
#pragma unroll
      for(int q = 0; q < 4; q++)
        carry[c][q] = T(0);
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kModalAhead) : "memory");
    __syncthreads();
    modal_face(sh.node[0], at, row, f0);
#pragma unroll 1
    for(int e = k0 - 1; e < k1; e++)
    {
      // node layer e + 1 has landed, the forces of layer e - 1 are written,
      // and the slots of layers up to e - 2 are free
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kModalAhead - 1) : "memory");
      __syncthreads();
      stage(e + 1 + kModalAhead);
      const T En = modulus(e + 1);
      if(e > k0)
        finish(e - 1);
      T f1[3][4], f[3][4];
      modal_face(sh.node[(e - k0 + 2) & (kModalRing - 1)], at, row, f1);
      modal_element(kh, Ee, f0, f1, carry, f);
      if(e >= k0)
      {
        T(&fb)[9][ModalCfg<T>::threads] = sh.force[e & 1];
#pragma unroll
        for(int c = 0; c < 3; c++)
        {
          const T a0 = f[c][0] - f[c][2], b0 = f[c][1] - f[c][3];
          const T a1 = f[c][0] + f[c][2], b1 = f[c][1] + f[c][3];
          own[c] = a0 - b0;
          fb[3 * c][t] = a0 + b0;     // to the node at +x
          fb[3 * c + 1][t] = a1 - b1; // +y
          fb[3 * c + 2][t] = a1 + b1; // +x +y
        }
        if(node)
          pre = load(n0 + e * plane);
      }
#pragma unroll
      for(int c = 0; c < 3; c++)
#pragma unroll
        for(int q = 0; q < 4; q++)
          f0[c][q] = f1[c][q];
      Ee = En;
    }
    __syncthreads();
    finish(k1 - 1);
  }
}

// the same on a node vector u
template <typename T, typename L, typename F>
__device__ __forceinline__ void modal_march(const GridDev &g, const ModalPlan &m,
                                            const KhParam<T> &kh, const T *__restrict__ E,
                                            const T *u, ModalShared<T> &sh, L &&load, F &&emit)
{
  modal_march(g, m, kh, E, ModalNodes<T>{u, g.numnp}, sh, load, emit);
}

} // namespace icarat_b200
