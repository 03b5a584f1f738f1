// Direct solver of the coarsest multigrid level in FP64.
//
// The coarsest operator A (n x n SPD, n = free DOFs of the coarsest grid)
// changes with every design, so each design computes W = L^-1 of its
// Cholesky factor A = L L^T, and every V-cycle solves A x = b as
// x = W^T (W b) with two triangular matrix-vector products.
//
// Order: nested dissection by node planes across the longest axis.  A node
// couples to the planes either side only, so a plane separates what lies
// left and right of it; the planes are split D times by middle planes, and the
// tree of 2^D leaves and 2^D - 1 separators is numbered in postorder.  Row r
// of W is then zero outside its node's subtree (one contiguous range), and
// nodes of one height do not depend on one another.  At 17 x 9 x 9 nodes
// (3,888 unknowns, D = 3) W holds 23 MB instead of the 60 MB of the plane
// order's dense triangle, so W and W^T stay in L2 between V-cycles, and the
// chain of 64-column steps is 20 instead of 61 long: the set-up takes 0.92 ms
// (3.58 before), the two products of a V-cycle 20 us (43).  At 9 x 5 x 5
// (600 unknowns, D = 2, 7 steps instead of 10) the set-up takes 0.26 ms (0.60).
//
// Factorization, heights from the leaves up, all nodes of a height together:
// the matrix [A | I] is eliminated 64 columns at a time.  A node's panel
// holds its columns for its own rows and for the rows of the (at most two)
// separators its subtree touches.  Per step
//   scaling (k_coarse_scale): D = W_kk^-1 .. the 64 x 64 diagonal block's
//     inverse factor W_kk, then L_ik = A_ik W_kk^T down the panel and
//     E_k = W_kk E_k along the rows of the identity side, which is row block
//     k of W, done (stored with its transpose);
//   update (k_coarse_update): A_ij -= L_ik L_jk^T in the panel and in the
//     separators' own panels, E_i -= L_ik E_k for every later row i.
// Each tile is one 64 x 64 x 64 product on the FP64 units: mma.sync m8n8k4 f64
// takes 17 us for one on a whole SM here, scalar FMAs 3.5 (7,000 cycles; 4,096
// at the pipe's rate).  A separator receives from the
// subtree on each of its sides: the right one adds into an accumulator of its
// own (no two tiles of a launch share a target) that k_coarse_add joins.
#include <algorithm>
#include <cstring>

#include "coarse.cuh"
#include "internal.cuh"

namespace icarat_b200
{

namespace
{
constexpr int kB = 64;  // block size
constexpr int kLd = 66; // row of a staged tile: 4 banks apart, so that 16-byte reads of 16 rows
                        // (two steps of k) take two passes over the banks, the fewest
constexpr int kTile = kB * kLd;
constexpr size_t kScaleSmem = 3 * kTile * sizeof(double);
constexpr size_t kUpdateSmem = 2 * kTile * sizeof(double);
constexpr int kLongRow = 1024; // rows of W longer than this take a block of their own

// 1 / x and 1 / sqrt(x) for x > 0 by Newton's method from the hardware's
// approximations (y <- y (2 - x y), and y <- y (3/2 - x y^2 / 2)): each step
// doubles the correct digits, so two steps take a seed of ~2^-20 past double
// precision.  Inline FMAs only: an out-of-line divide or square root would save
// the register-resident rows to the stack.
__device__ __forceinline__ double recip_newton(double x)
{
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#pragma unroll
  for(int it = 0; it < 2; it++)
    y = y * fma(-x, y, 2.0);
  return y;
}

__device__ __forceinline__ double rsqrt_newton(double x)
{
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#pragma unroll
  for(int it = 0; it < 2; it++)
    y = y * fma(-0.5 * x, y * y, 1.5);
  return y;
}

// Inverse of the 16 x 16 Cholesky factor of the block at S (lower part) into W
// (zeros above its diagonal), by one warp: lanes 0-15 hold the rows of the
// block (symmetric), lanes 16-31 the rows of the identity side.  A column j
// subtracts m_r = a_rj / a_jj times row j from the rows r > j of both sides;
// the pivots' square roots scale the inverse at the end.  The chain of pivots
// is what takes time, so two columns go together: the second pivot's
// reciprocal is p11 / (p11 p22 - p12^2) and does not wait for the first's.
// What lies left of the pivots on the block's side is not used again and may
// hold anything.
__device__ __forceinline__ void factor16(const double *S, double *W, int lane)
{
  constexpr unsigned all = 0xffffffffu;
  const int r = lane & 15;
  const bool block = lane < 16;
  double x[16], piv = 1.0;
#pragma unroll
  for(int c = 0; c < 16; c++)
    x[c] = block ? S[max(r, c) * kLd + min(r, c)] : (r == c ? 1.0 : 0.0);
#pragma unroll
  for(int j = 0; j < 16; j += 2)
  {
    const double p11 = __shfl_sync(all, x[j], j), p12 = __shfl_sync(all, x[j + 1], j);
    const double p22 = __shfl_sync(all, x[j + 1], j + 1);
    const double c1 = __shfl_sync(all, x[j], r), c2 = __shfl_sync(all, x[j + 1], r);
    const double i2 = p11 * recip_newton(fma(-p12, p12, p11 * p22));
    const double i1 = recip_newton(p11), l21 = p12 * i1;
    const double m1 = r > j ? -c1 * i1 : 0.0;
    const double m2 = r > j + 1 ? -fma(-c1, l21, c2) * i2 : 0.0;
    const double b1 = block ? m1 : 0.0, b2 = block ? m2 : 0.0;
    if(r == j)
      piv = p11;
    if(r == j + 1)
      piv = fma(-p12, l21, p22);
#pragma unroll
    for(int t = 0; t < 16; t++)
    {
      const int c = (t + j + 2) & 15; // the next pivots' columns first
      const bool right = c > j + 1;
      const double v1 = __shfl_sync(all, x[c], right ? j : 16 + j);
      const double v2 = fma(-l21, v1, __shfl_sync(all, x[c], right ? j + 1 : 17 + j));
      x[c] = fma(right ? b2 : m2, v2, fma(right ? b1 : m1, v1, x[c]));
    }
  }
  if(!block)
  {
    const double y = rsqrt_newton(piv);
#pragma unroll
    for(int c = 0; c < 16; c++)
      W[r * kLd + c] = c <= r ? x[c] * y : 0.0;
  }
}

// Columns [C, C + 16) of factor64, whose diagonal block has been factored.
__device__ __forceinline__ void factor64_step(int C, double *S, double *W)
{
  const int NB = (kB - 16 - C) / 16; // 16-row blocks below
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double *Wd = W + C * kLd + C;
  // 48 vectors x of 16: the rows of S below (L_i = S_i W_d^T) and the columns of
  // W left of the block (E = W_d E); W_d x in place
  double out[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for(int k = 0; k < 16; k++)
  {
    const double w = Wd[tx * kLd + k];
#pragma unroll
    for(int u = 0; u < 3; u++)
      out[u] = fma(w, u < NB ? S[(C + 16 + 16 * u + ty) * kLd + C + k]
                             : W[(C + k) * kLd + 16 * (u - NB) + ty], out[u]);
  }
  __syncthreads();
#pragma unroll
  for(int u = 0; u < 3; u++)
    if(u < NB)
      S[(C + 16 + 16 * u + ty) * kLd + C + tx] = out[u];
    else
      W[(C + tx) * kLd + 16 * (u - NB) + ty] = out[u];
  __syncthreads();
  if(NB == 0)
    return;
  double *L = S + (C + 16) * kLd + C; // rows below, 16 columns
  if(threadIdx.x < 32)
  {
    // the first warp: the next diagonal block and its factor
    const int r = threadIdx.x & 15, c0 = 8 * (threadIdx.x >> 4);
    double acc[8] = {};
#pragma unroll 4
    for(int k = 0; k < 16; k++)
    {
      const double a = L[r * kLd + k];
#pragma unroll
      for(int c = 0; c < 8; c++)
        acc[c] = fma(a, L[(c0 + c) * kLd + k], acc[c]);
    }
    double *D = L + 16;
#pragma unroll
    for(int c = 0; c < 8; c++)
      D[r * kLd + c0 + c] -= acc[c];
    __syncwarp();
    factor16(D, W + (C + 16) * kLd + C + 16, threadIdx.x);
  }
  else
  {
    // the others: the rest of the rows below, 64 columns in all, S_ij -= L_i L_j^T
    // (16-column blocks j <= i) and E_i -= L_i E; 14 rows at a time
    const int y = ty - 2;
    double acc[4][4] = {};
#pragma unroll 4
    for(int k = 0; k < 16; k++)
    {
      double b[4];
#pragma unroll
      for(int q = 0; q < 4; q++)
        b[q] = q < NB ? L[(16 * q + tx) * kLd + k] : W[(C + k) * kLd + 16 * (q - NB) + tx];
#pragma unroll
      for(int i = 0; i < 4; i++)
      {
        const double a = L[min(y + 14 * i, 16 * NB - 1) * kLd + k];
#pragma unroll
        for(int q = 0; q < 4; q++)
          acc[i][q] = fma(a, b[q], acc[i][q]);
      }
    }
#pragma unroll
    for(int i = 0; i < 4; i++)
    {
      const int row = y + 14 * i;
      if(row < 16 * NB)
#pragma unroll
        for(int q = 0; q < 4; q++)
          if(q >= NB)
            W[(C + 16 + row) * kLd + 16 * (q - NB) + tx] -= acc[i][q];
          else if(row >= 16 && q <= row / 16)
            L[row * kLd + 16 + 16 * q + tx] -= acc[i][q];
    }
  }
  __syncthreads();
}

// W (64 x 64, zero on entry) = inverse Cholesky factor of the block S (lower
// part; overwritten), 256 threads: [S | W] eliminated 16 columns at a time, as
// the whole matrix is by 64.  16 columns are what one warp holds in registers;
// the rest of a step is small products over the other warps meanwhile.
__device__ void factor64(double *S, double *W)
{
  if(threadIdx.x < 32)
    factor16(S, W, threadIdx.x);
  __syncthreads();
#pragma unroll 1
  for(int c = 0; c < kB; c += 16)
    factor64_step(c, S, W);
}

// stage rows x cols (<= 64 x 64, row length ld) as a 64 x 64 tile, zeros past
// the end
__device__ __forceinline__ void stage_tile(double *T, const double *g, int ld, int rows, int cols)
{
  const int c = threadIdx.x & 63;
  double v[16];
#pragma unroll
  for(int u = 0; u < 16; u++)
  {
    const int r = (threadIdx.x >> 6) + 4 * u;
    v[u] = (r < rows && c < cols) ? g[(long)r * ld + c] : 0.0;
  }
#pragma unroll
  for(int u = 0; u < 16; u++)
    T[((threadIdx.x >> 6) + 4 * u) * kLd + c] = v[u];
}

// 64 x 64 product of two staged tiles, A B (BT false) or A B^T: thread
// (ty, tx) of 16 x 16 has rows ty + 16 i and columns tx + 16 q, two steps of k
// at a time.  A warp reads 12 passes of shared memory for 64 FMA cycles.
template <bool BT>
__device__ __forceinline__ void tile_product(double (&acc)[4][4], const double *A,
                                             const double *B)
{
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 4
  for(int k = 0; k < kB; k += 2)
  {
    double2 a[4], b[4];
#pragma unroll
    for(int i = 0; i < 4; i++)
      a[i] = *reinterpret_cast<const double2 *>(A + (ty + 16 * i) * kLd + k);
#pragma unroll
    for(int q = 0; q < 4; q++)
      b[q] = BT ? *reinterpret_cast<const double2 *>(B + (tx + 16 * q) * kLd + k)
                : make_double2(B[k * kLd + tx + 16 * q], B[(k + 1) * kLd + tx + 16 * q]);
#pragma unroll
    for(int i = 0; i < 4; i++)
#pragma unroll
      for(int q = 0; q < 4; q++)
        acc[i][q] = fma(a[i].y, b[q].y, fma(a[i].x, b[q].x, acc[i][q]));
  }
}

// f(i, q, row, column) for each element [i][q] of a thread's share
template <typename F> __device__ __forceinline__ void tile_each(F f)
{
#pragma unroll
  for(int i = 0; i < 4; i++)
#pragma unroll
    for(int q = 0; q < 4; q++)
      f(i, q, (int)(threadIdx.x >> 4) + 16 * i, (int)(threadIdx.x & 15) + 16 * q);
}

// the 64 x kw block T of row block k0 of node X's part of W, columns from
// global unknown c: into W, and transposed into W^T (rows: the columns here)
__device__ __forceinline__ void store_inverse(const CoarseNode &X, const CoarseNode *nodes,
                                              const int *node_of, int k0, int kw, int c, int cols,
                                              const double *T, double *W, double *U)
{
  const int x = threadIdx.x & 63;
  for(int y = threadIdx.x >> 6; y < kw; y += 4)
    if(x < cols)
      W[X.W + (long)(k0 + y) * X.S + (c - X.lo) + x] = T[y * kLd + x];
  for(int y = threadIdx.x >> 6; y < cols; y += 4)
    if(x < kw)
    {
      const CoarseNode &Y = nodes[node_of[c + y]];
      U[Y.U + (long)(c + y - Y.s) * Y.C + (Y.C - X.C) + k0 + x] = T[x * kLd + y];
    }
}
} // namespace

// panels of the nodes of one height += their second accumulators
__global__ void k_coarse_add(const CoarseNode *__restrict__ nodes, int height,
                             double *__restrict__ P)
{
  chain_wait();
  const CoarseNode X = nodes[blockIdx.y];
  if(X.height != height)
    return;
  const int total = X.m * X.m;
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x)
    P[X.P + i] += P[X.Q + i];
}

// One step's scaling: every block factors its node's diagonal block itself,
// which saves a launch and a round trip through memory.  The pivots' serial
// chain bounds it (31,000 cycles in the kernel, 16 us; column by column 45,000;
// the product after it takes 3.5 us).  A launch of its own, with cold caches,
// takes 33 to 36 us under a profiler; in the set-up's graph a step of scaling
// and update takes 46 us.
__global__ void __launch_bounds__(256)
    k_coarse_scale(const CoarseNode *__restrict__ nodes, const int *__restrict__ node_of,
                   const CoarseScaleTile *__restrict__ tiles, double *P, double *W, double *U)
{
  chain_wait();
  extern __shared__ double coarse_smem[];
  double *S = coarse_smem, *Wk = S + kTile, *T = Wk + kTile;
  const CoarseScaleTile tile = tiles[blockIdx.x];
  const CoarseNode X = nodes[tile.node];
  const int k0 = tile.k0, kw = min(kB, X.m - k0);
  stage_tile(S, P + X.P + (long)k0 * X.m + k0, X.m, kw, kw);
  for(int i = threadIdx.x; i < kTile; i += 256)
    Wk[i] = 0.0;
  const int rows = min(kB, X.m + X.ml + X.mr - tile.first);       // of a panel tile
  const int cols = min(kB, X.s + k0 - X.lo - tile.first);         // of an inverse tile
  double *panel = P + X.P + (long)tile.first * X.m + k0;
  if(tile.kind == kTilePanel)
    stage_tile(T, panel, X.m, rows, kw);
  else if(tile.kind == kTileInverse)
    stage_tile(T, W + X.W + (long)k0 * X.S + tile.first, X.S, kw, cols);
  __syncthreads();
  if((int)threadIdx.x >= kw && threadIdx.x < kB) // identity past the last column
    S[threadIdx.x * kLd + threadIdx.x] = 1.0;
  __syncthreads();
  factor64(S, Wk);
  if(tile.kind == kTileDiag)
  {
    store_inverse(X, nodes, node_of, k0, kw, X.s + k0, kw, Wk, W, U);
    return;
  }
  double acc[4][4] = {};
  if(tile.kind == kTilePanel)
  {
    tile_product<true>(acc, T, Wk);
    tile_each([&](int i, int q, int row, int col) {
      if(row < rows && col < kw)
        panel[(long)row * X.m + col] = acc[i][q];
    });
    return;
  }
  tile_product<false>(acc, Wk, T);
  tile_each([&](int i, int q, int row, int col) { S[row * kLd + col] = acc[i][q]; });
  __syncthreads();
  store_inverse(X, nodes, node_of, k0, kw, X.lo + tile.first, cols, S, W, U);
}

// One step's updates, bound by the FP64 units where tiles are many; two blocks to
// an SM (three spill) hide the loads.
__global__ void __launch_bounds__(256, 2)
    k_coarse_update(const CoarseUpdateTile *__restrict__ tiles, double *P, double *W)
{
  chain_wait();
  extern __shared__ double coarse_smem[];
  double *A = coarse_smem, *B = A + kTile;
  const CoarseUpdateTile g = tiles[blockIdx.x];
  stage_tile(A, P + g.a, g.lda, g.M, g.K);
  if(g.from_w)
    stage_tile(B, W + g.b, g.ldb, g.K, g.N);
  else
    stage_tile(B, P + g.b, g.ldb, g.N, g.K);
  __syncthreads();
  // all of the tile is fetched before the first of it is stored, under the
  // product
  double *C = (g.to_w ? W : P) + g.c;
  double acc[4][4] = {}, old[4][4];
  tile_each([&](int i, int q, int row, int col) {
    const bool in = row < g.M && col < g.N && (!g.lower || col <= row);
    old[i][q] = in ? C[(long)row * g.ldc + col] : 0.0;
  });
  if(g.from_w)
    tile_product<false>(acc, A, B);
  else
    tile_product<true>(acc, A, B);
  tile_each([&](int i, int q, int row, int col) {
    if(row < g.M && col < g.N && (!g.lower || col <= row))
      C[(long)row * g.ldc + col] = old[i][q] - acc[i][q];
  });
}

// t = W v, blocks of 8 warps: a row each, or one long row together
__global__ void __launch_bounds__(256)
    k_coarse_lower(int n, CoarseRows R, const int *__restrict__ items,
                   const double *__restrict__ W, const double *v, double *__restrict__ t,
                   const int *__restrict__ halt)
{
  chain_wait();
  if(halted(halt))
    return;
  __shared__ double part[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int item = items[blockIdx.x];
  if(item >= 0) // up to the next item's first row
  {
    const int next = items[blockIdx.x + 1], r = item + warp;
    if(r < (next >= 0 ? next : -next - 1))
    {
      const double s = coarse_warp_sum(coarse_dot(W + R.wofs[r], v, R.lo[r], r + 1, lane, 0.0));
      if(lane == 0)
        t[r] = s;
    }
    return;
  }
  const int r = -item - 1, lo = R.lo[r], per = ((r + 1 - lo + 7) / 8 + 31) & ~31;
  const int j0 = lo + warp * per, j1 = min(r + 1, j0 + per);
  const double s = coarse_warp_sum(coarse_dot(W + R.wofs[r], v, j0, j1, lane, 0.0));
  if(lane == 0)
    part[warp] = s;
  __syncthreads();
  if(threadIdx.x == 0)
    t[r] = ((part[0] + part[1]) + (part[2] + part[3])) +
           ((part[4] + part[5]) + (part[6] + part[7]));
}

// x[rowmap] = W^T t, one warp per row
template <typename T>
__global__ void __launch_bounds__(256)
    k_coarse_upper(int n, CoarseRows R, const double *__restrict__ WT, const double *t,
                   const int *__restrict__ rowmap, T *__restrict__ x,
                   const int *__restrict__ halt)
{
  chain_wait();
  if(halted(halt))
    return;
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if(r >= n)
    return;
  const double s = coarse_upper_row(R, WT, t, r, lane);
  if(lane == 0)
    x[rowmap[r]] = (T)s;
}

// ---------------------------------------------------------------- the tree
namespace
{
struct TreeBuilder
{
  const std::vector<int> &pf; // first unknown of each plane
  std::vector<int> &order;
  std::vector<CoarseNode> nodes;
  std::vector<int> parent;

  // planes [p0, p1), `depth` levels of separators below; returns the root
  int build(int p0, int p1, int depth)
  {
    const int lo = (int)order.size();
    int kid[2] = {-1, -1}, s0 = p0, s1 = p1;
    if(depth > 0)
    {
      s0 = p0 + (p1 - p0) / 2;
      s1 = s0 + 1;
      kid[0] = build(p0, s0, depth - 1);
      kid[1] = build(s1, p1, depth - 1);
    }
    CoarseNode X{};
    X.s = (int)order.size();
    for(int i = pf[s0]; i < pf[s1]; i++)
      order.push_back(i);
    X.m = (int)order.size() - X.s;
    X.lo = lo;
    X.S = X.s + X.m - lo;
    X.left = X.right = -1;
    X.height = depth;
    const int id = (int)nodes.size();
    nodes.push_back(X);
    parent.push_back(-1);
    if(depth > 0)
    {
      parent[kid[0]] = parent[kid[1]] = id;
      border(kid[0], false, id);
      border(kid[1], true, id);
    }
    return id;
  }
  // separator `sep` lies left (right) of the subtree of x: of x itself and of
  // the nodes down its left (right) edge
  void border(int x, bool left, int sep)
  {
    for(;;)
    {
      (left ? nodes[x].left : nodes[x].right) = sep;
      if(nodes[x].height == 0)
        return;
      // children of x in postorder: the right one is x - 1, the left one
      // ends before the right one's subtree
      const int right_kid = x - 1;
      const int left_kid = right_kid - ((2 << nodes[right_kid].height) - 1);
      x = left ? left_kid : right_kid;
    }
  }
};

// the tree's tables, in one device allocation
struct TablePacker
{
  std::vector<char> bytes;
  template <typename T> size_t add(const std::vector<T> &v)
  {
    const size_t at = (bytes.size() + 15) & ~size_t(15);
    bytes.resize(at + v.size() * sizeof(T));
    if(!v.empty())
      memcpy(bytes.data() + at, v.data(), v.size() * sizeof(T));
    return at;
  }
};
} // namespace

void coarse_tree_free(CoarseTree &t)
{
  cudaFree(t.tables);
  t = CoarseTree{};
}

void coarse_tree_build(CoarseTree &t, const std::vector<int> &pf, std::vector<int> &order)
{
  const int planes = (int)pf.size() - 1;
  t.n = pf[planes];
  int widest = 1;
  for(int p = 0; p < planes; p++)
    widest = std::max(widest, pf[p + 1] - pf[p]);
  // depth: split while every leaf keeps a plane and the chain of 64-column
  // steps (a leaf's and one separator's per level) does not grow
  auto steps = [&](int d)
  {
    const int leaf = (planes - ((1 << d) - 1) + (1 << d) - 1) >> d; // planes of the largest
    return (leaf * widest + kB - 1) / kB + d * ((widest + kB - 1) / kB);
  };
  int depth = 0;
  while(depth < kCoarseDepth && planes >= (4 << depth) - 1 && steps(depth + 1) <= steps(depth))
    depth++;
  order.clear();
  TreeBuilder b{pf, order, {}, {}};
  if(t.n > 0)
    b.build(0, planes, depth);
  std::vector<CoarseNode> &N = b.nodes;
  const int nn = (int)N.size();
  t.nnodes = nn;
  std::vector<int2> chain((size_t)kCoarseChain * nn, make_int2(0, 0));
  for(int i = nn - 1; i >= 0; i--) // ancestors come after their descendants
  {
    CoarseNode &X = N[i];
    X.ml = X.left >= 0 ? N[X.left].m : 0;
    X.mr = X.right >= 0 ? N[X.right].m : 0;
    X.C = X.m + (b.parent[i] >= 0 ? N[b.parent[i]].C : 0);
    int k = 0;
    for(int y = i; y >= 0; y = b.parent[y])
      chain[(size_t)kCoarseChain * i + k++] = make_int2(N[y].s, N[y].m);
  }
  for(CoarseNode &X : N)
  {
    X.P = t.nP;
    t.nP += (long)(X.m + X.ml + X.mr) * X.m;
    X.Q = -1;
    if(X.height > 0)
    {
      X.Q = t.nP;
      t.nP += (long)X.m * X.m;
    }
    X.W = t.nW;
    t.nW += (long)X.m * X.S;
    X.U = t.nU;
    t.nU += (long)X.m * X.C;
  }
  std::vector<long> wofs(t.n), uofs(t.n);
  std::vector<int> lo(t.n), node(t.n), items;
  for(int i = 0; i < nn; i++)
    for(int q = 0; q < N[i].m; q++)
    {
      const CoarseNode &X = N[i];
      const int r = X.s + q;
      wofs[r] = X.W + (long)q * X.S - X.lo;
      uofs[r] = X.U + (long)q * X.C + q;
      lo[r] = X.lo;
      node[r] = i;
    }
  for(int r = 0; r < t.n;)
    if(r + 1 - lo[r] > kLongRow)
      items.push_back(-(r++) - 1);
    else
    {
      items.push_back(r);
      for(int k = 0; k < 8 && r < t.n && r + 1 - lo[r] <= kLongRow; k++)
        r++;
    }
  t.nitems = (int)items.size();
  items.push_back(t.n); // ends the last item
  // launch tables
  std::vector<CoarseScaleTile> scale;
  std::vector<CoarseUpdateTile> upd;
  auto product = [&](long a, int lda, long bo, int ldb, bool from_w, long c, int ldc, bool to_w,
                     int M, int Nc, int K, bool lower)
  {
    for(int i = 0; i < M; i += kB)
      for(int j = 0; j < Nc && (!lower || j <= i); j += kB)
        upd.push_back({a + (long)i * lda, from_w ? bo + j : bo + (long)j * ldb,
                       c + (long)i * ldc + j, lda, ldb, ldc, (short)std::min(kB, M - i),
                       (short)std::min(kB, Nc - j), (short)K, (short)from_w,
                       (short)(lower && i == j), (short)to_w});
  };
  // row of separator y in the panel of x
  auto panel_row = [&](int x, int y) { return N[x].m + (y == N[x].left ? 0 : N[x].ml); };
  for(int h = 0; h <= depth && nn > 0; h++)
  {
    int most = 0;
    for(const CoarseNode &X : N)
      if(X.height == h)
        most = std::max(most, X.m);
    for(int k0 = 0; k0 < most; k0 += kB)
    {
      CoarseStep st{};
      st.join = k0 == 0 ? h : 0;
      st.scale0 = (int)scale.size();
      st.upd0 = (int)upd.size();
      for(int x = 0; x < nn; x++)
      {
        const CoarseNode &X = N[x];
        if(X.height != h || k0 >= X.m)
          continue;
        const int kw = std::min(kB, X.m - k0), next = k0 + kw, rows = X.m + X.ml + X.mr;
        const int before = X.s + k0 - X.lo, done = before + kw; // columns of the inverse side
        scale.push_back({x, k0, kTileDiag, 0});
        for(int r = next; r < rows; r += kB)
          scale.push_back({x, k0, kTilePanel, r});
        for(int c = 0; c < before; c += kB)
          scale.push_back({x, k0, kTileInverse, c});
        auto L = [&](int row) { return X.P + (long)row * X.m + k0; };
        // own columns: the lower triangle of the node, all of the border rows
        product(L(next), X.m, L(next), X.m, false, X.P + (long)next * X.m + next, X.m, false,
                X.m - next, X.m - next, kw, true);
        product(L(X.m), X.m, L(next), X.m, false, X.P + (long)X.m * X.m + next, X.m, false,
                X.ml + X.mr, X.m - next, kw, false);
        // rows of the inverse side
        const long Ek = X.W + (long)k0 * X.S;
        product(L(next), X.m, Ek, X.S, true, X.W + (long)next * X.S, X.S, true, X.m - next, done,
                kw, false);
        for(int y : {X.left, X.right})
          if(y >= 0)
          {
            const CoarseNode &Y = N[y];
            product(L(panel_row(x, y)), X.m, Ek, X.S, true, Y.W + (X.lo - Y.lo), Y.S, true, Y.m,
                    done, kw, false);
            product(L(panel_row(x, y)), X.m, L(panel_row(x, y)), X.m, false,
                    y == X.left ? Y.Q : Y.P, Y.m, false, Y.m, Y.m, kw, true);
          }
        if(X.left >= 0 && X.right >= 0)
        {
          // the deeper separator's panel holds the rows of the other
          const int d = N[X.left].height < N[X.right].height ? X.left : X.right;
          const int u = d == X.left ? X.right : X.left;
          product(L(panel_row(x, u)), X.m, L(panel_row(x, d)), X.m, false,
                  N[d].P + (long)panel_row(d, u) * N[d].m, N[d].m, false, N[u].m, N[d].m, kw,
                  false);
        }
      }
      st.scales = (int)scale.size() - st.scale0;
      st.upds = (int)upd.size() - st.upd0;
      t.steps.push_back(st);
    }
  }
  TablePacker pk;
  const size_t at[9] = {pk.add(N),    pk.add(scale), pk.add(upd),  pk.add(items), pk.add(wofs),
                        pk.add(uofs), pk.add(lo),    pk.add(node), pk.add(chain)};
  const cudaError_t e = cudaMalloc(&t.tables, pk.bytes.size() + 1);
  if(e != cudaSuccess)
    throw Error{ICARAT_ERR_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e)};
  ICK(cudaMemcpy(t.tables, pk.bytes.data(), pk.bytes.size(), cudaMemcpyHostToDevice));
  t.nodes = reinterpret_cast<CoarseNode *>(t.tables + at[0]);
  t.scale = reinterpret_cast<CoarseScaleTile *>(t.tables + at[1]);
  t.upd = reinterpret_cast<CoarseUpdateTile *>(t.tables + at[2]);
  t.items = reinterpret_cast<int *>(t.tables + at[3]);
  t.rows.wofs = reinterpret_cast<long *>(t.tables + at[4]);
  t.rows.uofs = reinterpret_cast<long *>(t.tables + at[5]);
  t.rows.lo = reinterpret_cast<int *>(t.tables + at[6]);
  t.rows.node = reinterpret_cast<int *>(t.tables + at[7]);
  t.rows.chain = reinterpret_cast<int2 *>(t.tables + at[8]);
}

// W = L^-1 and W^T (in U) of the matrix in the panels P (which it overwrites)
void coarse_factor(cudaStream_t st, const CoarseTree &t, double *P, double *W, double *U)
{
  ICK(cudaFuncSetAttribute(k_coarse_scale, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kScaleSmem));
  ICK(cudaFuncSetAttribute(k_coarse_update, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kUpdateSmem));
  ICK(cudaMemsetAsync(W, 0, sizeof(double) * t.nW, st));
  for(const CoarseStep &s : t.steps)
  {
    if(s.join > 0)
    {
      note_launch();
      launch_chained(k_coarse_add, dim3(16, t.nnodes), 256, 0, st,
                     (const CoarseNode *)t.nodes, s.join, P);
    }
    note_launch();
    launch_chained(k_coarse_scale, s.scales, 256, kScaleSmem, st, (const CoarseNode *)t.nodes,
                   t.rows.node, (const CoarseScaleTile *)t.scale + s.scale0, P, W, U);
    if(s.upds > 0)
    {
      note_launch();
      launch_chained(k_coarse_update, s.upds, 256, kUpdateSmem, st,
                     (const CoarseUpdateTile *)t.upd + s.upd0, P, W);
    }
  }
  ICK(cudaGetLastError());
}

// x[rowmap] = W^T W v; both products return at entry while *halt != 0 (halt
// null: never)
template <typename T>
void coarse_solve(cudaStream_t st, const CoarseTree &t, const double *W, const double *U,
                  const double *v, double *y, const int *rowmap, T *x, const int *halt)
{
  note_launch(2);
  launch_chained(k_coarse_lower, t.nitems, 256, 0, st, t.n, t.rows, (const int *)t.items, W, v,
                 y, halt);
  launch_chained(k_coarse_upper<T>, (t.n * 32 + 255) / 256, 256, 0, st, t.n, t.rows, U,
                 (const double *)y, rowmap, x, halt);
}

template void coarse_solve<double>(cudaStream_t, const CoarseTree &, const double *,
                                   const double *, const double *, double *, const int *,
                                   double *, const int *);
template void coarse_solve<float>(cudaStream_t, const CoarseTree &, const double *,
                                  const double *, const double *, double *, const int *, float *,
                                  const int *);

} // namespace icarat_b200
