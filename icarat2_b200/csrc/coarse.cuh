// Coarsest-level direct solver: the data its kernels and the multigrid share.
#pragma once
#include <vector>

namespace icarat_b200
{

constexpr int kCoarseDepth = 5;               // levels of separators at most
constexpr int kCoarseChain = kCoarseDepth + 1; // a node and its ancestors

// The rows of W and of W^T by unknown.  Entry (r, j) of W, lo[r] <= j <= r,
// is W[wofs[r] + j]; the entries of row r of W^T are contiguous from
// WT[uofs[r]]: the rest of r's node, then each ancestor whole, as
// chain[kCoarseChain node[r] + k] = (first unknown, count) lists them
// (count 0 ends the list; entry 0 is the node itself).
struct CoarseRows
{
  const long *wofs, *uofs;
  const int *lo, *node;
  const int2 *chain;
};

// One node of the elimination tree: unknowns [s, s + m), the unknowns of its
// subtree from lo (S of them with its own), C unknowns from here up the chain
// of ancestors.  P: the panel, m columns by m own rows, then ml + mr rows of
// the separators left and right of the subtree; Q: a separator's second m x m
// accumulator; W: m rows of L^-1 by S columns; U: m rows of its transpose by C.
struct CoarseNode
{
  int s, m, lo, S, C, ml, mr, left, right, height;
  long P, Q, W, U;
};

// a 64 x 64 tile of the scaling pass of one 64-column step
enum CoarseTileKind : int { kTileDiag, kTilePanel, kTileInverse };
struct CoarseScaleTile
{
  int node, k0, kind, first; // first: panel row / column of the subtree
};

// a 64 x 64 tile of the update pass: C -= A B (B from W) or A B^T (B from P)
struct CoarseUpdateTile
{
  long a, b, c;
  int lda, ldb, ldc;
  short M, N, K, from_w, lower, to_w;
};

struct CoarseStep
{
  int join;           // height whose accumulators are joined first (0: none)
  int scale0, scales; // scaling tiles
  int upd0, upds;     // update tiles
};

struct CoarseTree
{
  int n = 0, nnodes = 0;
  long nP = 0, nW = 0, nU = 0; // doubles of the panels, of W and of W^T
  std::vector<CoarseStep> steps;
  char *tables = nullptr; // the device arrays below
  CoarseNode *nodes = nullptr;
  CoarseScaleTile *scale = nullptr;
  CoarseUpdateTile *upd = nullptr;
  int *items = nullptr; // blocks of the lower product
  int nitems = 0;
  CoarseRows rows{};
};

// plane_first[p]: first unknown of plane p (p = planes: their number), in
// the order of the planes; order[i] becomes the plane-order unknown that the
// solver numbers i
void coarse_tree_build(CoarseTree &t, const std::vector<int> &plane_first,
                       std::vector<int> &order);
void coarse_tree_free(CoarseTree &t);

// where entry (r, c), c <= r, of the coarsest matrix lies in the panels
__device__ __forceinline__ long coarse_entry(const CoarseNode *nodes, const int *node, int r,
                                             int c)
{
  const int x = node[c], y = node[r];
  const CoarseNode &X = nodes[x];
  int row = r - nodes[y].s;
  if(y != x)
    row += X.m + (y == X.left ? 0 : X.ml);
  return X.P + (long)row * X.m + (c - X.s);
}

// sum over j in [j0, j1) of row[j] v[j] by one warp: eight guarded loads of
// each in flight per lane.  v may be written by other blocks of the running
// kernel, so it is read past L1.
__device__ __forceinline__ double coarse_dot(const double *__restrict__ row, const double *v,
                                             int j0, int j1, int lane, double s)
{
  for(int j = j0 + lane; j < j1; j += 256)
  {
    double a[8], b[8];
#pragma unroll
    for(int u = 0; u < 8; u++)
    {
      const bool in = j + 32 * u < j1;
      a[u] = in ? row[j + 32 * u] : 0.0;
      b[u] = in ? __ldcg(v + j + 32 * u) : 0.0;
    }
    double p[4];
#pragma unroll
    for(int u = 0; u < 4; u++)
      p[u] = fma(a[u + 4], b[u + 4], a[u] * b[u]);
    s += (p[0] + p[1]) + (p[2] + p[3]);
  }
  return s;
}

__device__ __forceinline__ double coarse_warp_sum(double s)
{
  for(int o = 16; o > 0; o >>= 1)
    s += __shfl_down_sync(0xffffffffu, s, o);
  return s;
}

// row r of W^T times y by one warp (the sum in lane 0)
__device__ __forceinline__ double coarse_upper_row(const CoarseRows &R, const double *WT,
                                                   const double *y, int r, int lane)
{
  const int2 *ch = R.chain + kCoarseChain * R.node[r];
  const double *row = WT + R.uofs[r];
  double s = 0.0;
  int done = r - ch[0].x; // own unknowns before r
  for(int k = 0; k < kCoarseChain && ch[k].y > 0; k++)
  {
    const int first = ch[k].x + done, count = ch[k].y - done;
    s = coarse_dot(row - first, y, first, first + count, lane, s);
    row += count;
    done = 0;
  }
  return coarse_warp_sum(s);
}

} // namespace icarat_b200
