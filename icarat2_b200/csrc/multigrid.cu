// Geometric multigrid preconditioner for the SIMP stiffness (no reference
// counterpart: the reference solves with Jacobi-PCG or a direct solver).
//
// Level l + 1 halves every axis of level l.  Coarse operators are
// rediscretised: a coarse element's modulus is the mean of its 8 children
// times 2 (a hexa8 stiffness scales with its edge length), so every level
// reuses the fine Ke0 and the matrix-free node stencil.  A coarse node is
// constrained where its coincident fine node is.  Transfers are trilinear
// prolongation P and restriction R = P^T.  Smoothing is a Chebyshev
// polynomial in D^-1 K on [0.1 lmax, lmax], where lmax is the element bound
// of the Jacobi-scaled Ke0 (a rigorous bound for every SIMP design), applied
// identically before and after the coarse correction so that the V-cycle is
// a symmetric positive definite preconditioner.  The coarsest level is solved
// exactly: W = L^-1 of the Cholesky factor of its dense matrix is rebuilt on
// the GPU for every design (dense.cu) and each V-cycle applies W^T W.  The
// unknowns are ordered by nested dissection in node planes across the longest
// axis.
//
// The V-cycle exists in FP64 (preconditioner of the FP64 solver) and in FP32
// (inner solver of the mixed-precision solver); the coarsest solve is FP64 in
// both.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "modal.cuh"
#include "stencil.cuh"

namespace icarat_b200
{

// dense.cu
void coarse_factor(cudaStream_t st, const CoarseTree &t, double *P, double *W, double *U);
template <typename T>
void coarse_solve(cudaStream_t st, const CoarseTree &t, const double *W, const double *U,
                  const double *v, double *y, const int *rowmap, T *x,
                  const int *halt = nullptr);

// Galerkin coarse operators (galerkin.cu)
__global__ void k_gal_cells_free(GridDev f, GridDev c, const double *__restrict__ E,
                                 const double *__restrict__ G,
                                 const uint8_t *__restrict__ flag, double *__restrict__ Kc);
__global__ void k_gal_cells(GridDev f, GridDev c, KeParam ke, const double *__restrict__ E,
                            const double *__restrict__ Kf, const uint8_t *__restrict__ fix_f,
                            const uint8_t *__restrict__ fix_c, const int *__restrict__ cells,
                            int ncells, double *__restrict__ Kc, double *__restrict__ lmax);
__global__ void k_gal_stencil(GridDev g, const double *__restrict__ Kc,
                              const uint8_t *__restrict__ fix, double *__restrict__ S,
                              double *__restrict__ invd);
__global__ void k_gal_coefs(int levels, const double *__restrict__ lmax, double lam1,
                            double *__restrict__ coef);
double galerkin_child_matrices(const double *ke0, double *G);
template <typename T>
void st_first_launch(cudaStream_t st, int n, const T *b, const T *invd, const double *coef,
                     T *x, T *d, const int *halt);
template <typename T>
void st_cheb_launch(cudaStream_t st, const GridDev &g, const T *S, const uint8_t *fix,
                    const T *invd, const T *b, const T *x, T *d, T *xo, const double *coef, int k,
                    const int *halt);
template <typename T>
void st_residual_launch(cudaStream_t st, const GridDev &g, const T *S, const uint8_t *fix,
                        const T *b, const T *x, T *r, const int *halt);
__global__ void k_coarse_assemble_st(GridDev g, const double *__restrict__ S,
                                     const CoarseNode *__restrict__ nodes,
                                     const int *__restrict__ node,
                                     const int *__restrict__ rowmap,
                                     const int *__restrict__ colmap, int nfree,
                                     double *__restrict__ P);

// ---------------------------------------------------------------- level data
__global__ void k_coarsen_E(GridDev f, GridDev c, const double *__restrict__ Ef,
                            double *__restrict__ Ec)
{
  for(int e = blockIdx.x * blockDim.x + threadIdx.x; e < c.nelx;
      e += gridDim.x * blockDim.x)
  {
    const int I = e % c.nx, J = (e / c.nx) % c.ny, K = e / (c.nx * c.ny);
    double s = 0.0;
#pragma unroll
    for(int dz = 0; dz < 2; dz++)
#pragma unroll
      for(int dy = 0; dy < 2; dy++)
#pragma unroll
        for(int dx = 0; dx < 2; dx++)
          s += Ef[(2 * I + dx) + (long)(2 * J + dy) * f.nx +
                  (long)(2 * K + dz) * f.nx * f.ny];
    Ec[e] = 0.25 * s; // mean of 8 children x 2
  }
}

template <typename Tin, typename Tout>
__global__ void k_cast(long n, const Tin *__restrict__ in, Tout *__restrict__ out)
{
  chain_wait();
  for(long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
      i += (long)gridDim.x * blockDim.x)
    out[i] = (Tout)in[i];
}

// ---------------------------------------------------------------- transfers
// Blocks are 32 x 4 node columns of one plane (the parity of a row is uniform
// in its warp), numbered along the one grid axis that no size of a grid
// exceeds: planes or rows on the other two would end at 65,535.  NC components per thread: all three on
// large levels, one on levels below kSplitNodes nodes, where the sums are
// latency and more threads shorten them (33 x 17 x 17 nodes: restriction 10.7
// -> 6.7 us; 65 x 33 x 33 is faster with three, 9.6 against 11.1).  Every load
// is issued unconditionally: a neighbour outside the grid is read as one inside
// and left out of the sum.  Bound by memory on the finest level: 257 x 129 x
// 129 nodes FP64, prolongation 62 -> 40 us (220 MB), restriction 32 -> 30.
constexpr int kSplitNodes = 1 << 15;

// the node (i, j, k) and first component of this thread; false outside
template <int NC>
__device__ __forceinline__ bool transfer_node(const GridDev &g, int &i, int &j, int &k, int &q0)
{
  const unsigned tx = (g.NX + 31) / 32, ty = (g.NY + 3) / 4;
  const unsigned row = blockIdx.x / tx, plane = row / ty;
  i = (blockIdx.x - row * tx) * 32 + threadIdx.x;
  j = (row - plane * ty) * 4 + threadIdx.y;
  k = NC == 3 ? plane : plane / 3;
  q0 = NC == 3 ? 0 : plane % 3;
  return i < g.NX && j < g.NY;
}

// coarse b = R r  (R = P^T, 27 fine nodes per coarse node, weights 1/2^d).
// With xc set, also the coarse level's first Chebyshev step from zero
// (k_cheb_first fused): xc = inv_theta invd_c bc.  With v set (coarsest level)
// also the dense solve's right-hand side through its column map.
template <typename T, int NC>
__global__ void __launch_bounds__(128)
    k_restrict(GridDev f, GridDev c, const T *__restrict__ rf, const uint8_t *__restrict__ fixc,
               T *__restrict__ bc, const T *__restrict__ invd_c, T inv_theta, T *__restrict__ xc,
               const int *__restrict__ colmap, double *__restrict__ v,
               const int *__restrict__ halt)
{
  chain_wait();
  if(halted(halt))
    return;
  int I, J, K, q0;
  if(!transfer_node<NC>(c, I, J, K, q0))
    return;
  T s[NC];
#pragma unroll
  for(int q = 0; q < NC; q++)
    s[q] = T(0);
  const int m0 = 2 * (I + J * f.NX + K * f.NX * f.NY);
#pragma unroll
  for(int dz = -1; dz <= 1; dz++)
#pragma unroll
    for(int dy = -1; dy <= 1; dy++)
#pragma unroll
      for(int dx = -1; dx <= 1; dx++)
      {
        const int i = 2 * I + dx, j = 2 * J + dy, k = 2 * K + dz;
        const bool in = i >= 0 && i < f.NX && j >= 0 && j < f.NY && k >= 0 && k < f.NZ;
        const T w = T((dx ? 0.5 : 1.0) * (dy ? 0.5 : 1.0) * (dz ? 0.5 : 1.0));
        const int m = in ? m0 + dx + dy * f.NX + dz * f.NX * f.NY : m0;
#pragma unroll
        for(int q = 0; q < NC; q++)
        {
          const T r = rf[(long)(q0 + q) * f.numnp + m];
          s[q] += in ? w * r : T(0);
        }
      }
  const int n = I + J * c.NX + K * c.NX * c.NY;
  const unsigned fx = fixc[n];
#pragma unroll
  for(int q = 0; q < NC; q++)
  {
    const int qc = q0 + q;
    const long id = (long)qc * c.numnp + n;
    const T bq = ((fx >> qc) & 1u) ? T(0) : s[q];
    bc[id] = bq;
    if(xc)
      xc[id] = inv_theta * invd_c[id] * bq;
    if(v)
    {
      const int col = colmap[3 * n + qc];
      if(col >= 0)
        v[col] = (double)bq;
    }
  }
}

// fine xo = xf + P xc (masked; xo may be xf)
template <typename T, int NC>
__global__ void __launch_bounds__(128)
    k_prolong_add(GridDev f, GridDev c, const T *__restrict__ xc, const uint8_t *__restrict__ fixf,
                  const T *xf, T *xo, const int *__restrict__ halt)
{
  chain_wait();
  if(halted(halt))
    return;
  int i, j, k, q0;
  if(!transfer_node<NC>(f, i, j, k, q0))
    return;
  const int ox = i & 1, oy = j & 1, oz = k & 1;
  const int m0 = (i >> 1) + (j >> 1) * c.NX + (k >> 1) * c.NX * c.NY;
  const T w = (ox ? T(0.5) : T(1)) * (oy ? T(0.5) : T(1)) * (oz ? T(0.5) : T(1));
  const int n = i + j * f.NX + k * f.NX * f.NY;
  T x[NC], s[NC];
#pragma unroll
  for(int q = 0; q < NC; q++)
  {
    x[q] = xf[(long)(q0 + q) * f.numnp + n];
    s[q] = T(0);
  }
  const unsigned fx = fixf[n];
#pragma unroll
  for(int cz = 0; cz < 2; cz++)
#pragma unroll
    for(int cy = 0; cy < 2; cy++)
    {
      if((cz && !oz) || (cy && !oy)) // uniform in the warp
        continue;
      const int m = m0 + cy * c.NX + cz * c.NX * c.NY;
#pragma unroll
      for(int q = 0; q < NC; q++)
      {
        const T *src = xc + (long)(q0 + q) * c.numnp + m;
        const T r0 = src[0], r1 = src[ox];
        s[q] += w * r0;
        s[q] += ox ? w * r1 : T(0);
      }
    }
#pragma unroll
  for(int q = 0; q < NC; q++)
  {
    const int qc = q0 + q;
    xo[(long)qc * f.numnp + n] = ((fx >> qc) & 1u) ? x[q] : x[q] + s[q];
  }
}

static unsigned transfer_grid(const GridDev &g, int nc)
{
  return (unsigned)((g.NX + 31) / 32) * ((g.NY + 3) / 4) * g.NZ * (nc == 3 ? 1 : 3);
}

// ---------------------------------------------------------------- smoother
// First Chebyshev step from x = 0: d = x = invd b / theta (d null: not kept).
template <typename T>
__global__ void k_cheb_first(int n, const T *__restrict__ b, const T *__restrict__ invd,
                             T inv_theta, T *__restrict__ x, T *__restrict__ d,
                             const int *__restrict__ halt)
{
  chain_wait();
  if(halted(halt))
    return;
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
      i += gridDim.x * blockDim.x)
  {
    const T di = inv_theta * invd[i] * b[i];
    x[i] = di;
    if(d)
      d[i] = di;
  }
}

// The Krylov scalars that z . b (b the Krylov residual) of a V-cycle's last
// smoothing step gives: k_cg_zr and k_mx_zr of the separate pass.
__device__ __forceinline__ void finish_dot(const CycleDot<double> &k, const double (&t)[1])
{
  CgScalars *s = k.s;
  s->zr_new = t[0];
  s->beta = t[0] / s->zr;
  s->zr = t[0];
}
__device__ __forceinline__ void finish_dot(const CycleDot<float> &k, const double (&t)[2])
{
  MxScalars *s = k.s;
  s->zr = t[0];
  s->beta = k.first ? 0.0 : -t[1] / s->pAp;
}

// One Chebyshev step: r = b - K x, d = c1 d + c2 invd r, xo = x + d.
// x and xo are distinct buffers (neighbours of x are read by other threads).
// din null: d = x (the step after k_cheb_first) where c1 != 0; dout null: no
// step follows that reads d.  DOT: the last step of the cycle, whose result z
// the Krylov iteration takes with z . b (and z . K p where k.Ap is set).
template <typename T, bool DOT>
__global__ void __launch_bounds__(ModalCfg<T>::threads, ModalCfg<T>::blocks)
    k_cheb_step(GridDev g, ModalPlan m, KhParam<T> kh, const T *__restrict__ E,
                const uint8_t *__restrict__ fix, const T *__restrict__ invd,
                const T *__restrict__ b, const T *__restrict__ x, const T *din, T *dout,
                T *__restrict__ xo, T c1, T c2, const int *__restrict__ halt, CycleDot<T> k)
{
  chain_wait();
  ModalShared<T> &ms = modal_shared<T>();
  if(halted(halt))
    return;
  struct Pre
  {
    ModalRhs<T> r;
    T invd[3], d[3];
    T Ap[DOT && sizeof(T) == 4 ? 3 : 1];
  };
  // z . b, and z . K p in FP32; summed per thread in shared memory (the FP64
  // march has no registers left for them)
  constexpr int ND = sizeof(T) == 4 ? 2 : 1;
  __shared__ double sums[DOT ? ND : 1][DOT ? ModalCfg<T>::threads : 1];
  if(DOT)
#pragma unroll
    for(int q = 0; q < ND; q++)
      sums[DOT ? q : 0][DOT ? threadIdx.x : 0] = 0.0;
  modal_march(g, m, kh, E, x, ms,
              [&](int n) {
                Pre pre;
                pre.r = modal_rhs(g, fix, b, n);
#pragma unroll
                for(int q = 0; q < 3; q++)
                {
                  const long id = (long)q * g.numnp + n;
                  pre.invd[q] = invd[id];
                  pre.d[q] = din ? din[id] : T(0);
                  if constexpr(DOT && ND == 2)
                    pre.Ap[q] = k.Ap ? k.Ap[id] : T(0);
                }
                return pre;
              },
              [&](int n, const T(&acc)[3], const T(&uc)[3], const Pre &pre)
              {
                const unsigned f = pre.r.fix;
                double dot[ND] = {};
#pragma unroll
                for(int q = 0; q < 3; q++)
                {
                  const long id = (long)q * g.numnp + n;
                  T dn = 0;
                  if(!((f >> q) & 1u))
                    dn = (c1 != T(0) ? c1 * (din ? pre.d[q] : uc[q]) : T(0)) +
                         c2 * pre.invd[q] * (pre.r.b[q] - acc[q]);
                  if(dout)
                    dout[id] = dn;
                  const T z = uc[q] + dn;
                  xo[id] = z;
                  if(DOT)
                  {
                    dot[0] += (double)z * (double)pre.r.b[q];
                    if constexpr(DOT && ND == 2)
                      dot[1] += (double)z * (double)pre.Ap[q];
                  }
                }
                if(DOT)
#pragma unroll
                  for(int q = 0; q < ND; q++)
                    sums[DOT ? q : 0][DOT ? threadIdx.x : 0] += dot[q];
              });
  if(DOT)
  {
    __shared__ double sh[32 * ND];
    double dot[ND];
#pragma unroll
    for(int q = 0; q < ND; q++)
      dot[q] = sums[DOT ? q : 0][DOT ? threadIdx.x : 0];
    block_sum<ND>(dot, sh);
    if(threadIdx.x == 0)
#pragma unroll
      for(int q = 0; q < ND; q++)
        k.partials[q * gridDim.x + blockIdx.x] = dot[q];
    if(last_block(&k.s->counter))
    {
      double t[ND];
      sum_partials<ND>(k.partials, gridDim.x, t, sh);
      if(threadIdx.x == 0)
      {
        finish_dot(k, t);
        k.s->counter = 0;
      }
    }
  }
}

// r = b - K x (constrained rows 0)
template <typename T>
__global__ void __launch_bounds__(ModalCfg<T>::threads, ModalCfg<T>::blocks)
    k_mg_residual(GridDev g, ModalPlan m, KhParam<T> kh, const T *__restrict__ E,
                  const uint8_t *__restrict__ fix, const T *__restrict__ b,
                  const T *__restrict__ x, T *__restrict__ r, const int *__restrict__ halt)
{
  chain_wait();
  ModalShared<T> &ms = modal_shared<T>();
  if(halted(halt))
    return;
  modal_march(g, m, kh, E, x, ms,
              [&](int n) { return modal_rhs(g, fix, b, n); },
              [&](int n, const T(&acc)[3], const T(&)[3], const ModalRhs<T> &pre)
              {
                const unsigned f = pre.fix;
#pragma unroll
                for(int c = 0; c < 3; c++)
                  r[(long)c * g.numnp + n] =
                      ((f >> c) & 1u) ? T(0) : pre.b[c] - acc[c];
              });
}

// ---------------------------------------------------------------- coarse
// Coarse matrix into the panels of its factorization, one thread per free row
// and neighbour node (fixed summation order), lower part.  A thread per row
// walked its eight elements one after another: 71 us on 9 x 5 x 5 nodes,
// where ten blocks held all rows.
__global__ void k_coarse_assemble(GridDev g, KeParam ke, const double *__restrict__ E,
                                  const CoarseNode *__restrict__ nodes,
                                  const int *__restrict__ node, const int *__restrict__ rowmap,
                                  const int *__restrict__ colmap, int nfree,
                                  double *__restrict__ P)
{
  const long total = 27L * nfree;
  for(long id = blockIdx.x * (long)blockDim.x + threadIdx.x; id < total;
      id += (long)gridDim.x * blockDim.x)
  {
    const int r = (int)(id / 27), o = (int)(id % 27);
    const int full = rowmap[r]; // component-major index c * numnp + n
    const int n = full % g.numnp, c = full / g.numnp;
    const int i = n % g.NX, j = (n / g.NX) % g.NY, k = n / (g.NX * g.NY);
    const int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dz = o / 9 - 1;
    if(i + dx < 0 || i + dx >= g.NX || j + dy < 0 || j + dy >= g.NY || k + dz < 0 ||
       k + dz >= g.NZ)
      continue;
    double sum[3] = {0.0, 0.0, 0.0};
    for(int sz = 0; sz < 2; sz++)
      for(int sy = 0; sy < 2; sy++)
        for(int sx = 0; sx < 2; sx++)
        {
          const int ei = i - 1 + sx, ej = j - 1 + sy, ek = k - 1 + sz;
          const int bx = dx + 1 - sx, by = dy + 1 - sy, bz = dz + 1 - sz;
          if((unsigned)ei >= (unsigned)g.nx || (unsigned)ej >= (unsigned)g.ny ||
             (unsigned)ek >= (unsigned)g.nz || ((bx | by | bz) & ~1))
            continue;
          const double e = E[ei + (long)ej * g.nx + (long)ek * g.nx * g.ny];
          const int a = local_node(1 - sx, 1 - sy, 1 - sz), b = local_node(bx, by, bz);
#pragma unroll
          for(int d = 0; d < 3; d++)
            sum[d] += e * ke.k[(3 * a + c) * 24 + 3 * b + d];
        }
    const long m = n + dx + (long)dy * g.NX + (long)dz * g.NX * g.NY;
#pragma unroll
    for(int d = 0; d < 3; d++)
    {
      const int col = colmap[3 * m + d];
      if(col >= 0 && col <= r)
        P[coarse_entry(nodes, node, r, col)] = sum[d];
    }
  }
}

// ---------------------------------------------------------------- driver
static GridDev make_grid(int nx, int ny, int nz)
{
  return GridDev{nx, ny, nz, nx + 1, ny + 1, nz + 1, (nx + 1) * (ny + 1) * (nz + 1),
                 nx * ny * nz};
}

static int blocks_for(long n, int t)
{
  long b = (n + t - 1) / t;
  return b < 1 ? 1 : (b > 65535L * 16 ? 65535 * 16 : (int)b);
}

// level buffers of one precision
template <typename T> struct LevelBuf;
template <> struct LevelBuf<double>
{
  static double *E(MgLevel &L) { return L.E; }
  static double *invd(MgLevel &L) { return L.invd; }
  static double *x(MgLevel &L) { return L.x; }
  static double *b(MgLevel &L) { return L.b; }
  static double *r(MgLevel &L) { return L.r; }
  static double *t(MgLevel &L) { return L.t; }
  static double *S(MgLevel &L) { return L.S; }
  static const KhParam<double> &kh(icarat_ctx *c) { return c->kh; }
};
template <> struct LevelBuf<float>
{
  static float *E(MgLevel &L) { return L.E32; }
  static float *invd(MgLevel &L) { return L.invd32; }
  static float *x(MgLevel &L) { return L.x32; }
  static float *b(MgLevel &L) { return L.b32; }
  static float *r(MgLevel &L) { return L.r32; }
  static float *t(MgLevel &L) { return L.t32; }
  static float *S(MgLevel &L) { return L.S32; }
  static const KhParam<float> &kh(icarat_ctx *c) { return c->khf; }
};

void mg_free(icarat_ctx *c)
{
  for(size_t l = 0; l < c->mg.size(); l++)
  {
    MgLevel &L = c->mg[l];
    if(l > 0)
    {
      dfree(L.E);
      dfree(L.fix);
      dfree(L.invd);
      dfree(L.E32);
    }
    for(void *p : {(void *)L.x, (void *)L.b, (void *)L.r, (void *)L.t, (void *)L.invd32,
                   (void *)L.x32, (void *)L.b32, (void *)L.r32, (void *)L.t32, (void *)L.Kc,
                   (void *)L.S, (void *)L.S32})
      dfree(p);
  }
  c->mg.clear();
  dfree(c->gal_lmax);
  c->gal_lmax = nullptr;
  dfree(c->gal_G);
  c->gal_G = nullptr;
  dfree(c->gal_flag1);
  c->gal_flag1 = nullptr;
  dfree(c->gal_cells1);
  c->gal_cells1 = nullptr;
  c->gal_ncells1 = 0;
  c->gal_coef = nullptr; // part of the gal_lmax allocation
  c->mg_galerkin = 0;
  CoarseSolver &C = c->coarse;
  if(C.side)
    cudaStreamSynchronize(C.side); // a lagged factorization may still run
  for(int b = 0; b < 2; b++)
  {
    if(C.setup[b])
      cudaGraphExecDestroy(C.setup[b]);
    if(C.factor[b])
      cudaGraphExecDestroy(C.factor[b]);
    if(C.ev_factor[b])
      cudaEventDestroy(C.ev_factor[b]);
    dfree(C.P[b]);
    dfree(C.W[b]);
    dfree(C.U[b]);
  }
  if(C.levels)
    cudaGraphExecDestroy(C.levels);
  if(C.ev_levels)
    cudaEventDestroy(C.ev_levels);
  if(C.side)
    cudaStreamDestroy(C.side);
  coarse_tree_free(C.tree);
  dfree(C.map);
  dfree(C.vin);
  dfree(C.vout);
  c->coarse = CoarseSolver{};
  c->mg_built_levels = 0;
}

static float *falloc(size_t n)
{
  void *p = nullptr;
  cudaError_t e = cudaMalloc(&p, (n ? n : 1) * sizeof(float));
  if(e != cudaSuccess)
    throw Error{ICARAT_ERR_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e)};
  return static_cast<float *>(p);
}

static void allocate_factor(CoarseSolver &C, int b)
{
  C.P[b] = dalloc(C.tree.nP);
  C.W[b] = dalloc(C.tree.nW);
  C.U[b] = dalloc(C.tree.nU);
}

static void allocate_levels(icarat_ctx *c, int levels)
{
  release_graphs(c); // captured solver graphs hold pointers to level arrays
  mg_free(c);
  int nx = c->nx, ny = c->ny, nz = c->nz;
  for(int l = 0; l < levels; l++)
  {
    if(l > 0)
    {
      IREQUIRE(nx % 2 == 0 && ny % 2 == 0 && nz % 2 == 0, ICARAT_ERR_UNSUPPORTED,
               "multigrid needs divisions divisible by 2^(levels-1)");
      nx /= 2;
      ny /= 2;
      nz /= 2;
    }
    MgLevel L;
    L.g = make_grid(nx, ny, nz);
    const size_t nv = 3 * (size_t)L.g.numnp;
    if(l == 0)
    {
      L.E = c->d_E;
      L.E32 = c->d_E32;
      L.fix = c->d_fix;
      L.invd = c->d_invd;
    }
    else
    {
      L.E = dalloc(L.g.nelx);
      L.E32 = falloc(L.g.nelx);
      ICK(cudaMalloc(&L.fix, L.g.numnp));
      L.invd = dalloc(nv);
    }
    if(l > 0 && c->mg_galerkin_req)
    {
      L.Kc = dalloc(576 * (size_t)L.g.nelx);
      L.S = dalloc(126 * (size_t)L.g.numnp);
      L.S32 = falloc(126 * (size_t)L.g.numnp);
    }
    L.x = dalloc(nv);
    L.b = dalloc(nv);
    L.r = dalloc(nv);
    L.t = dalloc(nv);
    L.invd32 = falloc(nv);
    L.x32 = falloc(nv);
    L.b32 = falloc(nv);
    L.r32 = falloc(nv);
    L.t32 = falloc(nv);
    c->mg.push_back(L);
  }
  if(c->mg_galerkin_req)
  {
    // per level: the Chebyshev bound, then kGalCoef coefficients
    c->gal_lmax = dalloc((size_t)levels * (1 + kGalCoef));
    c->gal_coef = c->gal_lmax + levels;
    std::vector<double> G(8 * 576);
    c->gal_lam1 = 1.001 * galerkin_child_matrices(c->ke0.k, G.data());
    c->gal_G = dalloc(G.size());
    ICK(cudaMemcpy(c->gal_G, G.data(), sizeof(double) * G.size(), cudaMemcpyHostToDevice));
    // level-1 cells with a constrained child node (fixed for the context):
    // they take the general cell kernel, the others the free form
    const GridDev f0 = c->mg[0].g, g1 = c->mg[1].g;
    std::vector<uint8_t> flag(g1.nelx, 0);
    std::vector<int> cells;
    for(int cell = 0; cell < g1.nelx; cell++)
    {
      const int CI = cell % g1.nx, CJ = (cell / g1.nx) % g1.ny, CK = cell / (g1.nx * g1.ny);
      for(int t = 0; t < 27 && !flag[cell]; t++)
      {
        const int fx = t % 3, fy = (t / 3) % 3, fz = t / 9;
        if(c->fix_h[(2 * CI + fx) + (2L * CJ + fy) * f0.NX + (2L * CK + fz) * f0.NX * f0.NY])
          flag[cell] = 1;
      }
      if(flag[cell])
        cells.push_back(cell);
    }
    ICK(cudaMalloc(&c->gal_flag1, g1.nelx));
    ICK(cudaMemcpy(c->gal_flag1, flag.data(), g1.nelx, cudaMemcpyHostToDevice));
    c->gal_ncells1 = (int)cells.size();
    ICK(cudaMalloc(&c->gal_cells1, sizeof(int) * std::max<size_t>(1, cells.size())));
    if(!cells.empty())
      ICK(cudaMemcpy(c->gal_cells1, cells.data(), sizeof(int) * cells.size(),
                     cudaMemcpyHostToDevice));
  }
  c->mg_galerkin = c->mg_galerkin_req;
  // coarse constraint pattern on the host (fixed for the context)
  std::vector<uint8_t> fix = c->fix_h;
  GridDev gf = c->mg[0].g;
  for(int l = 1; l < levels; l++)
  {
    GridDev gc = c->mg[l].g;
    std::vector<uint8_t> fc(gc.numnp);
    for(int n = 0; n < gc.numnp; n++)
    {
      int I = n % gc.NX, J = (n / gc.NX) % gc.NY, K = n / (gc.NX * gc.NY);
      fc[n] = fix[2 * I + (long)2 * J * gf.NX + (long)2 * K * gf.NX * gf.NY];
    }
    ICK(cudaMemcpy(c->mg[l].fix, fc.data(), gc.numnp, cudaMemcpyHostToDevice));
    fix.swap(fc);
    gf = gc;
  }
  // coarse system: its unknowns by node planes across the longest axis (a node
  // couples to the planes either side only; nodes within a plane, then the 3
  // components), which the tree's order rearranges
  GridDev gc = c->mg[levels - 1].g;
  std::vector<int> full, node3; // of each unknown in the order of the planes
  std::vector<int> plane_first;
  const int ext[3] = {gc.NX, gc.NY, gc.NZ};
  int ax[3] = {0, 1, 2}; // slowest .. fastest
  std::stable_sort(ax, ax + 3, [&](int p, int q) { return ext[p] > ext[q]; });
  int id[3];
  for(id[ax[0]] = 0; id[ax[0]] < ext[ax[0]]; id[ax[0]]++)
  {
    const size_t first = full.size();
    for(id[ax[1]] = 0; id[ax[1]] < ext[ax[1]]; id[ax[1]]++)
      for(id[ax[2]] = 0; id[ax[2]] < ext[ax[2]]; id[ax[2]]++)
      {
        const int n = id[0] + gc.NX * (id[1] + gc.NY * id[2]);
        for(int q = 0; q < 3; q++)
          if(!((fix[n] >> q) & 1u))
          {
            full.push_back(q * gc.numnp + n); // component-major vector index
            node3.push_back(3 * n + q);       // node-major lookup index
          }
      }
    if(full.size() > first) // a plane without free unknowns is none
      plane_first.push_back((int)first);
  }
  const int nf = (int)full.size();
  plane_first.push_back(nf);
  IREQUIRE((double)nf * nf * 8.0 * 3 < 6.0e9, ICARAT_ERR_UNSUPPORTED,
           "coarsest multigrid level too large for the dense solve; add levels");
  c->coarse.n = nf;
  std::vector<int> order;
  coarse_tree_build(c->coarse.tree, plane_first, order);
  std::vector<int> map(nf + 3 * (size_t)gc.numnp, -1);
  for(int i = 0; i < nf; i++)
  {
    map[i] = full[order[i]];
    map[nf + (size_t)node3[order[i]]] = i;
  }
  ICK(cudaMalloc(&c->coarse.map, sizeof(int) * (map.size() + 1)));
  ICK(cudaMemcpy(c->coarse.map, map.data(), sizeof(int) * map.size(), cudaMemcpyHostToDevice));
  allocate_factor(c->coarse, 0);
  c->coarse.vin = dalloc(nf);
  c->coarse.vout = dalloc(nf);
  // the dense solve writes the free components; the constrained ones stay 0
  {
    const MgLevel &C = c->mg[levels - 1];
    ICK(cudaMemset(C.x, 0, sizeof(double) * 3 * C.g.numnp));
    ICK(cudaMemset(C.x32, 0, sizeof(float) * 3 * C.g.numnp));
  }
  c->mg_built_levels = levels;
}

// Everything on the levels that depends on the design: coarse moduli and
// Jacobi diagonals (and their FP32 copies).
static void enqueue_levels(icarat_ctx *c, int levels, cudaStream_t st)
{
  if(c->mg_galerkin)
    ICK(cudaMemsetAsync(c->gal_lmax, 0, sizeof(double) * levels, st));
  for(int l = 0; l < levels; l++)
  {
    MgLevel &L = c->mg[l];
    if(l > 0)
    {
      const MgLevel &F = c->mg[l - 1];
      note_launch();
      k_coarsen_E<<<blocks_for(L.g.nelx, 256), 256, 0, st>>>(F.g, L.g, F.E, L.E);
    }
    if(l > 0 && c->mg_galerkin)
    {
      // Galerkin: cell matrices from the level above, the node stencil, the
      // Jacobi diagonal from it, the FP32 copies
      const MgLevel &F = c->mg[l - 1];
      if(l == 1)
      {
        note_launch();
        k_gal_cells_free<<<blocks_for(576L * L.g.nelx, 256), 256, 0, st>>>(
            F.g, L.g, F.E, c->gal_G, c->gal_flag1, L.Kc);
        if(c->gal_ncells1 > 0)
        {
          note_launch();
          k_gal_cells<<<c->gal_ncells1, 128, 0, st>>>(F.g, L.g, c->ke0, F.E, nullptr, F.fix,
                                                      L.fix, c->gal_cells1, c->gal_ncells1, L.Kc,
                                                      c->gal_lmax + l);
        }
      }
      else
      {
        note_launch();
        k_gal_cells<<<L.g.nelx, 128, 0, st>>>(F.g, L.g, c->ke0, F.E, F.Kc, F.fix, L.fix, nullptr,
                                              L.g.nelx, L.Kc, c->gal_lmax + l);
      }
      note_launch(2);
      k_gal_stencil<<<blocks_for(14L * L.g.numnp, 256), 256, 0, st>>>(L.g, L.Kc, L.fix, L.S,
                                                                      L.invd);
      k_cast<<<blocks_for(126L * L.g.numnp, 256), 256, 0, st>>>(126L * L.g.numnp, L.S, L.S32);
    }
    else
      launch_diag(c, L.g, L.E, L.fix, L.invd, st);
    if(l > 0) // the finest FP32 moduli come with the design
    {
      note_launch();
      k_cast<<<blocks_for(L.g.nelx, 256), 256, 0, st>>>((long)L.g.nelx, L.E, L.E32);
    }
    note_launch();
    k_cast<<<blocks_for(3L * L.g.numnp, 256), 256, 0, st>>>(3L * L.g.numnp, L.invd,
                                                           L.invd32);
  }
  if(c->mg_galerkin)
  {
    note_launch();
    k_gal_coefs<<<1, 32, 0, st>>>(levels, c->gal_lmax, c->gal_lam1, c->gal_coef);
  }
}

// The dense coarsest matrix of the current coarsest moduli and W = L^-1 of
// its Cholesky factor, into factor buffer b.
static void enqueue_factor(icarat_ctx *c, int b, cudaStream_t st)
{
  const MgLevel &C = c->mg.back();
  const int n = c->coarse.n;
  if(n == 0)
    return;
  CoarseSolver &D = c->coarse;
  ICK(cudaMemsetAsync(D.P[b], 0, sizeof(double) * D.tree.nP, st));
  note_launch();
  if(c->mg_galerkin)
    k_coarse_assemble_st<<<blocks_for(27L * n, 256), 256, 0, st>>>(
        C.g, C.S, D.tree.nodes, D.tree.rows.node, D.map, D.map + n, n, D.P[b]);
  else
    k_coarse_assemble<<<blocks_for(27L * n, 256), 256, 0, st>>>(
        C.g, c->ke0, C.E, D.tree.nodes, D.tree.rows.node, D.map, D.map + n, n, D.P[b]);
  ICK(cudaGetLastError());
  coarse_factor(st, D.tree, D.P[b], D.W[b], D.U[b]);
}

// ||b - K_c x|| / ||b|| of the coarsest dense solve for a fixed right-hand
// side (a check of the factorization), K_c applied by the coarsest level's
// stencil.
double mg_coarse_check(icarat_ctx *c, int levels, int *n_coarse)
{
  mg_setup(c, levels);
  const MgLevel &C = c->mg.back();
  const int n = c->coarse.n;
  if(n_coarse)
    *n_coarse = n;
  if(n == 0)
    return 0.0;
  const size_t nv = 3 * (size_t)C.g.numnp;
  std::vector<int> rowmap(n);
  std::vector<double> b(n), y(nv);
  for(int i = 0; i < n; i++)
    b[i] = 1.0 + (i % 7) / 7.0;
  ICK(cudaStreamSynchronize(c->stream));
  ICK(cudaMemcpy(rowmap.data(), c->coarse.map, sizeof(int) * n, cudaMemcpyDeviceToHost));
  ICK(cudaMemcpy(c->coarse.vin, b.data(), sizeof(double) * n, cudaMemcpyHostToDevice));
  ICK(cudaMemsetAsync(C.x, 0, sizeof(double) * nv, c->stream));
  coarse_solve(c->stream, c->coarse.tree, c->coarse.W[c->coarse.cur], c->coarse.U[c->coarse.cur],
               c->coarse.vin, c->coarse.vout, c->coarse.map, C.x);
  if(c->mg_galerkin)
  {
    // A x with the stencil: the residual of b = 0 is -A x
    ICK(cudaMemsetAsync(C.b, 0, sizeof(double) * nv, c->stream));
    st_residual_launch<double>(c->stream, C.g, C.S, C.fix, C.b, C.x, C.t, nullptr);
    ICK(cudaStreamSynchronize(c->stream));
    std::vector<double> tmp(nv);
    ICK(cudaMemcpy(tmp.data(), C.t, sizeof(double) * nv, cudaMemcpyDeviceToHost));
    for(double &v : tmp)
      v = -v;
    ICK(cudaMemcpy(C.t, tmp.data(), sizeof(double) * nv, cudaMemcpyHostToDevice));
  }
  else
    launch_apply_K(c, C.g, C.E, C.fix, C.x, C.t, nullptr);
  ICK(cudaMemcpyAsync(y.data(), C.t, sizeof(double) * nv, cudaMemcpyDeviceToHost, c->stream));
  ICK(cudaStreamSynchronize(c->stream));
  double rr = 0.0, bb = 0.0;
  for(int i = 0; i < n; i++)
  {
    const double r = b[i] - y[rowmap[i]];
    rr += r * r;
    bb += b[i] * b[i];
  }
  return std::sqrt(rr / bb);
}

// y = A_level x on the host (component-major vectors of the level's 3 numnp
// entries): the operator the V-cycle applies on that level for the options'
// levels and coarse operators (constrained rows 0).
void mg_level_apply(icarat_ctx *c, const icarat_solve_opts *o, int level, const double *x,
                    double *y)
{
  const int levels = o->mg_levels > 0 ? o->mg_levels : 4;
  IREQUIRE(o->coarse_op == ICARAT_COARSE_REDISCRETISED || o->coarse_op == ICARAT_COARSE_GALERKIN,
           ICARAT_ERR_ARG, "coarse_op must be ICARAT_COARSE_REDISCRETISED or _GALERKIN");
  IREQUIRE(level >= 0 && level < levels, ICARAT_ERR_ARG, "level out of range");
  c->mg_galerkin_req = o->coarse_op == ICARAT_COARSE_GALERKIN ? 1 : 0;
  mg_setup(c, levels);
  MgLevel &L = c->mg[level];
  const size_t nv = 3 * (size_t)L.g.numnp;
  ICK(cudaMemcpyAsync(L.x, x, sizeof(double) * nv, cudaMemcpyHostToDevice, c->stream));
  // the coarsest level's constrained components are 0 between solves
  auto clear = [&] { ICK(cudaMemsetAsync(L.x, 0, sizeof(double) * nv, c->stream)); };
  if(level > 0 && c->mg_galerkin)
  {
    ICK(cudaMemsetAsync(L.b, 0, sizeof(double) * nv, c->stream));
    st_residual_launch<double>(c->stream, L.g, L.S, L.fix, L.b, L.x, L.t, nullptr);
    ICK(cudaMemcpyAsync(y, L.t, sizeof(double) * nv, cudaMemcpyDeviceToHost, c->stream));
    clear();
    ICK(cudaStreamSynchronize(c->stream));
    for(size_t i = 0; i < nv; i++)
      y[i] = -y[i];
    return;
  }
  launch_apply_K(c, L.g, L.E, L.fix, L.x, L.t, nullptr);
  ICK(cudaMemcpyAsync(y, L.t, sizeof(double) * nv, cudaMemcpyDeviceToHost, c->stream));
  clear();
  ICK(cudaStreamSynchronize(c->stream));
}

// Captures what f enqueues on stream st into an instantiated graph.
template <typename F>
static cudaGraphExec_t capture(cudaStream_t st, int &kernels, F f)
{
  cudaGraph_t graph;
  ICK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
  set_capturing(true);
  try
  {
    f();
  }
  catch(...)
  {
    set_capturing(false);
    cudaStreamEndCapture(st, &graph);
    throw;
  }
  set_capturing(false);
  ICK(cudaStreamEndCapture(st, &graph));
  size_t nn = 0;
  ICK(cudaGraphGetNodes(graph, nullptr, &nn));
  std::vector<cudaGraphNode_t> nodes(nn);
  ICK(cudaGraphGetNodes(graph, nodes.data(), &nn));
  kernels = 0;
  for(auto nd : nodes)
  {
    cudaGraphNodeType t;
    ICK(cudaGraphNodeGetType(nd, &t));
    kernels += (t == cudaGraphNodeTypeKernel) ? 1 : 0;
  }
  cudaGraphExec_t exec;
  ICK(cudaGraphInstantiate(&exec, graph, 0));
  cudaGraphDestroy(graph);
  return exec;
}

// Coarse operators and the dense inverse for the current design.  The fixed
// launch sequences are captured once per hierarchy into CUDA graphs and
// replayed for every new design.
//
// Lagged set-up (factor reuse across design iterations): the levels of the
// new design are built on the context's stream as usual, but its coarsest
// factor goes into the other buffer on a side stream, overlapped with the
// solve, which keeps the factor of the previous design; the next set-up
// waits for it and switches buffers.  The coarse correction then belongs to
// a slightly different operator, which costs at most a few iterations while
// the design changes slowly; the solve's stopping test is unchanged.
void mg_setup(icarat_ctx *c, int levels, bool lag)
{
  IREQUIRE(levels >= 2 && levels <= 12, ICARAT_ERR_ARG, "mg_levels must be in [2, 12]");
  if((int)c->mg.size() != levels || c->mg_galerkin != c->mg_galerkin_req)
    allocate_levels(c, levels);
  else if(c->mg_version == c->design_version)
  {
    // operators of this design are built; its lagged factor replaces the
    // previous design's once it has finished (a synchronous request waits
    // for it)
    CoarseSolver &C = c->coarse;
    if(C.pending >= 0 && (!lag || cudaEventQuery(C.ev_factor[C.pending]) == cudaSuccess))
    {
      ICK(cudaStreamWaitEvent(c->stream, C.ev_factor[C.pending], 0));
      C.cur = C.pending;
      C.pending = -1;
    }
    return;
  }
  c->mg_version = c->design_version;
  CoarseSolver &C = c->coarse;
  if(C.pending >= 0)
  {
    // the previous design's factor (lagged) is needed now, and its inputs
    // (the coarsest moduli) are about to be overwritten
    ICK(cudaStreamWaitEvent(c->stream, C.ev_factor[C.pending], 0));
    C.cur = C.pending;
    C.pending = -1;
  }
  if(!lag || !C.have || C.n == 0)
  {
    const int b = C.cur;
    if(!C.setup[b])
      C.setup[b] = capture(c->stream, C.setup_kernels, [&] {
        enqueue_levels(c, levels, c->stream);
        enqueue_factor(c, b, c->stream);
      });
    ICK(cudaGraphLaunch(C.setup[b], c->stream));
    note_launch(C.setup_kernels);
    C.have = true;
    return;
  }
  const int nb = 1 - C.cur;
  if(!C.P[nb])
    allocate_factor(C, nb);
  if(!C.side)
  {
    ICK(cudaStreamCreateWithFlags(&C.side, cudaStreamNonBlocking));
    ICK(cudaEventCreateWithFlags(&C.ev_levels, cudaEventDisableTiming));
    for(int b = 0; b < 2; b++)
      ICK(cudaEventCreateWithFlags(&C.ev_factor[b], cudaEventDisableTiming));
  }
  if(!C.levels)
    C.levels = capture(c->stream, C.levels_kernels, [&] { enqueue_levels(c, levels, c->stream); });
  if(!C.factor[nb])
    C.factor[nb] = capture(C.side, C.factor_kernels, [&] { enqueue_factor(c, nb, C.side); });
  ICK(cudaGraphLaunch(C.levels, c->stream));
  note_launch(C.levels_kernels);
  ICK(cudaEventRecord(C.ev_levels, c->stream));
  ICK(cudaStreamWaitEvent(C.side, C.ev_levels, 0));
  ICK(cudaGraphLaunch(C.factor[nb], C.side));
  note_launch(C.factor_kernels);
  ICK(cudaEventRecord(C.ev_factor[nb], C.side));
  C.pending = nb;
}

void mg_join(icarat_ctx *c)
{
  if(c->coarse.pending >= 0)
    ICK(cudaStreamWaitEvent(c->stream, c->coarse.ev_factor[c->coarse.pending], 0));
}

// the finest level of the FP32 V-cycle may run on the tensor-core operator
template <typename T> static bool tc_level(icarat_ctx *c, int lvl)
{
  return std::is_same<T, float>::value && lvl == 0 &&
         (c->mx_fine_op == ICARAT_OP_TC_BF16X3 || c->mx_fine_op == ICARAT_OP_TC_BF16);
}

// one Chebyshev step d = c1 d + c2 invd (b - K x), xo = x + d on level lvl;
// d_is_x: the d of the step before is x; last: no step follows that reads d.
// With dot set the step also takes the cycle's dot products where its kernel
// does (dot cleared then).
template <typename T>
static void cheb_step(icarat_ctx *c, MgLevel &L, int lvl, const T *b, const T *x, T *d, T *xo,
                      double c1, double c2, bool d_is_x, bool last, const CycleDot<T> **dot)
{
  using B = LevelBuf<T>;
  if(tc_level<T>(c, lvl))
  {
    if(d_is_x) // this operator reads d
      ICK(cudaMemcpyAsync(d, x, sizeof(T) * 3 * L.g.numnp, cudaMemcpyDeviceToDevice, c->stream));
    TcArgs a;
    a.g = L.g;
    a.E = reinterpret_cast<const float *>(B::E(L));
    a.fix = L.fix;
    a.u = reinterpret_cast<const float *>(x);
    a.y = reinterpret_cast<float *>(xo);
    a.b = reinterpret_cast<const float *>(b);
    a.invd = reinterpret_cast<const float *>(B::invd(L));
    a.d = reinterpret_cast<float *>(d);
    a.c1 = (float)c1;
    a.c2 = (float)c2;
    a.halt = c->mg_halt;
    launch_ku_tc(c, TC_CHEB, c->mx_fine_op == ICARAT_OP_TC_BF16X3 ? 3 : 1, a, c->stream);
    return;
  }
  if constexpr(std::is_same<T, double>::value)
    if(use_dmma(c, L.g))
    {
      if(d_is_x)
        ICK(cudaMemcpyAsync(d, x, sizeof(T) * 3 * L.g.numnp, cudaMemcpyDeviceToDevice,
                            c->stream));
      DmArgs a;
      a.g = L.g;
      a.E = B::E(L);
      a.fix = L.fix;
      a.u = x;
      a.y = xo;
      a.b = b;
      a.invd = B::invd(L);
      a.d = d;
      a.c1 = c1;
      a.c2 = c2;
      a.halt = c->mg_halt;
      launch_ku_dmma(c, TC_CHEB, a, c->stream);
      return;
    }
  int blocks;
  size_t smem;
  const T *din = c1 != 0.0 && !d_is_x ? d : nullptr;
  T *dout = last ? nullptr : d;
  note_launch();
  if(dot && *dot)
  {
    const ModalPlan m = modal_launch<T>(L.g, (const void *)k_cheb_step<T, true>, c->sm_count,
                                        kMaxRedBlocks, blocks, smem);
    launch_chained(k_cheb_step<T, true>, blocks, ModalCfg<T>::threads, smem, c->stream, L.g, m,
                   B::kh(c), B::E(L), L.fix, B::invd(L), b, x, din, dout, xo, T(c1), T(c2),
                   c->mg_halt, **dot);
    *dot = nullptr;
    return;
  }
  const ModalPlan m = modal_launch<T>(L.g, (const void *)k_cheb_step<T, false>, c->sm_count,
                                      1 << 30, blocks, smem);
  launch_chained(k_cheb_step<T, false>, blocks, ModalCfg<T>::threads, smem, c->stream, L.g, m,
                 B::kh(c), B::E(L), L.fix, B::invd(L), b, x, din, dout, xo, T(c1), T(c2),
                 c->mg_halt, CycleDot<T>{});
}

// r = b - K x on level lvl
template <typename T>
static void mg_residual(icarat_ctx *c, MgLevel &L, int lvl, const T *b, const T *x, T *r)
{
  using B = LevelBuf<T>;
  if(lvl > 0 && c->mg_galerkin)
  {
    st_residual_launch<T>(c->stream, L.g, B::S(L), L.fix, b, x, r, c->mg_halt);
    return;
  }
  if(tc_level<T>(c, lvl))
  {
    TcArgs a;
    a.g = L.g;
    a.E = reinterpret_cast<const float *>(B::E(L));
    a.fix = L.fix;
    a.u = reinterpret_cast<const float *>(x);
    a.y = reinterpret_cast<float *>(r);
    a.b = reinterpret_cast<const float *>(b);
    a.halt = c->mg_halt;
    launch_ku_tc(c, TC_RESID, c->mx_fine_op == ICARAT_OP_TC_BF16X3 ? 3 : 1, a, c->stream);
    return;
  }
  if constexpr(std::is_same<T, double>::value)
    if(use_dmma(c, L.g))
    {
      DmArgs a;
      a.g = L.g;
      a.E = B::E(L);
      a.fix = L.fix;
      a.u = x;
      a.y = r;
      a.b = b;
      a.halt = c->mg_halt;
      launch_ku_dmma(c, TC_RESID, a, c->stream);
      return;
    }
  int blocks;
  size_t smem;
  const ModalPlan m =
      modal_launch<T>(L.g, (const void *)k_mg_residual<T>, c->sm_count, 1 << 30, blocks, smem);
  note_launch();
  launch_chained(k_mg_residual<T>, blocks, ModalCfg<T>::threads, smem, c->stream, L.g, m, B::kh(c),
                 B::E(L), L.fix, b, x, r, c->mg_halt);
}

// Chebyshev smoothing of K x = b on level lvl, deg steps, from x (one of the
// level's buffers x and t) to the buffer returned.  from_zero: x = 0 on entry
// (the first step needs no product).
template <typename T>
static T *smooth(icarat_ctx *c, MgLevel &L, int lvl, const T *b, int deg, T *x, bool from_zero,
                 bool first_done, const CycleDot<T> **dot)
{
  using B = LevelBuf<T>;
  T *xo = x == B::x(L) ? B::t(L) : B::x(L), *d = B::r(L);
  const int nv = 3 * L.g.numnp;
  if(lvl > 0 && c->mg_galerkin)
  {
    // the same Chebyshev sequence with the level's own bound: coefficients
    // from the device (computed at set-up from the design's cell matrices)
    IREQUIRE(deg <= (kGalCoef + 1) / 2, ICARAT_ERR_ARG,
             "mg_smooth too large for the Galerkin coarse levels");
    const double *coef = c->gal_coef + (size_t)lvl * kGalCoef;
    if(from_zero)
      st_first_launch<T>(c->stream, nv, b, B::invd(L), coef, x, d, c->mg_halt);
    for(int k = from_zero ? 1 : 0; k < deg; k++)
    {
      st_cheb_launch<T>(c->stream, L.g, B::S(L), L.fix, B::invd(L), b, x, d, xo, coef, k,
                        c->mg_halt);
      std::swap(x, xo);
    }
    return x;
  }
  const double lmax = c->lam_max_dk;
  const double lmin = 0.1 * lmax;
  const double theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin);
  const double sigma = theta / delta;
  double rho_old = 1.0 / sigma;
  // the tensor-core operators read d from memory, the march takes x for it
  bool d_is_x = from_zero;
  if(from_zero)
  {
    if(!first_done) // else the kernel that produced b took this step
    {
      bool keep = tc_level<T>(c, lvl);
      if constexpr(std::is_same<T, double>::value)
        keep = keep || use_dmma(c, L.g);
      d_is_x = !keep;
      note_launch();
      launch_chained(k_cheb_first<T>, blocks_for(nv, 256), 256, 0, c->stream, nv, b,
                     B::invd(L), T(1.0 / theta), x, keep ? d : (T *)nullptr, c->mg_halt);
    }
  }
  else
  {
    // first step from the current x: d = invd (b - K x) / theta
    cheb_step<T>(c, L, lvl, b, x, d, xo, 0.0, 1.0 / theta, false, deg == 1,
                 deg == 1 ? dot : nullptr);
    std::swap(x, xo);
  }
  for(int k = 1; k < deg; k++)
  {
    const double rho = 1.0 / (2.0 * sigma - rho_old);
    cheb_step<T>(c, L, lvl, b, x, d, xo, rho * rho_old, 2.0 * rho / delta, d_is_x && k == 1,
                 k == deg - 1, k == deg - 1 ? dot : nullptr);
    std::swap(x, xo);
    rho_old = rho;
  }
  return x;
}

// One V-cycle from level l on; the result is in the level's x.  dot: the dot
// products of the finest level's last step (cleared where they were taken).
template <typename T>
static void vcycle(icarat_ctx *c, int l, const T *b, int deg, bool first_done,
                   const CycleDot<T> **dot)
{
  using B = LevelBuf<T>;
  MgLevel &L = c->mg[l];
  const int levels = (int)c->mg.size();
  if(l == levels - 1)
  {
    // the restriction has left the right-hand side in vin
    const int n = c->coarse.n;
    if(n > 0)
      coarse_solve<T>(c->stream, c->coarse.tree, c->coarse.W[c->coarse.cur],
                      c->coarse.U[c->coarse.cur], c->coarse.vin, c->coarse.vout, c->coarse.map,
                      B::x(L), c->mg_halt);
    return;
  }
  MgLevel &C = c->mg[l + 1];
  T *x = smooth<T>(c, L, l, b, deg, B::x(L), true, first_done, nullptr);
  // residual into r (smooth() used r as scratch; done with it now)
  mg_residual<T>(c, L, l, b, x, B::r(L));
  // the coarse level's first smoothing step rides on the restriction when
  // that level is smoothed with the shared rediscretised bound
  const bool coarsest = l + 1 == levels - 1;
  const bool fuse = !coarsest && !c->mg_galerkin;
  const double lm = c->lam_max_dk, theta = 0.5 * (lm + 0.1 * lm);
  note_launch();
  const bool split_c = C.g.numnp < kSplitNodes, split_f = L.g.numnp < kSplitNodes;
  launch_chained(split_c ? k_restrict<T, 1> : k_restrict<T, 3>,
                 transfer_grid(C.g, split_c ? 1 : 3), dim3(32, 4), 0, c->stream, L.g, C.g,
                 B::r(L), C.fix, B::b(C), B::invd(C), T(1.0 / theta),
                 fuse ? B::x(C) : (T *)nullptr, c->coarse.map + c->coarse.n,
                 coarsest ? c->coarse.vin : (double *)nullptr, c->mg_halt);
  vcycle<T>(c, l + 1, B::b(C), deg, fuse, nullptr);
  // into the buffer from which deg steps end in the level's x
  T *to = deg % 2 == 0 ? B::x(L) : B::t(L);
  note_launch();
  launch_chained(split_f ? k_prolong_add<T, 1> : k_prolong_add<T, 3>,
                 transfer_grid(L.g, split_f ? 1 : 3), dim3(32, 4), 0, c->stream, L.g, C.g,
                 B::x(C), L.fix, (const T *)x, to, c->mg_halt);
  smooth<T>(c, L, l, b, deg, to, false, false, l == 0 ? dot : nullptr);
}

bool mg_vcycle(icarat_ctx *c, const double *r, int deg, bool first_done,
               const CycleDot<double> *dot)
{
  vcycle<double>(c, 0, r, deg, first_done, &dot);
  ICK(cudaGetLastError());
  return dot == nullptr;
}

bool mg_vcycle_f32(icarat_ctx *c, const float *r, int deg, bool first_done,
                   const CycleDot<float> *dot)
{
  vcycle<float>(c, 0, r, deg, first_done, &dot);
  ICK(cudaGetLastError());
  return dot == nullptr;
}

} // namespace icarat_b200
