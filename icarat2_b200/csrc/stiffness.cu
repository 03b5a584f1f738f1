// Matrix-free FP64 stiffness operator on the voxel grid.
//
// Replaces LinearAnalysis::assemblingK and the sparse product inside the CG
// (src/analysis/linear.hpp:117-166, src/analysis/solver/CG.cpp:76-99).
// The products run in the parity blocks of the box element (modal.cuh): about 165
// FP64 operations per element, against 576 FMAs for Ke0's dense products;
// compulsory bytes per node: 24 read + 24 written (+ 8 per element modulus).
#include "modal.cuh"
#include "stencil.cuh"

namespace icarat_b200
{

// y = K u (constrained rows zeroed); optional per-block partial of u . y.
__global__ void __launch_bounds__(ModalCfg<double>::threads, ModalCfg<double>::blocks)
    k_apply_K_f64(GridDev g, ModalPlan m, KhParam<double> kh, const double *__restrict__ E,
                  const uint8_t *__restrict__ fix, const double *__restrict__ u,
                  double *__restrict__ y, double *__restrict__ partials)
{
  ModalShared<double> &ms = modal_shared<double>();
  __shared__ double sh[32];
  double dot = 0.0;
  modal_march(g, m, kh, E, u, ms,
              [&](int n) { return (unsigned)fix[n]; },
              [&](int n, const double(&acc)[3], const double(&uc)[3], unsigned f)
              {
#pragma unroll
                for(int q = 0; q < 3; q++)
                {
                  const double yq = ((f >> q) & 1u) ? 0.0 : acc[q];
                  y[(long)q * g.numnp + n] = yq;
                  dot += uc[q] * yq;
                }
              });
  if(partials)
  {
    double v[1] = {dot};
    block_sum<1>(v, sh);
    if(threadIdx.x == 0)
      partials[blockIdx.x] = v[0];
  }
}

// y = K u on equation vectors (free components only) in one launch: the march
// reads u through the nodes' first equation numbers and writes y the same
// way.  With the scatter into a node vector before and the gather after it was
// four launches (memset, scatter, product, gather) and twice the traffic.
__global__ void __launch_bounds__(ModalCfg<double>::threads, ModalCfg<double>::blocks)
    k_apply_K_eq(GridDev g, ModalPlan m, KhParam<double> kh, const double *__restrict__ E,
                 const uint8_t *__restrict__ fix, const int *__restrict__ base,
                 const double *__restrict__ u, double *__restrict__ y)
{
  ModalShared<double> &ms = modal_shared<double>();
  ModalEquations src;
  src.u = u;
  src.base = base;
  src.fix = fix;
  struct Pre
  {
    unsigned f;
    int at;
  };
  modal_march(g, m, kh, E, src, ms,
              [&](int n) { return Pre{fix[n], base[n]}; },
              [&](int, const double(&acc)[3], const double(&)[3], const Pre &pre)
              {
                double *out = y + pre.at;
#pragma unroll
                for(int q = 0; q < 3; q++)
                  if(!((pre.f >> q) & 1u))
                    *out++ = acc[q];
              });
}

bool apply_K_equations(icarat_ctx *c, const double *u, double *y)
{
  const GridDev g{c->nx, c->ny, c->nz, c->NX, c->NY, c->NZ, c->numnp, c->nelx};
  // blocks read u while others write y: they must not overlap
  if(c->numeq == 0 || use_dmma(c, g) || (u < y + c->numeq && y < u + c->numeq))
    return false;
  int blocks;
  size_t smem;
  const ModalPlan m = modal_launch<double>(g, (const void *)k_apply_K_eq, c->sm_count, 1 << 30,
                                           blocks, smem);
  note_launch();
  k_apply_K_eq<<<blocks, ModalCfg<double>::threads, smem, c->stream>>>(
      g, m, c->kh, c->d_E, c->d_fix, c->d_eqbase, u, y);
  ICK(cudaGetLastError());
  return true;
}

// 1 / diag(K): d_(n,c) = sum_{e ∋ n} E_e Ke0[3a+c][3a+c]; 0 on constrained.
__global__ void k_inv_diag(GridDev g, KeParam ke, const double *__restrict__ E,
                           const uint8_t *__restrict__ fix,
                           double *__restrict__ invd)
{
  for(int n = blockIdx.x * blockDim.x + threadIdx.x; n < g.numnp;
      n += gridDim.x * blockDim.x)
  {
    const int i = n % g.NX;
    const int j = (n / g.NX) % g.NY;
    const int k = n / (g.NX * g.NY);
    double d[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for(int sz = 0; sz < 2; sz++)
#pragma unroll
      for(int sy = 0; sy < 2; sy++)
#pragma unroll
        for(int sx = 0; sx < 2; sx++)
        {
          const double e = load_E(E, g, i - 1 + sx, j - 1 + sy, k - 1 + sz);
          const int a = local_node(1 - sx, 1 - sy, 1 - sz);
#pragma unroll
          for(int c = 0; c < 3; c++)
            d[c] = fma(e, ke.k[(3 * a + c) * 25], d[c]);
        }
    const unsigned f = fix[n];
#pragma unroll
    for(int c = 0; c < 3; c++)
      // a zero diagonal is treated as 1, as Eigen's DiagonalPreconditioner
      // does for the "Eigen_CG" solver (solvers.cpp:63-91)
      invd[(long)c * g.numnp + n] = ((f >> c) & 1u) ? 0.0 : (d[c] != 0.0 ? 1.0 / d[c] : 1.0);
  }
}

// K u_D restricted to free rows: fint of the first assembly, whose element
// displacements are the prescribed values (linear.hpp:63-77 followed by
// elasticity.cpp:244-254).
__global__ void __launch_bounds__(128)
    k_fint_f64(GridDev g, KeParam ke, const double *__restrict__ E,
               const uint8_t *__restrict__ fix, const double *__restrict__ uD,
               double *__restrict__ y)
{
  for(int n = blockIdx.x * blockDim.x + threadIdx.x; n < g.numnp;
      n += gridDim.x * blockDim.x)
  {
    double acc[3], uc[3];
    node_Ku(g, ke, E, uD, n, acc, uc);
    const unsigned f = fix[n];
#pragma unroll
    for(int c = 0; c < 3; c++)
      y[(long)c * g.numnp + n] = ((f >> c) & 1u) ? 0.0 : acc[c];
  }
}

__global__ void k_dot(int n, const double *__restrict__ a,
                      const double *__restrict__ b, double *__restrict__ partials,
                      unsigned int *counter, double *__restrict__ result)
{
  __shared__ double sh[32];
  double s = 0.0;
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
      i += gridDim.x * blockDim.x)
    s = fma(a[i], b[i], s);
  double v[1] = {s};
  block_sum<1>(v, sh);
  if(threadIdx.x == 0)
    partials[blockIdx.x] = v[0];
  if(last_block(counter))
  {
    double t[1];
    sum_partials<1>(partials, gridDim.x, t, sh);
    if(threadIdx.x == 0)
    {
      *result = t[0];
      *counter = 0;
    }
  }
}

static int node_blocks(const GridDev &g, int threads)
{
  int b = (g.numnp + threads - 1) / threads;
  return b < 1 ? 1 : b;
}

// Below kDmmaMinNodes the element tiles would leave most SMs idle.  The
// parity-block march is the faster FP64 operator at every grid size measured
// on a B200 (24.6 us against 62 us at 129 x 65 x 65 nodes, 128 us against 331 us
// at 257 x 129 x 129), so the default (fp64_tc 0) is the march and the FP64
// tensor cores run only when asked for.
constexpr int kDmmaMinNodes = 1 << 15;

bool use_dmma(const icarat_ctx *c, const GridDev &g)
{
  if(c->fp64_tc <= 0 || !dmma_fits(g))
    return false;
  return c->fp64_tc == 1 ? g.numnp >= kDmmaMinNodes : true;
}

void launch_apply_K(icarat_ctx *c, const GridDev &g, const double *E,
                    const uint8_t *fix, const double *u, double *y,
                    double *dot_partials)
{
  if(!dot_partials && use_dmma(c, g))
  {
    DmArgs a;
    a.g = g;
    a.E = E;
    a.fix = fix;
    a.u = u;
    a.y = y;
    launch_ku_dmma(c, TC_APPLY, a, c->stream);
    return;
  }
  int blocks;
  size_t smem;
  const ModalPlan m =
      modal_launch<double>(g, (const void *)k_apply_K_f64,
                           c->sm_count, kMaxRedBlocks, blocks, smem);
  note_launch();
  k_apply_K_f64<<<blocks, ModalCfg<double>::threads, smem, c->stream>>>(g, m, c->kh, E, fix, u, y,
                                                         dot_partials);
  ICK(cudaGetLastError());
}

// y = K u in FP32 (the FP32 copies of Ke0 and of the moduli)
__global__ void __launch_bounds__(ModalCfg<float>::threads, ModalCfg<float>::blocks)
    k_apply_K_f32(GridDev g, ModalPlan m, KhParam<float> kh, const float *__restrict__ E,
                  const uint8_t *__restrict__ fix, const float *__restrict__ u,
                  float *__restrict__ y)
{
  ModalShared<float> &ms = modal_shared<float>();
  modal_march(g, m, kh, E, u, ms,
              [&](int n) { return (unsigned)fix[n]; },
              [&](int n, const float(&acc)[3], const float(&)[3], unsigned f)
              {
#pragma unroll
                for(int c = 0; c < 3; c++)
                  y[(long)c * g.numnp + n] = ((f >> c) & 1u) ? 0.0f : acc[c];
              });
}

void launch_apply_K_f32(icarat_ctx *c, const GridDev &g, const float *E,
                        const uint8_t *fix, const float *u, float *y)
{
  int blocks;
  size_t smem;
  const ModalPlan m =
      modal_launch<float>(g, (const void *)k_apply_K_f32, c->sm_count, 1 << 30, blocks, smem);
  note_launch();
  k_apply_K_f32<<<blocks, ModalCfg<float>::threads, smem, c->stream>>>(g, m, c->khf, E, fix, u, y);
  ICK(cudaGetLastError());
}

void launch_diag(icarat_ctx *c, const GridDev &g, const double *E,
                 const uint8_t *fix, double *invd, cudaStream_t st)
{
  note_launch();
  k_inv_diag<<<node_blocks(g, 256), 256, 0, st ? st : c->stream>>>(g, c->ke0, E, fix, invd);
  ICK(cudaGetLastError());
}

void launch_fint(icarat_ctx *c, double *out)
{
  GridDev g{c->nx, c->ny, c->nz, c->NX, c->NY, c->NZ, c->numnp, c->nelx};
  note_launch();
  k_fint_f64<<<node_blocks(g, 128), 128, 0, c->stream>>>(g, c->ke0, c->d_E,
                                                         c->d_fix, c->d_uD, out);
  ICK(cudaGetLastError());
}

double device_dot(icarat_ctx *c, const double *a, const double *b, int n)
{
  note_launch();
  k_dot<<<c->red_blocks, kRedThreads, 0, c->stream>>>(
      n, a, b, c->d_partials, c->d_counter, c->d_scalar);
  ICK(cudaGetLastError());
  ICK(cudaMemcpyAsync(c->h_scalar, c->d_scalar, sizeof(double),
                      cudaMemcpyDeviceToHost, c->stream));
  ICK(cudaStreamSynchronize(c->stream));
  return c->h_scalar[0];
}

} // namespace icarat_b200
