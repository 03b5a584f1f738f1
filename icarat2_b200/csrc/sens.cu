// Post-solve element quantities: nodal values, compliance and the compliance
// sensitivity of the sample drivers.
#include <cmath>

#include "stencil.cuh"

namespace icarat_b200
{

// divideValIntoNode (src/analysis/analysis_utility.hpp:9-31): free values from
// the solution, prescribed values on constrained components, |v| < 1e-15 -> 0.
__device__ __forceinline__ double node_value(const double *__restrict__ u,
                                             const double *__restrict__ uD,
                                             unsigned fix, long id, int q)
{
  double v = ((fix >> q) & 1u) ? (uD ? uD[id] : 0.0) : u[id];
  return fabs(v) < 1.0e-15 ? 0.0 : v;
}

__global__ void k_node_values(int numnp, const double *__restrict__ u,
                              const double *__restrict__ uD,
                              const uint8_t *__restrict__ fix,
                              double *__restrict__ out)
{
  for(int n = blockIdx.x * blockDim.x + threadIdx.x; n < numnp;
      n += gridDim.x * blockDim.x)
  {
    const unsigned f = fix[n];
#pragma unroll
    for(int q = 0; q < 3; q++)
      out[3L * n + q] = node_value(u, uD, f, (long)q * numnp + n, q);
  }
}

// Driver sensitivity() (sample/algorithm/opt-macro-oc/opt_macro_oc.cpp:182-212):
//   young  = (1 - rho^p) E1 + rho^p E2,  dyoung = p rho^(p-1) (E2 - E1)
//   dfds_e = -(dyoung / young) u_e^T (young Ke0) u_e,   dgds_e = volume * scale
// with u_e the truncated nodal values.
//
// The quadratic form is taken in the corner sums and differences of the box
// element, where Ke0 falls apart into blocks of at most three (KhParam): 33
// coefficients and about 130 operations for it instead of 600, bound by the
// loads after that.  The powers of a whole exponent up to 3 are products (1 ulp;
// pow 2 ulp).  256 x 128 x 128 elements: 705 -> 180 us.
__device__ __forceinline__ double simp_power(double x, double p)
{
  if(p == 3.0)
    return x * x * x;
  if(p == 2.0)
    return x * x;
  return p == 1.0 ? x : pow(x, p);
}

__global__ void __launch_bounds__(128)
    k_sensitivity(GridDev g, KhParam<double> kh, const double *__restrict__ rho,
                  const double *__restrict__ u, const double *__restrict__ uD,
                  const uint8_t *__restrict__ fix, double e1, double e2, double p,
                  double vol, double scale, double *__restrict__ dfds,
                  double *__restrict__ dgds)
{
  auto pair = [](const double(&m)[3], double x, double y)
  { return fma(x, fma(m[1], y, m[0] * x), y * fma(m[2], y, m[1] * x)); };
  auto full = [](const double(&m)[6], double x, double y, double z)
  {
    return fma(x, fma(m[2], z, fma(m[1], y, m[0] * x)),
               fma(y, fma(m[4], z, fma(m[3], y, m[1] * x)),
                   z * fma(m[5], z, fma(m[4], y, m[2] * x))));
  };
  for(int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.nelx;
      e += gridDim.x * blockDim.x)
  {
    const int i = e % g.nx, j = (e / g.nx) % g.ny, k = e / (g.nx * g.ny);
    // sums s and differences d along z of the faces' sums and differences
    // (bit 0 of the index the x difference, bit 1 the y difference)
    double s[3][4], d[3][4];
    double v[2][2][2][3];
#pragma unroll
    for(int bz = 0; bz < 2; bz++)
#pragma unroll
      for(int by = 0; by < 2; by++)
#pragma unroll
        for(int bx = 0; bx < 2; bx++)
        {
          const long m = (i + bx) + (long)(j + by) * g.NX + (long)(k + bz) * g.NX * g.NY;
          const unsigned f = fix[m];
#pragma unroll
          for(int q = 0; q < 3; q++)
            v[bz][by][bx][q] = node_value(u, uD, f, (long)q * g.numnp + m, q);
        }
#pragma unroll
    for(int q = 0; q < 3; q++)
    {
      double f[2][4];
#pragma unroll
      for(int bz = 0; bz < 2; bz++)
      {
        const double s0 = v[bz][0][0][q] + v[bz][0][1][q], d0 = v[bz][0][1][q] - v[bz][0][0][q];
        const double s1 = v[bz][1][0][q] + v[bz][1][1][q], d1 = v[bz][1][1][q] - v[bz][1][0][q];
        f[bz][0] = s0 + s1;
        f[bz][1] = d0 + d1;
        f[bz][2] = s1 - s0;
        f[bz][3] = d1 - d0;
      }
#pragma unroll
      for(int h = 0; h < 4; h++)
      {
        s[q][h] = f[0][h] + f[1][h];
        d[q][h] = f[1][h] - f[0][h];
      }
    }
    double q = full(kh.c0, s[0][1], s[1][2], d[2][0]) + pair(kh.c4, d[0][1], d[1][2]);
    q += pair(kh.c1, s[1][3], d[2][1]) + pair(kh.c5, d[0][0], s[2][1]) +
         kh.s5 * d[1][3] * d[1][3];
    q += pair(kh.c2, s[0][3], d[2][2]) + pair(kh.c6, d[1][0], s[2][2]) +
         kh.s6 * d[0][3] * d[0][3];
    q += pair(kh.c3, s[0][2], s[1][1]) + full(kh.c7, d[0][2], d[1][1], s[2][3]) +
         kh.s3 * d[2][3] * d[2][3];
    const double dens = rho[e];
    const double rp = simp_power(dens, p);
    const double young = (1.0 - rp) * e1 + rp * e2;
    const double dyoung = p * simp_power(dens, p - 1.0) * (e2 - e1);
    if(dfds)
      dfds[e] = -(dyoung / young) * (young * q);
    if(dgds)
      dgds[e] = vol * scale;
  }
}

// von Mises stress of the last solve per element (Elastic::makeMisesStress,
// src/problem/elasticity.cpp:166-207): sigma = E(rho) S u_e with the
// Gauss-averaged stress operator S and the truncated nodal values,
// mises = sqrt(sigma^T V sigma), V = [1 -1/2 -1/2; ..] (+) 3 I on the shears
__global__ void __launch_bounds__(128)
    k_mises(GridDev g, StressParam sp, const double *__restrict__ rho,
            const double *__restrict__ u, const double *__restrict__ uD,
            const uint8_t *__restrict__ fix, double e1, double e2, double p,
            double *__restrict__ out)
{
  for(int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.nelx;
      e += gridDim.x * blockDim.x)
  {
    const int i = e % g.nx, j = (e / g.nx) % g.ny, k = e / (g.nx * g.ny);
    double ue[24];
#pragma unroll
    for(int bz = 0; bz < 2; bz++)
#pragma unroll
      for(int by = 0; by < 2; by++)
#pragma unroll
        for(int bx = 0; bx < 2; bx++)
        {
          const int b = local_node(bx, by, bz);
          const long m = (i + bx) + (long)(j + by) * g.NX + (long)(k + bz) * g.NX * g.NY;
          const unsigned f = fix[m];
#pragma unroll
          for(int q = 0; q < 3; q++)
            ue[3 * b + q] = node_value(u, uD, f, (long)q * g.numnp + m, q);
        }
    const double dens = rho[e];
    const double young = (1.0 - pow(dens, p)) * e1 + pow(dens, p) * e2;
    double sg[6];
#pragma unroll
    for(int r = 0; r < 6; r++)
    {
      double t = 0.0;
#pragma unroll
      for(int c = 0; c < 24; c++)
        t = fma(sp.s[24 * r + c], ue[c], t);
      sg[r] = young * t;
    }
    const double q = sg[0] * (sg[0] - 0.5 * sg[1] - 0.5 * sg[2]) +
                     sg[1] * (sg[1] - 0.5 * sg[0] - 0.5 * sg[2]) +
                     sg[2] * (sg[2] - 0.5 * sg[0] - 0.5 * sg[1]) +
                     3.0 * (sg[3] * sg[3] + sg[4] * sg[4] + sg[5] * sg[5]);
    out[e] = sqrt(fmax(q, 0.0)); // V is positive semidefinite: q < 0 is rounding
  }
}

void mises_dev(icarat_ctx *c, double *out)
{
  IREQUIRE(c->solved, ICARAT_ERR_STATE, "Mises stress needs a solve first");
  GridDev g{c->nx, c->ny, c->nz, c->NX, c->NY, c->NZ, c->numnp, c->nelx};
  note_launch();
  k_mises<<<(c->nelx + 127) / 128, 128, 0, c->stream>>>(g, c->sb0, c->d_rho, c->d_u, c->d_uD,
                                                        c->d_fix, c->mat.young_min,
                                                        c->mat.young_max, c->mat.penalty, out);
  ICK(cudaGetLastError());
}

void node_values_dev(icarat_ctx *c, double *out)
{
  note_launch();
  k_node_values<<<(c->numnp + 255) / 256, 256, 0, c->stream>>>(c->numnp, c->d_u,
                                                               c->d_uD, c->d_fix, out);
  ICK(cudaGetLastError());
}

double compliance_dev(icarat_ctx *c)
{
  return device_dot(c, c->d_u, c->d_fext, c->neq);
}

void sensitivity_dev(icarat_ctx *c, double scale, double *dfds, double *dgds)
{
  IREQUIRE(c->solved, ICARAT_ERR_STATE, "sensitivity needs a solve first");
  GridDev g{c->nx, c->ny, c->nz, c->NX, c->NY, c->NZ, c->numnp, c->nelx};
  note_launch();
  k_sensitivity<<<(c->nelx + 127) / 128, 128, 0, c->stream>>>(
      g, c->kh, c->d_rho, c->d_u, c->d_uD, c->d_fix, c->mat.young_min,
      c->mat.young_max, c->mat.penalty, c->vol0, scale, dfds, dgds);
  ICK(cudaGetLastError());
}

} // namespace icarat_b200
