// Radius density filter on the voxel grid (Filter<E,N>,
// src/optimization/filter.hpp).
//
// On a MeshIcarat box the neighbour list of preNeighbour (:254-297) is the
// same stencil for every element, clipped at the box faces: offsets (di, dj,
// dk) whose centroid distance d <= R, visited in ascending neighbour element
// id (dk, dj, di lexicographic), weight w = R - d.  The kernels accumulate in
// that order with separate multiply and add (no contraction), so forward and
// transposed results match the reference loop operation for operation.
#include <algorithm>
#include <atomic>
#include <cmath>

#include "filter_tile.cuh"
#include "internal.cuh"

namespace icarat_b200
{

// box elements; mask (null without a selection): 1 on the elements a
// selection keeps.  Removed elements are no neighbours and get 0.
struct ElemGrid
{
  int nx, ny, nz, nelx;
  const uint8_t *mask;
};

// dfilters_ds: a_i = sum over valid neighbours of w (geometry only)
__global__ void k_filter_aa(ElemGrid g, int nofs, const int *__restrict__ ofs,
                            const double *__restrict__ w, double *__restrict__ aa)
{
  for(int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.nelx;
      e += gridDim.x * blockDim.x)
  {
    if(g.mask && !g.mask[e])
    {
      aa[e] = 0.0;
      continue;
    }
    const int i = e % g.nx, j = (e / g.nx) % g.ny, k = e / (g.nx * g.ny);
    double a = 0.0;
    for(int q = 0; q < nofs; q++)
    {
      const int ii = i + ofs[3 * q], jj = j + ofs[3 * q + 1], kk = k + ofs[3 * q + 2];
      if(ii < 0 || ii >= g.nx || jj < 0 || jj >= g.ny || kk < 0 || kk >= g.nz)
        continue;
      if(g.mask && !g.mask[ii + (long)jj * g.nx + (long)kk * g.nx * g.ny])
        continue;
      a = __dadd_rn(a, w[q]);
    }
    aa[e] = a;
  }
}

// forward: out_i = sum w x_j / sum w   (filter.hpp:118-137)
__global__ void k_filter_fwd(ElemGrid g, int nofs, const int *__restrict__ ofs,
                             const double *__restrict__ w,
                             const double *__restrict__ in, double *__restrict__ out)
{
  for(int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.nelx;
      e += gridDim.x * blockDim.x)
  {
    if(g.mask && !g.mask[e])
    {
      out[e] = 0.0;
      continue;
    }
    const int i = e % g.nx, j = (e / g.nx) % g.ny, k = e / (g.nx * g.ny);
    double a = 0.0, b = 0.0;
    for(int q = 0; q < nofs; q++)
    {
      const int ii = i + ofs[3 * q], jj = j + ofs[3 * q + 1], kk = k + ofs[3 * q + 2];
      if(ii < 0 || ii >= g.nx || jj < 0 || jj >= g.ny || kk < 0 || kk >= g.nz)
        continue;
      const long f = ii + (long)jj * g.nx + (long)kk * g.nx * g.ny;
      if(g.mask && !g.mask[f])
        continue;
      const double wq = w[q];
      a = __dadd_rn(a, wq);
      b = __dadd_rn(b, __dmul_rn(wq, __ldg(in + f)));
    }
    out[e] = __ddiv_rn(b, a);
  }
}

// n / b rounded to nearest from y = RN(1 / b): q0 = RN(n y) is within one ulp
// of n / b, the remainder n - b q0 is exact in one FMA, and RN(q0 + r y) is
// the correctly rounded quotient (Markstein's theorem: P. Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34 (1990); Muller et al., Handbook of Floating-Point Arithmetic, on
// division with a fused multiply-add), for normal operands as here (sums of
// positive filter weights, finite terms).  Two FMAs and a product instead of
// a full division per term; the transposed filters stay bit-identical to the
// per-term division of the reference.
__device__ __forceinline__ double div_by_recip(double n, double b, double y)
{
  const double q0 = __dmul_rn(n, y);
  const double r = __fma_rn(-q0, b, n);
  return __fma_rn(r, y, q0);
}

// ra = RN(1 / aa) (IEEE division, once per filter set-up)
__global__ void k_filter_recip(int n, const double *__restrict__ aa, double *__restrict__ ra)
{
  for(int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    ra[e] = __ddiv_rn(1.0, aa[e]);
}

// transposed: out_i = sum_j w_ij in_j / a_j   (filter.hpp:145-152)
__global__ void k_filter_trans(ElemGrid g, int nofs, const int *__restrict__ ofs,
                               const double *__restrict__ w,
                               const double *__restrict__ aa,
                               const double *__restrict__ ra,
                               const double *__restrict__ in,
                               double *__restrict__ out)
{
  for(int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.nelx;
      e += gridDim.x * blockDim.x)
  {
    if(g.mask && !g.mask[e])
    {
      out[e] = 0.0;
      continue;
    }
    const int i = e % g.nx, j = (e / g.nx) % g.ny, k = e / (g.nx * g.ny);
    double s = 0.0;
    for(int q = 0; q < nofs; q++)
    {
      const int ii = i + ofs[3 * q], jj = j + ofs[3 * q + 1], kk = k + ofs[3 * q + 2];
      if(ii < 0 || ii >= g.nx || jj < 0 || jj >= g.ny || kk < 0 || kk >= g.nz)
        continue;
      const long f = ii + (long)jj * g.nx + (long)kk * g.nx * g.ny;
      if(g.mask && !g.mask[f])
        continue;
      s = __dadd_rn(s, div_by_recip(__dmul_rn(w[q], __ldg(in + f)), __ldg(aa + f), __ldg(ra + f)));
    }
    out[e] = s;
  }
}

// the transposed filter of two inputs in one pass (the loop's objective and
// volume sensitivities): neighbour offsets, weights and a_j read once, each
// output summed in the order and with the operations of k_filter_trans
__global__ void k_filter_trans2(ElemGrid g, int nofs, const int *__restrict__ ofs,
                                const double *__restrict__ w, const double *__restrict__ aa,
                                const double *__restrict__ ra,
                                const double *__restrict__ in1, const double *__restrict__ in2,
                                double *__restrict__ out1, double *__restrict__ out2)
{
  for(int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.nelx;
      e += gridDim.x * blockDim.x)
  {
    if(g.mask && !g.mask[e])
    {
      out1[e] = 0.0;
      out2[e] = 0.0;
      continue;
    }
    const int i = e % g.nx, j = (e / g.nx) % g.ny, k = e / (g.nx * g.ny);
    double s1 = 0.0, s2 = 0.0;
    for(int q = 0; q < nofs; q++)
    {
      const int ii = i + ofs[3 * q], jj = j + ofs[3 * q + 1], kk = k + ofs[3 * q + 2];
      if(ii < 0 || ii >= g.nx || jj < 0 || jj >= g.ny || kk < 0 || kk >= g.nz)
        continue;
      const long f = ii + (long)jj * g.nx + (long)kk * g.nx * g.ny;
      if(g.mask && !g.mask[f])
        continue;
      const double wq = w[q], af = __ldg(aa + f), rf = __ldg(ra + f);
      s1 = __dadd_rn(s1, div_by_recip(__dmul_rn(wq, __ldg(in1 + f)), af, rf));
      s2 = __dadd_rn(s2, div_by_recip(__dmul_rn(wq, __ldg(in2 + f)), af, rf));
    }
    out1[e] = s1;
    out2[e] = s2;
  }
}

// forward on a compiled ball: one staged array, a_i from the set-up (the same
// sum in the same order)
template <int D2>
__global__ void __launch_bounds__(kBallX *kBallY)
    k_ball_fwd(BallGrid g, const __grid_constant__ BallWeights<D2> W, const double *__restrict__ aa,
               const double *__restrict__ in, double *__restrict__ out)
{
  extern __shared__ double s_ball[];
  int x0, y0, z0;
  ball_origin(g, blockIdx.x, x0, y0, z0);
  ball_stage<D2>(g, x0, y0, z0, [&](int q, int e) { ball_copy(s_ball + q, in, e); });
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  double acc[kBallZ];
#pragma unroll
  for(int o = 0; o < kBallZ; o++)
    acc[o] = 0.0;
  ball_sum<D2>([&](int at) { return s_ball[at]; },
               [&](int o, int t, double v) { acc[o] = __dadd_rn(acc[o], __dmul_rn(W.w[t], v)); });
  const int x = x0 + threadIdx.x % kBallX, y = y0 + threadIdx.x / kBallX;
  if(x >= g.nx || y >= g.ny)
    return;
#pragma unroll
  for(int o = 0; o < kBallZ; o++)
    if(z0 + o < g.nz)
    {
      const int e = x + y * g.nx + (z0 + o) * g.nx * g.ny;
      out[e] = (g.mask && !g.mask[e]) ? 0.0 : __ddiv_rn(acc[o], aa[e]);
    }
}

// transposed on a compiled ball, NIN inputs at once; a_j and its reciprocal
// are staged beside the inputs
template <int D2, int NIN>
__global__ void __launch_bounds__(kBallX *kBallY)
    k_ball_trans(BallGrid g, const __grid_constant__ BallWeights<D2> W,
                 const double *__restrict__ aa, const double *__restrict__ ra, const double *__restrict__ in1,
                 const double *__restrict__ in2, double *__restrict__ out1,
                 double *__restrict__ out2)
{
  constexpr int tile = Ball<D2>::tile;
  extern __shared__ double s_ball[];
  double *s_a = s_ball, *s_r = s_ball + tile, *s_1 = s_ball + 2 * tile, *s_2 = s_ball + 3 * tile;
  int x0, y0, z0;
  ball_origin(g, blockIdx.x, x0, y0, z0);
  ball_stage<D2>(g, x0, y0, z0, [&](int q, int e) {
    ball_copy(s_a + q, aa, e);
    ball_copy(s_r + q, ra, e);
    ball_copy(s_1 + q, in1, e);
    if(NIN == 2)
      ball_copy(s_2 + q, in2, e);
  });
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  double acc[NIN][kBallZ];
#pragma unroll
  for(int o = 0; o < kBallZ; o++)
    for(int q = 0; q < NIN; q++)
      acc[q][o] = 0.0;
  struct Value
  {
    double a, r, v[NIN];
  };
  ball_sum<D2>(
      [&](int at) {
        Value v;
        v.a = s_a[at];
        v.r = s_r[at];
        v.v[0] = s_1[at];
        if(NIN == 2)
          v.v[NIN - 1] = s_2[at];
        return v;
      },
      [&](int o, int t, const Value &v) {
#pragma unroll
        for(int q = 0; q < NIN; q++)
          acc[q][o] = __dadd_rn(acc[q][o], div_by_recip(__dmul_rn(W.w[t], v.v[q]), v.a, v.r));
      });
  const int x = x0 + threadIdx.x % kBallX, y = y0 + threadIdx.x / kBallX;
  if(x >= g.nx || y >= g.ny)
    return;
#pragma unroll
  for(int o = 0; o < kBallZ; o++)
    if(z0 + o < g.nz)
    {
      const int e = x + y * g.nx + (z0 + o) * g.nx * g.ny;
      const bool keep = !(g.mask && !g.mask[e]);
      out1[e] = keep ? acc[0][o] : 0.0;
      if(NIN == 2)
        out2[e] = keep ? acc[NIN - 1][o] : 0.0;
    }
}

// sensitivityFilter (filter.hpp:77-104)
__global__ void k_sens_filter(ElemGrid g, int nofs, const int *__restrict__ ofs,
                              const double *__restrict__ w, double vol,
                              const double *__restrict__ s,
                              const double *__restrict__ df, double *__restrict__ out)
{
  for(int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.nelx;
      e += gridDim.x * blockDim.x)
  {
    if(g.mask && !g.mask[e])
    {
      out[e] = 0.0;
      continue;
    }
    const int i = e % g.nx, j = (e / g.nx) % g.ny, k = e / (g.nx * g.ny);
    double a = 0.0, b = 0.0;
    for(int q = 0; q < nofs; q++)
    {
      const int ii = i + ofs[3 * q], jj = j + ofs[3 * q + 1], kk = k + ofs[3 * q + 2];
      if(ii < 0 || ii >= g.nx || jj < 0 || jj >= g.ny || kk < 0 || kk >= g.nz)
        continue;
      const long f = ii + (long)jj * g.nx + (long)kk * g.nx * g.ny;
      if(g.mask && !g.mask[f])
        continue;
      const double wq = w[q], sf = s[f];
      a = __dadd_rn(a, wq);
      b = __dadd_rn(b, __ddiv_rn(__dmul_rn(__dmul_rn(wq, sf), df[f]),
                                 __dmul_rn(sf, vol)));
    }
    const double cc = __ddiv_rn(__dmul_rn(s[e], vol), __dmul_rn(s[e], a));
    out[e] = __dmul_rn(cc, b);
  }
}

// threshold / thresholdDerivative (filter.hpp:217-249)
__global__ void k_threshold(int n, const double *__restrict__ in, double beta,
                            double T, double *__restrict__ out, int derivative)
{
  const double tb = tanh(T * beta);
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
      i += gridDim.x * blockDim.x)
  {
    const double t = tanh(beta * (in[i] - T));
    out[i] = derivative ? (0.5 * (beta * (1.0 - t * t))) / tb
                        : 0.5 * (tb + t) / tb;
  }
}

static ElemGrid egrid(const icarat_ctx *c)
{
  return ElemGrid{c->nx, c->ny, c->nz, c->nelx, c->d_emask};
}

static BallGrid bgrid(const icarat_ctx *c)
{
  return BallGrid{c->nx, c->ny, c->nz, c->nelx, c->d_emask};
}

// dynamic shared memory of Arrays staged arrays of ball D2, the kernel's limit
// raised (once per device) where that passes 48 KB
template <int D2, int Arrays> static size_t ball_smem(const void *kernel)
{
  static std::atomic<bool> ready[kMaxDevices];
  const size_t n = sizeof(double) * (size_t)Arrays * Ball<D2>::tile;
  if(n > 48 * 1024)
  {
    const int d = device_slot();
    if(!ready[d].load())
    {
      ICK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n));
      ready[d].store(true);
    }
  }
  return n;
}

static int eblocks(const icarat_ctx *c)
{
  int b = (c->nelx + 255) / 256;
  return b < 1 ? 1 : b;
}

void filter_free(icarat_ctx *c)
{
  dfree(c->filt.d_ofs);
  dfree(c->filt.d_w);
  dfree(c->filt.d_aa);
  dfree(c->filt.d_ra);
  c->filt = FilterState{};
}

// The compiled ball whose taps are exactly the list's, with its octant of
// weights in cube, or 0 (larger radii, stretched voxels).
static int find_ball(const FilterState &F, std::vector<double> &cube)
{
  int found = 0;
  for(int d2 : {1, 2, 3, 4, 5, 6, 8, 9})
    ball_dispatch(d2, [&](auto D) {
      using B = Ball<decltype(D)::value>;
      int n = 0;
      bool same = true;
      std::vector<double> w(B::weights, -1.0);
      for(int dk = -B::r; dk <= B::r; dk++)
        for(int dj = -B::r; dj <= B::r; dj++)
          for(int di = -B::r; di <= B::r; di++)
            if(B::in(dk, dj, di))
            {
              same = same && n < F.nofs && F.ofs[3 * n] == di && F.ofs[3 * n + 1] == dj &&
                     F.ofs[3 * n + 2] == dk;
              if(same)
              {
                double &v = w[B::index(dk, dj, di)];
                same = v == -1.0 || v == F.w[n]; // weights are >= 0
                v = F.w[n];
              }
              n++;
            }
      if(same && n == F.nofs)
      {
        found = D();
        cube = w;
      }
    });
  return found;
}

void filter_setup(icarat_ctx *c, double R)
{
  IREQUIRE(R >= 0.0 && std::isfinite(R), ICARAT_ERR_ARG, "filter radius must be >= 0");
  FilterState &F = c->filt;
  if(F.ready && F.radius == R)
  {
    // the same stencil on the same mesh (a loop started again): it stands
    F.have_forward = false;
    return;
  }
  filter_free(c);
  F.radius = R;
  F.rx = (int)std::ceil(R / c->hx);
  F.ry = (int)std::ceil(R / c->hy);
  F.rz = (int)std::ceil(R / c->hz);
  for(int dk = -F.rz; dk <= F.rz; dk++)
    for(int dj = -F.ry; dj <= F.ry; dj++)
      for(int di = -F.rx; di <= F.rx; di++)
      {
        const double x = di * c->hx, y = dj * c->hy, z = dk * c->hz;
        const double d = std::sqrt(x * x + y * y + z * z);
        if(d <= R)
        {
          F.ofs.push_back(di);
          F.ofs.push_back(dj);
          F.ofs.push_back(dk);
          F.w.push_back(R - d);
        }
      }
  F.nofs = (int)F.w.size();
  F.ball = find_ball(F, F.cube);
  ICK(cudaMalloc(&F.d_ofs, sizeof(int) * F.ofs.size()));
  ICK(cudaMemcpy(F.d_ofs, F.ofs.data(), sizeof(int) * F.ofs.size(),
                 cudaMemcpyHostToDevice));
  F.d_w = dalloc(F.w.size());
  ICK(cudaMemcpy(F.d_w, F.w.data(), sizeof(double) * F.w.size(),
                 cudaMemcpyHostToDevice));
  F.d_aa = dalloc(c->nelx);
  note_launch();
  k_filter_aa<<<eblocks(c), 256, 0, c->stream>>>(egrid(c), F.nofs, F.d_ofs, F.d_w,
                                                 F.d_aa);
  F.d_ra = dalloc(c->nelx);
  note_launch();
  k_filter_recip<<<eblocks(c), 256, 0, c->stream>>>(c->nelx, F.d_aa, F.d_ra);
  ICK(cudaGetLastError());
  F.have_forward = false;
  F.ready = true;
}

template <int D2> static BallWeights<D2> ball_weights(const FilterState &F)
{
  BallWeights<D2> W;
  std::copy(F.cube.begin(), F.cube.end(), W.w);
  return W;
}

// The compiled ball is the faster form from about 1e5 taps in all: below, the
// launch is all the time there is and the tile's halo only adds to it (7 taps
// on 7 k elements: 5.8 us by the list, 6.6 staged; 19 taps: 8.3 and 6.0).
static bool use_ball(const icarat_ctx *c, BallUse use)
{
  return c->filt.ball > 0 && (double)c->filt.nofs * c->nelx >= 1.0e5 &&
         ball_pays(c->filt.ball, use, c->nx, c->ny, c->nz);
}

template <int NIN>
static void launch_ball_trans(icarat_ctx *c, const double *in1, const double *in2, double *out1,
                              double *out2)
{
  const FilterState &F = c->filt;
  ball_dispatch(F.ball, [&](auto D) {
    constexpr int d2 = decltype(D)::value;
    const auto kernel = k_ball_trans<d2, NIN>;
    kernel<<<(unsigned)ball_blocks(c->nx, c->ny, c->nz), kBallX * kBallY,
             ball_smem<d2, 2 + NIN>((const void *)kernel), c->stream>>>(
        bgrid(c), ball_weights<d2>(F), F.d_aa, F.d_ra, in1, in2, out1, out2);
  });
}

// The forward pass fails like the reference when a weight sum is below 1e-10
// (filter.hpp:130-134); that can only happen for R < 1e-10.
void filter_apply(icarat_ctx *c, const double *in, double *out, bool is_sens)
{
  FilterState &F = c->filt;
  IREQUIRE(F.d_w != nullptr, ICARAT_ERR_STATE, "filter not set up");
  if(!is_sens)
  {
    IREQUIRE(F.radius >= 1.0e-10, ICARAT_ERR_FILTER,
             "coefficient aa is too small in the density filter");
    note_launch();
    if(use_ball(c, kBallForward))
      ball_dispatch(F.ball, [&](auto D) {
        constexpr int d2 = decltype(D)::value;
        k_ball_fwd<d2><<<(unsigned)ball_blocks(c->nx, c->ny, c->nz), kBallX * kBallY,
                         ball_smem<d2, 1>((const void *)k_ball_fwd<d2>), c->stream>>>(
            bgrid(c), ball_weights<d2>(F), F.d_aa, in, out);
      });
    else
      k_filter_fwd<<<eblocks(c), 256, 0, c->stream>>>(egrid(c), F.nofs, F.d_ofs, F.d_w, in, out);
    F.have_forward = true;
  }
  else
  {
    IREQUIRE(F.have_forward, ICARAT_ERR_STATE,
             "transposed filter needs a forward call first (filter.hpp:140-153)");
    note_launch();
    if(use_ball(c, kBallTransposed))
      launch_ball_trans<1>(c, in, nullptr, out, nullptr);
    else
      k_filter_trans<<<eblocks(c), 256, 0, c->stream>>>(egrid(c), F.nofs, F.d_ofs, F.d_w, F.d_aa,
                                                        F.d_ra, in, out);
  }
  ICK(cudaGetLastError());
}

// transposed filter of in1 and in2 (a forward call must have come first)
void filter_trans2(icarat_ctx *c, const double *in1, const double *in2, double *out1,
                   double *out2)
{
  FilterState &F = c->filt;
  IREQUIRE(F.d_w != nullptr, ICARAT_ERR_STATE, "filter not set up");
  IREQUIRE(F.have_forward, ICARAT_ERR_STATE,
           "transposed filter needs a forward call first (filter.hpp:140-153)");
  note_launch();
  if(use_ball(c, kBallTransposed))
    launch_ball_trans<2>(c, in1, in2, out1, out2);
  else
    k_filter_trans2<<<eblocks(c), 256, 0, c->stream>>>(egrid(c), F.nofs, F.d_ofs, F.d_w, F.d_aa,
                                                       F.d_ra, in1, in2, out1, out2);
  ICK(cudaGetLastError());
}

void sensitivity_filter_dev(icarat_ctx *c, const double *s, const double *df,
                            double *out)
{
  FilterState &F = c->filt;
  IREQUIRE(F.d_w != nullptr, ICARAT_ERR_STATE, "filter not set up");
  note_launch();
  k_sens_filter<<<eblocks(c), 256, 0, c->stream>>>(egrid(c), F.nofs, F.d_ofs, F.d_w,
                                                   c->vol0, s, df, out);
  ICK(cudaGetLastError());
}

void threshold_dev(icarat_ctx *c, const double *in, double beta, double T,
                   double *out, bool derivative)
{
  note_launch();
  k_threshold<<<eblocks(c), 256, 0, c->stream>>>(c->nelx, in, beta, T, out,
                                                 derivative ? 1 : 0);
  ICK(cudaGetLastError());
}

} // namespace icarat_b200
