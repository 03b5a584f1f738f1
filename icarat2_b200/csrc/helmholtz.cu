// Helmholtz PDE density filter (FilterHelmholtz<E,N>,
// src/optimization/filter_helm.hpp) on the voxel grid.
//
// The reference assembles, per element and Gauss point (makeKeFint,
// :179-223), Ke += (N N^T + B^T (R / (2 sqrt 3))^2 I B) jac and
// fe += s N jac (fe /= ipmax for the sensitivity call), solves the nodal
// scalar system K val = F with "Eigen_CG" (a Jacobi-preconditioned CG,
// solvers.cpp:63-91, tolerance 1e-10 and 10000 iterations by default,
// solvers.hpp:89-90) and maps back per element (divideToElement, :225-257):
// out = sum_gp N . val_e, divided by ipmax for the density call.
//
// On the uniform voxel box every element has the same 8 x 8 matrix, so the
// assembled K is a 27-point node stencil whose coefficients depend only on
// which of the node's 8 neighbouring elements exist: 3 x 3 x 3 node classes
// (lower face, interior, upper face per axis).  The table of 27 classes x 27
// neighbour slots is assembled once on the host in the reference's order
// (ascending element id) for the Jacobi diagonal; the solve runs
// matrix-free with the same operator in sum-factorised form (k_helm_step).
// The CG iteration
// keeps the device-resident scalar logic of the elasticity solve (one
// stop-flag read per graph replay of `kHelmChunk` iterations).
#include <cmath>

#include "internal.cuh"

namespace icarat_b200
{

namespace
{

constexpr int kHelmChunk = 16;
constexpr int kHelmThreads = 256;
constexpr int kHelmClasses = 27;

struct HelmGrid
{
  int nx, ny, nz, NX, NY, numnp, nelx;
};

// integrals of the shape functions over the element: sum_gp N_a jac (the
// right-hand side weights) and sum_gp N_a (the readout weights); corners in
// bit order a = ax + 2 ay + 4 az
struct HelmWeights
{
  double nj[8], ns[8];
};

HelmGrid hgrid(const icarat_ctx *c)
{
  return HelmGrid{c->nx, c->ny, c->nz, c->NX, c->NY, c->numnp, c->nelx};
}

__device__ __forceinline__ int node_class(int i, int n)
{
  return i == 0 ? 0 : (i == n - 1 ? 2 : 1);
}

// Jacobi inverse diagonal per node class (27 values, 1 / centre coefficient
// of the class row)
struct HelmInvd
{
  double v[kHelmClasses];
};

__device__ __forceinline__ int helm_class(const HelmGrid &g, int n)
{
  const int i = n % g.NX, rest = n / g.NX, j = rest % g.NY, k = rest / g.NY;
  return node_class(i, g.NX) + 3 * node_class(j, g.NY) + 9 * node_class(k, g.nz + 1);
}

// The CG's start: r = F = sum over the node's elements of s_e nj[a] (/8 for the
// sensitivity call), elements in ascending id like the reference's assembly,
// x = 0, z.r with z = D^-1 r, ||F|| and the loop's scalars (as k_cg_init of
// pcg.cu sets them; beta = 0 makes the first direction z).
__global__ void k_helm_start(HelmGrid g, HelmWeights w, HelmInvd iv, const double *__restrict__ in,
                             double *__restrict__ x, double *__restrict__ r, int sens,
                             double *__restrict__ partials, CgScalars *s, double tol, int maxit)
{
  __shared__ double sh[64];
  double zr = 0.0, bb = 0.0;
  for(int n = blockIdx.x * blockDim.x + threadIdx.x; n < g.numnp;
      n += gridDim.x * blockDim.x)
  {
    const int i = n % g.NX, rest = n / g.NX, j = rest % g.NY, k = rest / g.NY;
    // all eight loads first (an element outside is read as the node's own and
    // left out)
    const int e0 = min(i, g.nx - 1) + min(j, g.ny - 1) * g.nx + min(k, g.nz - 1) * g.nx * g.ny;
    double se[8];
    bool have[8];
#pragma unroll
    for(int q = 0; q < 8; q++) // ascending element id
    {
      const int ei = i - 1 + (q & 1), ej = j - 1 + ((q >> 1) & 1), ek = k - 1 + (q >> 2);
      have[q] = ei >= 0 && ei < g.nx && ej >= 0 && ej < g.ny && ek >= 0 && ek < g.nz;
      se[q] = __ldg(in + (have[q] ? ei + ej * g.nx + ek * g.nx * g.ny : e0));
    }
    double f = 0.0;
#pragma unroll
    for(int q = 0; q < 8; q++)
    {
      double fe = __dmul_rn(se[q], w.nj[7 - q]);
      if(sens)
        fe = __dmul_rn(fe, 0.125); // = fe / 8 in every case
      f = have[q] ? __dadd_rn(f, fe) : f;
    }
    x[n] = 0.0;
    r[n] = f;
    const double z = f * iv.v[helm_class(g, n)];
    zr += z * f;
    bb += f * f;
  }
  double v[2] = {zr, bb};
  block_sum<2>(v, sh);
  if(threadIdx.x == 0)
  {
    partials[blockIdx.x] = v[0];
    partials[gridDim.x + blockIdx.x] = v[1];
  }
  if(last_block(&s->counter))
  {
    double t[2];
    sum_partials<2>(partials, gridDim.x, t, sh);
    if(threadIdx.x == 0)
    {
      s->zr = t[0];
      s->beta = 0.0;
      s->bnorm = sqrt(t[1]);
      s->rnorm = s->bnorm;
      s->tol = tol;
      s->maxit = maxit;
      s->iter = 0;
      s->status = ICARAT_OK;
      s->done = (t[1] == 0.0) ? 1 : 0;
      if(!(t[1] == t[1]))
      {
        s->done = 1;
        s->status = ICARAT_ERR_NAN;
      }
      s->counter = 0;
    }
  }
}

// p = z + beta p (z = D^-1 r), Ap = K p and alpha = zr / (p . Ap), by sum
// factorisation.
//
// With trilinear shape functions and exact 2-point Gauss rules the element
// matrix is a tensor product, Ke = Mx (x) My (x) Mz + c (Sx (x) My (x) Mz +
// Mx (x) Sy (x) Mz + Mx (x) My (x) Sz), c = (R / (2 sqrt 3))^2, with the 1-D
// element mass h/6 [2 1; 1 2] and stiffness 1/h [1 -1; -1 1]; assembled on
// the box it stays one, with the 3-point 1-D stencils m, s of each node
// class (lower face, inside, upper face).  So every plane of p contributes
// through two in-plane sums per node, A = (mx my + c (sx my + mx sy)) p and
// B = mx my p, and Ap(k) = sum_dz mz A(k+dz) + c sz B(k+dz).
//
// A block of 8 warps owns 32 x 16 node columns and marches through kz planes,
// holding A and B of planes k-1, k, k+1 in registers.  r and the old p come
// through rings of halo tiles filled by cp.async kHelmAhead planes ahead; one
// plane ahead of the sums the block forms the new p in a tile of its own (and
// its owner stores it, into the other of two vectors: neighbours still read
// the old one), so a plane costs one barrier and p costs no pass of its own.
// Positions outside the box are stored as 0 (their stencil weights are 0 as
// well).  Bound by memory (32 bytes per node) and the barrier per plane.
// Measured on a B200 at 257 x 129 x 129 nodes: the product alone took 50 us and
// the update of p another 24; this kernel takes 49.
// Two rows per thread at two blocks per SM: one row 56 us, three blocks (80
// registers) 48 there but slower on smaller grids, and a variant that spills
// 80 bytes 95.  Grids of up to 8 nodes along y take the one row: they fill half
// of its tile's rows at most (601 x 2 x 601 nodes: 529 us a call before this
// kernel, 622 with two rows, 497 with one).
constexpr int kHelmTx = 32, kHelmRing = 4, kHelmAhead = 2, kHelmBlocks = 2;
constexpr int kHaloX = kHelmTx + 2;
template <int Rows> struct HelmTile
{
  static constexpr int ty = Rows * kHelmThreads / 32;
  static constexpr int halo = kHaloX * (ty + 2);
  static constexpr int stage = (halo + kHelmThreads - 1) / kHelmThreads; // cells per thread
};
inline int helm_rows(int NY) { return NY <= HelmTile<1>::ty ? 1 : 2; }

// 1-D stencils per axis: neighbour weights mo, so (a neighbour outside the box
// is staged as 0, so they hold for every node) and centre weights md, sd of a
// face node (twice that inside); the diffusion coefficient c
struct HelmAxes
{
  double mo[3], so[3], md[3], sd[3];
  double c;
};

// tiles of kHelmTx x HelmTile::ty columns and chunks of kz planes
struct HelmPlan
{
  int tiles_x, tiles_y, kz, items;
};

template <int Rows> struct HelmShared
{
  double r[kHelmRing][HelmTile<Rows>::halo], p[kHelmRing][HelmTile<Rows>::halo],
      q[2][HelmTile<Rows>::halo];
};

// 8-byte global -> shared copy, 0 where !valid
__device__ __forceinline__ void cp_async8(double *dst, const double *src, bool valid)
{
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = valid ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n)
               : "memory");
}

template <int Rows>
__global__ void __launch_bounds__(kHelmThreads, kHelmBlocks)
    k_helm_step(HelmGrid g, HelmPlan pl, const __grid_constant__ HelmAxes ax,
                const __grid_constant__ HelmInvd iv, const double *__restrict__ r,
                const double *__restrict__ p, double *__restrict__ pn, double *__restrict__ Ap,
                double *__restrict__ partials, CgScalars *s)
{
  chain_wait();
  extern __shared__ __align__(16) unsigned char helm_raw[];
  constexpr int kTy = HelmTile<Rows>::ty, kHalo = HelmTile<Rows>::halo;
  constexpr int kStage = HelmTile<Rows>::stage;
  HelmShared<Rows> &S = *reinterpret_cast<HelmShared<Rows> *>(helm_raw);
  __shared__ double sh[32], s_iv[kHelmClasses];
  if(s->done)
    return;
  if(threadIdx.x < kHelmClasses)
    s_iv[threadIdx.x] = iv.v[threadIdx.x];
  const double beta = s->beta;
  const int NZ = g.nz + 1;
  const int plane = g.NX * g.NY;
  const double c = ax.c;
  const int lx = threadIdx.x & 31, ly = (threadIdx.x >> 5) * Rows;
  double dot = 0.0;
  for(int t = blockIdx.x; t < pl.items; t += gridDim.x)
  {
    const int i0 = t % pl.tiles_x * kHelmTx, j0 = t / pl.tiles_x % pl.tiles_y * kTy;
    const int k0 = t / (pl.tiles_x * pl.tiles_y) * pl.kz;
    const int k1 = min(k0 + pl.kz, NZ);
    const int i = i0 + lx, j = j0 + ly;
    // this thread's staged cells: in-plane offset (-1 outside), class of x and
    // y, whether the block owns the column
    int off[kStage], cls[kStage];
    bool own[kStage];
#pragma unroll
    for(int q = 0; q < kStage; q++)
    {
      const int e = threadIdx.x + q * kHelmThreads;
      const int hx = e % kHaloX, hy = e / kHaloX;
      const int x = i0 - 1 + hx, y = j0 - 1 + hy;
      const bool in = e < kHalo && x >= 0 && x < g.NX && y >= 0 && y < g.NY;
      off[q] = in ? x + y * g.NX : -1;
      cls[q] = in ? node_class(x, g.NX) + 3 * node_class(y, g.NY) : 0;
      own[q] = in && hx > 0 && hx <= kHelmTx && hy > 0 && hy <= kTy;
    }
    auto stage = [&](int k) { // raw plane k into its ring slot
      if(k <= k1)
      {
        const int slot = (k - k0 + 1) & (kHelmRing - 1);
        const bool inz = k >= 0 && k < NZ;
#pragma unroll
        for(int q = 0; q < kStage; q++)
        {
          const int e = threadIdx.x + q * kHelmThreads;
          if(e < kHalo)
          {
            const bool v = inz && off[q] >= 0;
            const int n = v ? off[q] + k * plane : 0;
            cp_async8(&S.r[slot][e], r + n, v);
            cp_async8(&S.p[slot][e], p + n, v);
          }
        }
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto combine = [&](int k) { // new p of plane k
      if(k > k1)
        return;
      const int slot = (k - k0 + 1) & (kHelmRing - 1);
      const int cz = 9 * node_class(min(max(k, 0), NZ - 1), NZ);
      const bool mine = k >= k0 && k < k1;
#pragma unroll
      for(int q = 0; q < kStage; q++)
      {
        const int e = threadIdx.x + q * kHelmThreads;
        if(e < kHalo)
        {
          const double z = S.r[slot][e] * s_iv[cls[q] + cz];
          const double v = beta == 0.0 ? z : fma(beta, S.p[slot][e], z);
          S.q[(k - k0) & 1][e] = v;
          if(mine && own[q])
            pn[off[q] + k * plane] = v;
        }
      }
    };
    // centre weights of this thread's nodes
    const double ex = node_class(min(i, g.NX - 1), g.NX) == 1 ? 2.0 : 1.0;
    const double mx = ex * ax.md[0], sx = ex * ax.sd[0];
    double my[Rows], sy[Rows];
#pragma unroll
    for(int q = 0; q < Rows; q++)
    {
      const double ey = node_class(min(j + q, g.NY - 1), g.NY) == 1 ? 2.0 : 1.0;
      my[q] = ey * ax.md[1];
      sy[q] = ey * ax.sd[1];
    }
    __syncthreads(); // the previous item's tiles have been read, s_iv is set
#pragma unroll
    for(int q = 0; q <= kHelmAhead; q++)
      stage(k0 - 1 + q);
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kHelmAhead) : "memory");
    __syncthreads();
    combine(k0 - 1);
    // per row: L = this plane's share of either neighbour plane's K p, done =
    // the output plane's sum but for the plane above, its p
    double L[Rows] = {}, done[Rows] = {}, pc[Rows] = {};
    for(int m = k0 - 1; m <= k1; m++)
    {
      // raw plane m + 1 has landed and the new p of plane m is complete
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kHelmAhead - 1) : "memory");
      __syncthreads();
      stage(m + 1 + kHelmAhead);
      combine(m + 1);
      const double *buf = S.q[(m - k0) & 1] + ly * kHaloX + lx;
      double rm[Rows + 2], rs[Rows + 2], pn0[Rows];
#pragma unroll
      for(int q = 0; q < Rows + 2; q++)
      {
        const double v0 = buf[q * kHaloX + 1], t = buf[q * kHaloX] + buf[q * kHaloX + 2];
        rm[q] = fma(ax.mo[0], t, mx * v0);
        rs[q] = fma(ax.so[0], t, sx * v0);
        if(q >= 1 && q <= Rows)
          pn0[q - 1] = v0;
      }
      const double ez = node_class(min(max(m, 0), NZ - 1), NZ) == 1 ? 2.0 : 1.0;
      const double mz = ez * ax.md[2], sz = ez * ax.sd[2] * ax.c, so = ax.so[2] * ax.c;
#pragma unroll
      for(int q = 0; q < Rows; q++)
      {
        const double tm = rm[q] + rm[q + 2], ts = rs[q] + rs[q + 2];
        const double B = fma(ax.mo[1], tm, my[q] * rm[q + 1]);
        const double D = fma(ax.so[1], tm, sy[q] * rm[q + 1]) +
                         fma(ax.mo[1], ts, my[q] * rs[q + 1]);
        const double A = fma(ax.c, D, B);
        const double up = fma(so, B, ax.mo[2] * A);
        if(m >= k0 + 1)
        {
          const double y = done[q] + up;
          if(i < g.NX && j + q < g.NY)
          {
            Ap[i + (j + q) * g.NX + (m - 1) * plane] = y;
            dot += pc[q] * y;
          }
        }
        done[q] = L[q] + fma(sz, B, mz * A);
        L[q] = up;
        pc[q] = pn0[q];
      }
    }
  }
  double v[1] = {dot};
  block_sum<1>(v, sh);
  if(threadIdx.x == 0)
    partials[blockIdx.x] = v[0];
  if(last_block(&s->counter))
  {
    double t[1];
    sum_partials<1>(partials, gridDim.x, t, sh);
    if(threadIdx.x == 0)
    {
      s->pAp = t[0];
      s->alpha = s->zr / t[0];
      s->counter = 0;
    }
  }
}

// The Jacobi CG update of k_cg_update_jacobi (x += alpha p, r -= alpha Ap,
// z = D^-1 r, beta, stop test) with D^-1 taken from the node's class instead
// of a vector and z not stored: the next k_helm_step forms it again from r.
__global__ void k_helm_update(HelmGrid g, HelmInvd iv, double *__restrict__ x,
                              double *__restrict__ r, const double *__restrict__ p,
                              const double *__restrict__ Ap, double *__restrict__ partials,
                              CgScalars *s)
{
  chain_wait();
  __shared__ double sh[64];
  if(s->done)
    return;
  const double alpha = s->alpha;
  double zr = 0.0, rr = 0.0;
  for(int n = blockIdx.x * blockDim.x + threadIdx.x; n < g.numnp;
      n += gridDim.x * blockDim.x)
  {
    x[n] += alpha * p[n];
    const double ri = r[n] - alpha * Ap[n];
    r[n] = ri;
    const double zi = ri * iv.v[helm_class(g, n)];
    zr += zi * ri;
    rr += ri * ri;
  }
  double v[2] = {zr, rr};
  block_sum<2>(v, sh);
  if(threadIdx.x == 0)
  {
    partials[blockIdx.x] = v[0];
    partials[gridDim.x + blockIdx.x] = v[1];
  }
  if(last_block(&s->counter))
  {
    double t[2];
    sum_partials<2>(partials, gridDim.x, t, sh);
    if(threadIdx.x == 0)
    {
      s->zr_new = t[0];
      s->beta = t[0] / s->zr;
      s->zr = t[0];
      cg_check(s, t[1]);
      s->counter = 0;
    }
  }
}

// out_e = sum_a ns[a] val[node_a] (/8 for the density call)
__global__ void k_helm_out(HelmGrid g, HelmWeights w, const double *__restrict__ val,
                           double *__restrict__ out, int sens)
{
  const long plane = (long)g.NX * g.NY;
  for(int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.nelx;
      e += gridDim.x * blockDim.x)
  {
    const int i = e % g.nx, j = (e / g.nx) % g.ny, k = e / (g.nx * g.ny);
    const long n0 = i + (long)j * g.NX + k * plane;
    double s = 0.0;
#pragma unroll
    for(int a = 0; a < 8; a++)
    {
      const long m = n0 + (a & 1) + ((a >> 1) & 1) * (long)g.NX + ((a >> 2) & 1) * plane;
      s = __dadd_rn(s, __dmul_rn(w.ns[a], __ldg(val + m)));
    }
    out[e] = sens ? s : __dmul_rn(s, 0.125); // = s / 8 in every case
  }
}

int blocks_for(long n, int threads, int cap)
{
  long b = (n + threads - 1) / threads;
  if(b > cap)
    b = cap;
  return b < 1 ? 1 : (int)b;
}

} // namespace

// The 8 x 8 element matrix of one hx x hy x hz voxel and its shape-function
// integrals, 2 x 2 x 2 Gauss points (makeKeFint, filter_helm.hpp:203-217).
// The voxel's Jacobian is diag(hx, hy, hz) / 2.
void helm_element(double hx, double hy, double hz, double R, double *ke, double *nj,
                  double *ns)
{
  const double g = 1.0 / std::sqrt(3.0);
  const double cdiff = std::pow(R / (2.0 * std::sqrt(3.0)), 2);
  const double h[3] = {hx, hy, hz};
  const double jac = (hx * 0.5) * (hy * 0.5) * (hz * 0.5);
  for(int t = 0; t < 64; t++)
    ke[t] = 0.0;
  for(int a = 0; a < 8; a++)
    nj[a] = ns[a] = 0.0;
  for(int ip = 0; ip < 8; ip++)
  {
    const double r[3] = {(ip & 1) ? g : -g, (ip & 2) ? g : -g, (ip & 4) ? g : -g};
    double N[8], B[3][8];
    for(int a = 0; a < 8; a++)
    {
      double f[3], df[3];
      for(int d = 0; d < 3; d++)
      {
        const double sgn = ((a >> d) & 1) ? 1.0 : -1.0;
        f[d] = 1.0 + sgn * r[d];
        df[d] = sgn;
      }
      N[a] = 0.125 * f[0] * f[1] * f[2];
      B[0][a] = 0.125 * df[0] * f[1] * f[2] * (2.0 / h[0]);
      B[1][a] = 0.125 * f[0] * df[1] * f[2] * (2.0 / h[1]);
      B[2][a] = 0.125 * f[0] * f[1] * df[2] * (2.0 / h[2]);
    }
    for(int a = 0; a < 8; a++)
    {
      for(int b = 0; b < 8; b++)
      {
        double sb = 0.0;
        for(int d = 0; d < 3; d++)
          sb += B[d][a] * cdiff * B[d][b];
        ke[8 * a + b] += (N[a] * N[b] + sb) * jac;
      }
      nj[a] += N[a] * jac;
      ns[a] += N[a];
    }
  }
}

// 27 node classes x 27 neighbour slots: class (cx, cy, cz), c = 0 on the
// lower face, 1 inside, 2 on the upper face of an axis; the node's elements
// sit at offsets o in {-1, 0}^3 (o = -1 exists unless c = 0, o = 0 unless
// c = 2) and are summed in ascending element id like the assembly of
// setFromTriplets over the reference's element loop.
static void helm_class_table(const double *ke, double *coef)
{
  for(int cz = 0; cz < 3; cz++)
    for(int cy = 0; cy < 3; cy++)
      for(int cx = 0; cx < 3; cx++)
      {
        const int cls = cx + 3 * cy + 9 * cz;
        const int cc[3] = {cx, cy, cz};
        for(int q = 0; q < 27; q++)
        {
          const int dd[3] = {q % 3 - 1, q / 3 % 3 - 1, q / 9 - 1};
          double v = 0.0;
          for(int oz = -1; oz <= 0; oz++)
            for(int oy = -1; oy <= 0; oy++)
              for(int ox = -1; ox <= 0; ox++)
              {
                const int o[3] = {ox, oy, oz};
                bool ok = true;
                int a = 0, b = 0;
                for(int d = 0; d < 3; d++)
                {
                  if((o[d] == -1 && cc[d] == 0) || (o[d] == 0 && cc[d] == 2))
                    ok = false;
                  const int ad = -o[d], bd = ad + dd[d];
                  if(bd < 0 || bd > 1)
                    ok = false;
                  a |= ad << d;
                  b |= (bd & 1) << d;
                }
                if(ok)
                  v += ke[8 * a + b];
              }
          coef[27 * cls + q] = v;
        }
      }
}

// the assembled 1-D stencils of each axis: element mass h/6 [2 1; 1 2] and
// stiffness 1/h [1 -1; -1 1] summed over the one (face) or two (inside)
// elements of a node
static HelmAxes helm_axes(const icarat_ctx *c)
{
  HelmAxes a{};
  const double h[3] = {c->hx, c->hy, c->hz};
  for(int d = 0; d < 3; d++)
  {
    a.mo[d] = h[d] / 6.0;
    a.md[d] = h[d] / 3.0;
    a.so[d] = -1.0 / h[d];
    a.sd[d] = 1.0 / h[d];
  }
  a.c = std::pow(c->helm.radius / (2.0 * std::sqrt(3.0)), 2);
  return a;
}

void helm_free(icarat_ctx *c)
{
  HelmState &H = c->helm;
  if(H.exec)
    cudaGraphExecDestroy(H.exec);
  for(double *p : {H.d_val, H.d_r, H.d_p[0], H.d_p[1], H.d_Ap, H.d_partials, H.d_oc})
    dfree(p);
  dfree(H.d_cg);
  H = HelmState{};
}

void helm_setup(icarat_ctx *c, double R)
{
  IREQUIRE(R >= 0.0 && std::isfinite(R), ICARAT_ERR_ARG, "filter radius must be >= 0");
  HelmState &H = c->helm;
  if(H.ready && H.radius == R)
    return; // the same operator on the same mesh: every buffer is a call's own
  helm_free(c);
  H.radius = R;
  helm_element(c->hx, c->hy, c->hz, R, H.ke, H.nj, H.ns);
  double coef[kHelmClasses * 27];
  helm_class_table(H.ke, coef);
  for(int q = 0; q < kHelmClasses; q++)
    H.invd_cls[q] = 1.0 / coef[27 * q + 13];
  const size_t n = (size_t)c->numnp;
  H.d_val = dalloc(n);
  H.d_r = dalloc(n);
  H.d_p[0] = dalloc(n);
  H.d_p[1] = dalloc(n);
  H.d_Ap = dalloc(n);
  H.d_partials = dalloc((size_t)kMaxRedBlocks * 2);
  H.d_oc = dalloc(3 * (size_t)c->nelx);
  ICK(cudaMalloc(&H.d_cg, sizeof(CgScalars)));
  ICK(cudaMemsetAsync(H.d_cg, 0, sizeof(CgScalars), c->stream));
  ICK(cudaFuncSetAttribute(k_helm_step<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(HelmShared<2>)));
  H.ready = true;
}

// grid of the streaming CG kernels: 8 blocks of 256 threads per SM (full
// occupancy; 4 per SM left them at 3-4 TB/s on the B200)
static int helm_red_blocks(const icarat_ctx *c)
{
  const int need = (c->numnp + 511) / 512;
  const int most = 8 * c->sm_count < kMaxRedBlocks ? 8 * c->sm_count : kMaxRedBlocks;
  return need < 1 ? 1 : (need < most ? need : most);
}

// Planes per item for the least of waves x (planes + start-up): two planes of
// halo are formed again per chunk and kHelmBlocks blocks fit an SM.
static HelmPlan helm_plan(const icarat_ctx *c)
{
  const int ty = helm_rows(c->NY) == 1 ? HelmTile<1>::ty : HelmTile<2>::ty;
  HelmPlan p{(c->NX + kHelmTx - 1) / kHelmTx, (c->NY + ty - 1) / ty, c->NZ, 0};
  const long tiles = (long)p.tiles_x * p.tiles_y, slots = (long)kHelmBlocks * c->sm_count;
  double best = 0.0;
  for(int kz = 1; kz <= c->NZ; kz++)
  {
    const long items = tiles * ((c->NZ + kz - 1) / kz);
    const double cost = (double)((items + slots - 1) / slots) * (kz + 4.0);
    if(best == 0.0 || cost <= best)
    {
      best = cost;
      p.kz = kz;
    }
  }
  p.items = (int)(tiles * ((c->NZ + p.kz - 1) / p.kz));
  return p;
}

static HelmInvd helm_invd(const icarat_ctx *c)
{
  HelmInvd iv;
  for(int q = 0; q < kHelmClasses; q++)
    iv.v[q] = c->helm.invd_cls[q];
  return iv;
}

// iteration k of a chunk: the directions alternate between the two vectors
static void helm_iteration(icarat_ctx *c, int k)
{
  HelmState &H = c->helm;
  const HelmPlan pl = helm_plan(c);
  const HelmInvd iv = helm_invd(c);
  const int blocks = pl.items < kMaxRedBlocks ? pl.items : kMaxRedBlocks;
  double *from = H.d_p[k & 1], *to = H.d_p[1 - (k & 1)];
  note_launch(2);
  if(helm_rows(c->NY) == 1)
    launch_chained(k_helm_step<1>, blocks, kHelmThreads, sizeof(HelmShared<1>), c->stream,
                   hgrid(c), pl, helm_axes(c), iv, H.d_r, from, to, H.d_Ap, H.d_partials, H.d_cg);
  else
    launch_chained(k_helm_step<2>, blocks, kHelmThreads, sizeof(HelmShared<2>), c->stream,
                   hgrid(c), pl, helm_axes(c), iv, H.d_r, from, to, H.d_Ap, H.d_partials, H.d_cg);
  launch_chained(k_helm_update, helm_red_blocks(c), kRedThreads, 0, c->stream, hgrid(c), iv,
                 H.d_val, H.d_r, to, H.d_Ap, H.d_partials, H.d_cg);
  ICK(cudaGetLastError());
}

// densityFilter (filter_helm.hpp:75-138) of the device vector in (nelx) into
// out (nelx); rtol / maxit of the CG (<= 0: the reference's 1e-10 / 10000)
int helm_filter(icarat_ctx *c, const double *in, double *out, bool is_sens, double rtol,
                int maxit, icarat_solve_info *info)
{
  HelmState &H = c->helm;
  IREQUIRE(H.ready, ICARAT_ERR_STATE, "Helmholtz filter not set up");
  IREQUIRE(std::isfinite(rtol), ICARAT_ERR_ARG, "rtol must be finite");
  if(rtol <= 0.0)
    rtol = 1.0e-10;
  if(maxit <= 0)
    maxit = 10000;
  HelmWeights w;
  for(int a = 0; a < 8; a++)
  {
    w.nj[a] = H.nj[a];
    w.ns[a] = H.ns[a];
  }
  note_launch();
  k_helm_start<<<helm_red_blocks(c), kRedThreads, 0, c->stream>>>(
      hgrid(c), w, helm_invd(c), in, H.d_val, H.d_r, is_sens ? 1 : 0, H.d_partials, H.d_cg, rtol,
      maxit);
  ICK(cudaGetLastError());
  if(!H.exec)
  {
    cudaGraph_t graph;
    ICK(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
    set_capturing(true);
    try
    {
      for(int k = 0; k < kHelmChunk; k++)
        helm_iteration(c, k);
    }
    catch(...)
    {
      set_capturing(false);
      cudaStreamEndCapture(c->stream, &graph);
      throw;
    }
    set_capturing(false);
    ICK(cudaStreamEndCapture(c->stream, &graph));
    ICK(cudaGraphInstantiate(&H.exec, graph, 0));
    cudaGraphDestroy(graph);
  }
  const long max_chunks = ((long)maxit + 1 + kHelmChunk - 1) / kHelmChunk + 1;
  for(long ch = 0; ch < max_chunks; ch++)
  {
    ICK(cudaMemcpyAsync(c->h_cg, H.d_cg, sizeof(CgScalars), cudaMemcpyDeviceToHost,
                        c->stream));
    ICK(cudaStreamSynchronize(c->stream));
    if(c->h_cg->done)
      break;
    ICK(cudaGraphLaunch(H.exec, c->stream));
    note_launch(2 * kHelmChunk);
  }
  note_launch();
  k_helm_out<<<blocks_for(c->nelx, kHelmThreads, 4 * c->sm_count), kHelmThreads, 0,
               c->stream>>>(hgrid(c), w, H.d_val, out, is_sens ? 1 : 0);
  ICK(cudaGetLastError());
  ICK(cudaMemcpyAsync(c->h_cg, H.d_cg, sizeof(CgScalars), cudaMemcpyDeviceToHost,
                      c->stream));
  ICK(cudaStreamSynchronize(c->stream));
  const CgScalars &s = *c->h_cg;
  const int status = s.done ? s.status : ICARAT_WARN_MAXITER;
  if(info)
  {
    *info = icarat_solve_info{};
    info->iterations = s.iter;
    info->rel_residual = s.bnorm > 0 ? s.rnorm / s.bnorm : 0.0;
    info->status = status;
  }
  return status;
}

} // namespace icarat_b200
