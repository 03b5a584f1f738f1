// Jacobi-PCG in one cooperative launch for grids that fit the SMs' shared
// memory.
//
// On small grids an iteration of three launches (K p with p.Kp, the update
// with z.r and r.r, p = z + beta p) is all latency: 16 us at 33 x 17 x 17
// nodes, whose products and sums take well under one.  Here every block (one
// per SM) keeps x, r, D^-1, K p and its tile of p with a halo of one node in
// shared memory for the whole solve, and an iteration has two grid-wide
// steps, one per reduction.
//
// What blocks tell each other carries its own mark: a double travels as two
// 64-bit words of 32 data bits and the step's number each (single stores, so
// a word is never seen half written), and the reader repeats its load until
// both marks are the step's.  No fence, barrier or second load is needed:
// partial sums are posted, added group by group and then over the groups by
// every block alike, so all take the same scalars; the values
// of z = D^-1 r that a neighbour's halo needs go the same way while the second
// reduction is under way, and p = beta p + z is formed in the tile.  Partial
// sums alternate between two sets: a block writes a set again only after a
// step that every block entered having read it; z of the next iteration is
// written after a reduction that every block entered having read this one's.
// Marks start at 1 in buffers cleared before the launch.
//
// K p is the march of modal.cuh over the tile (threads: element columns times
// slabs of kc layers).  Scalars and stop rule are those of pcg.cu.
//
// Measured on a B200, per iteration, three launches before (with the old
// product) and now: 33 x 17 x 17 nodes 16.4 -> 9.0 us, 48 x 30 x 21 18.0 -> 9.7,
// 126 x 26 x 26 27.9 -> 11.7.  A trip through the L2 costs about 1 us and an
// iteration makes five (two per reduction, one for z); a march step takes 0.9.
//
// Solves of several contexts share the GPU as far as their blocks fit side by
// side: two threads with eight solves each take 41.6 ms at 33 x 17 x 17 nodes (one
// after another 79.6; with three launches per iteration 82.3), and 358 ms at 126
// x 26 x 26, where one solve fills the GPU (366; 544).
//
// Waits are bounded: a block whose wait runs out reports an error status and
// leaves, and so does every other that still waits for it.
#include "modal.cuh"
#include "resident_cg.cuh"

namespace icarat_b200
{

namespace
{

constexpr int kResThreads = 384; // 12 warps: 168 registers for the march
constexpr size_t kResSmem = 225 * 1024;
constexpr unsigned kResPolls = 1u << 22;
constexpr int kNone = -1, kOwn = -2, kEdge = 1 << 30;

struct ResidentShape
{
  int cells, nodes; // tile with halo, owned nodes (slab layers rounded up)
};

__host__ __device__ inline ResidentShape shape(const ResidentPlan &p)
{
  const int bz = p.S * p.kc;
  return ResidentShape{(p.BX + 2) * (p.BY + 2) * (bz + 2), p.BX * p.BY * bz};
}

// blocks per group of the reductions: about the square root, at most 16
__host__ __device__ inline int group_size(int nb)
{
  int s = 1;
  while(s * s < nb && s < 16)
    s++;
  return s;
}

size_t smem_of(const ResidentPlan &p)
{
  const ResidentShape h = shape(p);
  return sizeof(double) * (6 * (size_t)h.cells + 12 * (size_t)h.nodes + 18 * (size_t)kResThreads) +
         sizeof(int) * ((size_t)h.cells + 2 * h.nodes);
}

// a double as two marked words (see above), and back: false until both words
// carry the mark
__device__ __forceinline__ void post(unsigned long long *lo, unsigned long long *hi, double v,
                                     unsigned mark)
{
  const unsigned long long m = (unsigned long long)mark << 32;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(lo),
               "l"(m | (unsigned)__double2loint(v))
               : "memory");
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(hi),
               "l"(m | (unsigned)__double2hiint(v))
               : "memory");
}
__device__ __forceinline__ unsigned long long word(const unsigned long long *p)
{
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// waits (with a limit) for N marked doubles, all loads of a round in flight
template <int N>
__device__ __forceinline__ bool collect(const unsigned long long *const (&lo)[N],
                                        const unsigned long long *const (&hi)[N], unsigned mark,
                                        double (&v)[N])
{
  for(unsigned n = 0; n < kResPolls; n++)
  {
    unsigned long long a[N], b[N];
    bool all = true;
#pragma unroll
    for(int q = 0; q < N; q++)
    {
      a[q] = word(lo[q]);
      b[q] = word(hi[q]);
    }
#pragma unroll
    for(int q = 0; q < N; q++)
    {
      all = all && (unsigned)(a[q] >> 32) == mark && (unsigned)(b[q] >> 32) == mark;
      v[q] = __hiloint2double((int)(unsigned)b[q], (int)(unsigned)a[q]);
    }
    if(all)
      return true;
  }
  return false;
}

// sum of the marked doubles set[0 .. n) (n <= 16) over the lanes of a warp, in
// lane 0; words of value q of slot b at (2 q) stride + b and (2 q + 1) stride + b
template <int NV>
__device__ __forceinline__ void warp_collect(const unsigned long long *set, int stride, int n,
                                             unsigned mark, int lane, double (&t)[NV], int *bad)
{
  const unsigned long long *lo[NV], *hi[NV];
#pragma unroll
  for(int q = 0; q < NV; q++)
  {
    lo[q] = set + (2 * q) * stride + lane;
    hi[q] = set + (2 * q + 1) * stride + lane;
    t[q] = 0.0;
  }
  if(lane < n && !collect<NV>(lo, hi, mark, t))
    *bad = 1;
  __syncwarp();
#pragma unroll
  for(int q = 0; q < NV; q++)
    for(int o = 8; o > 0; o >>= 1)
      t[q] += __shfl_down_sync(0xffffffffu, t[q], o);
}

// Grid-wide sums of NV values per thread, the same bits in every block:
// last(sums) runs in one thread, before a barrier.  between() runs between this
// block's post and the wait for the others.  Blocks go in groups of up to 16
// whose first block adds the group's sums, and every block adds the groups':
// two trips through the L2, but each word has few readers (every block reading every block's words took 5 us at
// 128 blocks, the readers' repeated loads queueing in the L2).
// sums: [2][NV <= 2][2 words][blocks + groups].
template <int NV, typename F, typename L>
__device__ void grid_sum(double (&v)[NV], unsigned mark, int nb, unsigned long long *sums,
                         double *sh, int *bad, F &&between, L &&last)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int size = group_size(nb), groups = (nb + size - 1) / size, stride = nb + groups;
  unsigned long long *set = sums + (size_t)(mark & 1) * 4 * stride;
#pragma unroll
  for(int q = 0; q < NV; q++)
    for(int o = 16; o > 0; o >>= 1)
      v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
  if(lane == 0)
#pragma unroll
    for(int q = 0; q < NV; q++)
      sh[q * 32 + w] = v[q];
  __syncthreads();
  if(w == 0)
  {
#pragma unroll
    for(int q = 0; q < NV; q++)
    {
      v[q] = lane < kResThreads / 32 ? sh[q * 32 + lane] : 0.0;
      for(int o = 8; o > 0; o >>= 1)
        v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
      if(lane == 0)
        post(set + (2 * q) * stride + blockIdx.x, set + (2 * q + 1) * stride + blockIdx.x, v[q],
             mark);
    }
    if(blockIdx.x % size == 0)
    {
      double t[NV];
      warp_collect<NV>(set + blockIdx.x, stride, min(size, nb - (int)blockIdx.x), mark, lane, t,
                       bad);
      const int g = nb + blockIdx.x / size;
      if(lane == 0)
#pragma unroll
        for(int q = 0; q < NV; q++)
          post(set + (2 * q) * stride + g, set + (2 * q + 1) * stride + g, t[q], mark);
    }
  }
  between();
  if(w == 0)
  {
    double t[NV];
    warp_collect<NV>(set + nb, stride, groups, mark, lane, t, bad);
    if(lane == 0)
      last(t);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kResThreads, 1)
    k_resident_cg(GridDev g, ResidentPlan pl, const __grid_constant__ KhParam<double> kh,
                  const double *__restrict__ E, const double *__restrict__ invd, double *x,
                  double *r, double *p, unsigned long long *zlo, unsigned long long *zhi,
                  unsigned long long *sums, CgScalars *s, int chunk)
{
  extern __shared__ __align__(16) unsigned char res_raw[];
  __shared__ double sh[64];
  __shared__ int bad;
  __shared__ CgScalars S; // the block's copy; every block's holds the same bits
  if(s->done)
    return;
  const ResidentShape h = shape(pl);
  const int t = threadIdx.x, nb = gridDim.x;
  const int bz = pl.S * pl.kc;
  double *sp = reinterpret_cast<double *>(res_raw); // p tile [3][cells]
  double *sz = sp + 3 * h.cells;                    // z tile [3][cells]
  double *sq = sz + 3 * h.cells;                    // K p [3][nodes]
  double *sx = sq + 3 * h.nodes, *sr = sx + 3 * h.nodes, *sd = sr + 3 * h.nodes;
  double *sf = sd + 3 * h.nodes; // forces [2][9][threads]
  // node of a halo cell, kOwn for an owned one, kNone outside the box; node of
  // an owned node (kEdge set where a neighbour's halo holds it) or kNone
  int *cell = reinterpret_cast<int *>(sf + 18 * kResThreads);
  int *own = cell + h.cells, *inner = own + h.nodes; // inner: its tile cell
  const int x0 = (int)blockIdx.x % pl.nbx * pl.BX;
  const int y0 = (int)blockIdx.x / pl.nbx % pl.nby * pl.BY;
  const int z0 = (int)blockIdx.x / (pl.nbx * pl.nby) * bz;
  const int row = pl.BX + 2, plane = row * (pl.BY + 2);
  if(t == 0)
  {
    bad = 0;
    S = *s;
  }
  for(int q = t; q < h.cells; q += kResThreads)
  {
    const int i = x0 - 1 + q % row, j = y0 - 1 + q / row % (pl.BY + 2), k = z0 - 1 + q / plane;
    const bool in = i >= 0 && i < g.NX && j >= 0 && j < g.NY && k >= 0 && k < g.NZ;
    const int n = in ? i + j * g.NX + k * g.NX * g.NY : 0;
    const bool mine = i >= x0 && i < x0 + pl.BX && j >= y0 && j < y0 + pl.BY && k >= z0 &&
                      k < z0 + bz;
    cell[q] = in ? (mine ? kOwn : n) : kNone;
#pragma unroll
    for(int c = 0; c < 3; c++)
      sp[c * h.cells + q] = in ? __ldcg(p + (long)c * g.numnp + n) : 0.0;
  }
  for(int q = t; q < h.nodes; q += kResThreads)
  {
    const int i = x0 + q % pl.BX, j = y0 + q / pl.BX % pl.BY, k = z0 + q / (pl.BX * pl.BY);
    const bool in = i < g.NX && j < g.NY && k < g.NZ;
    const int n = in ? i + j * g.NX + k * g.NX * g.NY : 0;
    const bool edge = i == x0 || i == x0 + pl.BX - 1 || j == y0 || j == y0 + pl.BY - 1 ||
                      k == z0 || k == z0 + bz - 1;
    own[q] = in ? n | (edge ? kEdge : 0) : kNone;
    inner[q] = (k - z0 + 1) * plane + (j - y0 + 1) * row + i - x0 + 1;
#pragma unroll
    for(int c = 0; c < 3; c++)
    {
      const long id = (long)c * g.numnp + n;
      sx[c * h.nodes + q] = in ? x[id] : 0.0;
      sr[c * h.nodes + q] = in ? r[id] : 0.0;
      sd[c * h.nodes + q] = in ? invd[id] : 0.0;
      sq[c * h.nodes + q] = 0.0;
    }
  }
  // this thread's element column and slab
  const int cw = pl.BX + 1, ch = pl.BY + 1;
  const int cx = t % cw, cy = t / cw % ch, slab = t / (cw * ch);
  const bool active = slab < pl.S;
  const int l0 = active ? slab * pl.kc : 0; // tile layer of the slab's first lower face
  const int at0 = active ? cy * row + cx : 0;
  const int ei = x0 - 1 + cx, ej = y0 - 1 + cy;
  const bool elem = active && ei >= 0 && ei < g.nx && ej >= 0 && ej < g.ny;
  const bool column = active && cx > 0 && cy > 0;
  auto face = [&](int layer, double(&f)[3][4]) {
    const int at = at0 + layer * plane;
#pragma unroll
    for(int c = 0; c < 3; c++)
    {
      const double *tile = sp + c * h.cells + at;
      const double a = tile[0], b = tile[1], d = tile[row], e = tile[row + 1];
      const double s0 = a + b, d0 = b - a, s1 = d + e, d1 = e - d;
      f[c][0] = s0 + s1;
      f[c][1] = d0 + d1;
      f[c][2] = s1 - s0;
      f[c][3] = d1 - d0;
    }
  };
  auto modulus = [&](int layer) { // element between tile layers `layer` and + 1
    const int ek = z0 - 1 + layer;
    return elem && ek >= 0 && ek < g.nz ? __ldg(E + ei + ej * g.nx + ek * g.nx * g.ny) : 0.0;
  };
  unsigned mark = 0;
  __syncthreads();
  for(int it = 0; it < chunk && !S.done; it++)
  {
    // K p and p . K p
    double dot = 0.0;
    double f0[3][4], carry[3][4];
#pragma unroll
    for(int c = 0; c < 3; c++)
#pragma unroll
      for(int q = 0; q < 4; q++)
        carry[c][q] = 0.0;
    double Ee = modulus(l0);
    face(l0, f0);
#pragma unroll 1
    for(int q = 0; q <= pl.kc; q++)
    {
      const double En = modulus(l0 + q + 1);
      double f1[3][4], f[3][4];
      face(l0 + q + 1, f1);
      modal_element(kh, Ee, f0, f1, carry, f);
      if(q > 0)
      {
        double *fb = sf + (q & 1) * 9 * kResThreads;
        double acc[3];
#pragma unroll
        for(int c = 0; c < 3; c++)
        {
          const double a0 = f[c][0] - f[c][2], b0 = f[c][1] - f[c][3];
          const double a1 = f[c][0] + f[c][2], b1 = f[c][1] + f[c][3];
          acc[c] = a0 - b0;
          fb[(3 * c) * kResThreads + t] = a0 + b0;     // to the node at +x
          fb[(3 * c + 1) * kResThreads + t] = a1 - b1; // +y
          fb[(3 * c + 2) * kResThreads + t] = a1 + b1; // +x +y
        }
        __syncthreads();
        if(column)
        {
          const int n = ((l0 + q - 1) * pl.BY + cy - 1) * pl.BX + cx - 1;
#pragma unroll
          for(int c = 0; c < 3; c++)
          {
            acc[c] += fb[(3 * c) * kResThreads + t - 1];
            acc[c] += fb[(3 * c + 1) * kResThreads + t - cw];
            acc[c] += fb[(3 * c + 2) * kResThreads + t - cw - 1];
            const double y = sd[c * h.nodes + n] == 0.0 ? 0.0 : acc[c];
            sq[c * h.nodes + n] = y;
            dot += sp[c * h.cells + at0 + (l0 + q) * plane] * y;
          }
        }
      }
#pragma unroll
      for(int c = 0; c < 3; c++)
#pragma unroll
        for(int m = 0; m < 4; m++)
          f0[c][m] = f1[c][m];
      Ee = En;
    }
    double v1[1] = {dot};
    grid_sum<1>(v1, ++mark, nb, sums, sh, &bad, [] {}, [&](const double(&sum)[1]) {
      S.pAp = sum[0];
      S.alpha = S.zr / sum[0];
    });
    if(bad)
      break;
    const double alpha = S.alpha;
    // x += alpha p, r -= alpha K p, z = D^-1 r
    double v2[2] = {0.0, 0.0};
    ++mark;
    for(int q = t; q < h.nodes; q += kResThreads)
    {
      if(own[q] == kNone)
        continue;
      const int n = own[q] & ~kEdge;
      const int in = inner[q];
#pragma unroll
      for(int c = 0; c < 3; c++)
      {
        const int a = c * h.nodes + q;
        sx[a] = fma(alpha, sp[c * h.cells + in], sx[a]);
        const double ri = fma(-alpha, sq[a], sr[a]);
        sr[a] = ri;
        const double zi = ri * sd[a];
        sz[c * h.cells + in] = zi;
        if(own[q] & kEdge)
          post(zlo + (long)c * g.numnp + n, zhi + (long)c * g.numnp + n, zi, mark);
        v2[0] += zi * ri;
        v2[1] += ri * ri;
      }
    }
    auto halo = [&] {
      for(int q = t; q < h.cells; q += kResThreads)
      {
        const int n = cell[q];
        if(n < 0)
          continue;
        const unsigned long long *lo[3], *hi[3];
        double zn[3];
#pragma unroll
        for(int c = 0; c < 3; c++)
        {
          lo[c] = zlo + (long)c * g.numnp + n;
          hi[c] = zhi + (long)c * g.numnp + n;
        }
        if(!collect<3>(lo, hi, mark, zn))
          bad = 1;
#pragma unroll
        for(int c = 0; c < 3; c++)
          sz[c * h.cells + q] = zn[c];
      }
    };
    grid_sum<2>(v2, mark, nb, sums, sh, &bad, halo, [&](const double(&sum)[2]) {
      S.zr_new = sum[0];
      S.beta = sum[0] / S.zr;
      S.zr = sum[0];
      S.rr = sum[1];
    });
    if(bad)
      break;
    const double beta = S.beta;
    if(t == kResThreads - 32) // one thread of the last warp, beside the update of p
      cg_check(&S, S.rr);
    // p = z + beta p in the tile and its halo
    for(int q = t; q < h.cells; q += kResThreads)
      if(cell[q] != kNone)
#pragma unroll
        for(int c = 0; c < 3; c++)
        {
          const int a = c * h.cells + q;
          sp[a] = fma(beta, sp[a], sz[a]);
        }
    __syncthreads();
  }
  for(int q = t; q < h.nodes; q += kResThreads)
  {
    if(own[q] == kNone)
      continue;
    const int n = own[q] & ~kEdge;
    const int in = inner[q];
#pragma unroll
    for(int c = 0; c < 3; c++)
    {
      const long id = (long)c * g.numnp + n;
      x[id] = sx[c * h.nodes + q];
      r[id] = sr[c * h.nodes + q];
      p[id] = sp[c * h.cells + in];
    }
  }
  // Block 0 reports the solve.  A block that lost a wait is not always seen by
  // the others (they enter no further step after the launch's last), and may
  // report before or after block 0: the verdict is settled by atomics, whose
  // outcome is the error in either order.
  if(t == 0 && blockIdx.x == 0)
  {
    s->alpha = S.alpha;
    s->beta = S.beta;
    s->zr = S.zr;
    s->zr_new = S.zr_new;
    s->pAp = S.pAp;
    s->rr = S.rr;
    s->rnorm = S.rnorm;
    s->iter = S.iter;
    if(S.done)
    {
      atomicCAS(&s->status, ICARAT_OK, S.status);
      atomicExch(&s->done, 1);
    }
  }
  if(t == 0 && bad)
  {
    atomicExch(&s->status, ICARAT_ERR_CUDA);
    atomicExch(&s->done, 1);
  }
}

} // namespace

// Every split of the box into at most one block per SM.  Cost of an iteration
// in units of about 95 cycles, fitted to the phases' measured cycles: march
// steps by their warps (1590 cycles at 6 warps, 1830 at 12), rounds of the
// vector passes, and the reductions by the number of blocks.
ResidentPlan resident_plan(const GridDev &g, int sms)
{
  static std::mutex mu;
  static std::map<std::tuple<int, int, int, int>, ResidentPlan> cache;
  ResidentPlan best{0, 0, 0, 0, 0, 0, 0, 0, 0};
  double best_cost = 0.0;
  sms = sms < 256 ? sms : 256; // 16 groups of 16
  if(g.numnp > 1200L * sms)
    return best; // beyond the shared memory of all SMs
  const auto key = std::make_tuple(g.NX, g.NY, g.NZ, sms);
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if(it != cache.end())
    return it->second;
  for(int nbx = 1; nbx <= g.NX && nbx <= sms; nbx++)
    for(int nby = 1; nby <= g.NY && nbx * nby <= sms; nby++)
    {
      const int BX = (g.NX + nbx - 1) / nbx, BY = (g.NY + nby - 1) / nby;
      const int cols = (BX + 1) * (BY + 1);
      if(cols > kResThreads || (nbx - 1) * BX >= g.NX || (nby - 1) * BY >= g.NY)
        continue;
      const int nbz_max = sms / (nbx * nby) < g.NZ ? sms / (nbx * nby) : g.NZ;
      for(int nbz = 1; nbz <= nbz_max; nbz++)
      {
        const int bz = (g.NZ + nbz - 1) / nbz;
        int S = kResThreads / cols;
        S = S > bz ? bz : S;
        const int kc = (bz + S - 1) / S;
        S = (bz + kc - 1) / kc;
        ResidentPlan p{BX, BY, S, kc, nbx, nby, (g.NZ + S * kc - 1) / (S * kc), 0, 0};
        p.blocks = nbx * nby * p.nbz;
        p.smem = smem_of(p);
        if(p.smem > kResSmem)
          continue;
        const ResidentShape h = shape(p);
        const double warps = (cols * S + 31) / 32;
        const double cost = (kc + 1.0) * (13.0 + 0.55 * warps) +
                            6.0 * ((h.nodes + kResThreads - 1) / kResThreads) +
                            4.0 * ((h.cells + kResThreads - 1) / kResThreads) + 0.2 * p.blocks;
        if(best.blocks == 0 || cost < best_cost)
        {
          best = p;
          best_cost = cost;
        }
      }
    }
  if(cache.size() > 256)
    cache.clear();
  cache[key] = best;
  return best;
}

size_t resident_work(const ResidentPlan &p) { return 16 * (size_t)p.blocks; }

const void *resident_kernel() { return (const void *)k_resident_cg; }

void resident_cg(cudaStream_t st, const ResidentPlan &p, const GridDev &g,
                 const KhParam<double> &kh, const double *E, const double *invd, double *x,
                 double *r, double *z, double *Ap, double *pv, double *work, CgScalars *s,
                 int chunk)
{
  auto *sums = reinterpret_cast<unsigned long long *>(work);
  auto *zlo = reinterpret_cast<unsigned long long *>(z);
  auto *zhi = reinterpret_cast<unsigned long long *>(Ap);
  ICK(cudaFuncSetAttribute(k_resident_cg, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kResSmem));
  // marks of earlier launches, and what else these buffers held, are gone
  ICK(cudaMemsetAsync(sums, 0, sizeof(double) * resident_work(p), st));
  ICK(cudaMemsetAsync(zlo, 0, sizeof(double) * 3 * g.numnp, st));
  ICK(cudaMemsetAsync(zhi, 0, sizeof(double) * 3 * g.numnp, st));
  GridDev gg = g;
  ResidentPlan pp = p;
  KhParam<double> kk = kh;
  void *args[] = {&gg, &pp, &kk, &E, &invd, &x, &r, &pv, &zlo, &zhi, &sums, &s, &chunk};
  note_launch();
  ICK(cudaLaunchCooperativeKernel((const void *)k_resident_cg, dim3(p.blocks), dim3(kResThreads),
                                  args, p.smem, st));
}

} // namespace icarat_b200
