// Radius filter sums of a tile of elements from shared memory.
//
// The stencil of a radius R on cubic voxels is the ball di^2 + dj^2 + dk^2 <=
// D2 with D2 = floor((R / h)^2): for R up to 3 voxels (D2 <= 9) the taps are
// compile-time constants, so a thread's sums unroll with no offset loads,
// bounds tests or predicates and with the weights in the constant bank.  A
// block of 32 x kBallY threads stages its elements and their halo once (cp.async,
// positions outside the box hold 0, which adds exactly nothing); a thread
// owns kBallZ consecutive elements along z and every staged value it reads
// serves all of them.  Each sum still runs over (dk, dj, di) ascending, the
// order of the reference's neighbour list, without contraction.
//
// Bound by shared-memory reads and the FP64 pipe about equally (r = 2: 37
// reads and 57 to 81 products and sums per element).  Measured on a B200 at
// 128 x 64 x 64 elements, per-tap offset list before and now, call by call:
// forward 66 -> 14.7 us and transposed 82 -> 26.9 us at R = 2.5, 21 -> 8.9 and
// 25 -> 12.5 us at R = 1.5, 97 -> 18.7 and 123 -> 51 us at R = 3 (three staged
// arrays leave one block per SM there).
#pragma once
#include <type_traits>

#include "internal.cuh"

namespace icarat_b200
{

constexpr int kBallX = 32, kBallY = 8, kBallZ = 4;

template <int D2> struct Ball
{
  static constexpr int r = D2 >= 9 ? 3 : (D2 >= 4 ? 2 : 1);
  static constexpr int sx = kBallX + 2 * r, sy = kBallY + 2 * r, sz = kBallZ + 2 * r;
  static constexpr int tile = sx * sy * sz;
  static constexpr __host__ __device__ bool in(int dk, int dj, int di)
  {
    return dk * dk + dj * dj + di * di <= D2;
  }
  // a tap's weight: it depends on the offsets' sizes only, so one octant
  // (the launch carries at most 64 values)
  static constexpr __host__ __device__ int index(int dk, int dj, int di)
  {
    const int a = di < 0 ? -di : di, b = dj < 0 ? -dj : dj, c = dk < 0 ? -dk : dk;
    return (c * (r + 1) + b) * (r + 1) + a;
  }
  static constexpr int weights = (r + 1) * (r + 1) * (r + 1);
  // some element of a thread's kBallZ has a tap at staged layer z, (dj, di)
  static constexpr __host__ __device__ bool used(int z, int dj, int di)
  {
    for(int o = 0; o < kBallZ; o++)
      if(in(z - r - o, dj, di))
        return true;
    return false;
  }
};

template <int D2> struct BallWeights
{
  double w[Ball<D2>::weights];
};

// the elements a block works on: origin and box
struct BallGrid
{
  int nx, ny, nz, nelx;
  const uint8_t *mask; // elements kept by a selection (null: all)
};

__host__ __device__ inline int ball_tiles(int n, int t) { return (n + t - 1) / t; }
inline long ball_blocks(int nx, int ny, int nz)
{
  return (long)ball_tiles(nx, kBallX) * ball_tiles(ny, kBallY) * ball_tiles(nz, kBallZ);
}

// A tile costs the same however few of its elements lie in the box, so thin
// grids (plates, bars) are faster by the offset list: the share of the tiles'
// elements from which the ball is, measured on plates of 1 to 33 elements and
// bars (list time over ball time 1.0 to 1.1 there, 0.1 to 0.4 at a share of
// 0.03, 1.4 to 7.5 on full tiles).
enum BallUse
{
  kBallForward,
  kBallTransposed,
  kBallBisect
};
inline bool ball_pays(int d2, BallUse use, int nx, int ny, int nz)
{
  double share = 0.15;
  if(use == kBallForward)
    share = d2 == 1 ? 0.5 : d2 <= 4 ? 0.3 : 0.15;
  if(use == kBallTransposed)
    share = d2 == 1 ? 0.5 : 0.4;
  const long blocks = ball_blocks(nx, ny, nz);
  return blocks < (1L << 31) &&
         (double)nx * ny * nz >= share * (double)blocks * (kBallX * kBallY * kBallZ);
}

__device__ __forceinline__ void ball_origin(const BallGrid &g, long b, int &x0, int &y0, int &z0)
{
  const int tx = ball_tiles(g.nx, kBallX), ty = ball_tiles(g.ny, kBallY);
  x0 = (int)(b % tx) * kBallX;
  y0 = (int)(b / tx % ty) * kBallY;
  z0 = (int)(b / ((long)tx * ty)) * kBallZ;
}

// put(position in the tile, element or -1) for the tile and its halo
template <int D2, typename F>
__device__ __forceinline__ void ball_stage(const BallGrid &g, int x0, int y0, int z0, F &&put)
{
  using B = Ball<D2>;
  for(int q = threadIdx.x; q < B::tile; q += kBallX * kBallY)
  {
    const int x = x0 - B::r + q % B::sx, y = y0 - B::r + q / B::sx % B::sy,
              z = z0 - B::r + q / (B::sx * B::sy);
    const bool in = x >= 0 && x < g.nx && y >= 0 && y < g.ny && z >= 0 && z < g.nz;
    int e = in ? x + y * g.nx + z * g.nx * g.ny : -1;
    if(e >= 0 && g.mask && !g.mask[e])
      e = -1;
    put(q, e);
  }
}

__device__ __forceinline__ void ball_copy(double *dst, const double *src, int e)
{
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = e >= 0 ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d),
               "l"(src + (e >= 0 ? e : 0)), "r"(n)
               : "memory");
}

// Every tap of this thread's kBallZ elements: v = load(position in the tile)
// once per staged value, then term(o, weight index, v) for each element o that
// has it as a neighbour, each element's taps in ascending (dk, dj, di).
template <int D2, typename L, typename F>
__device__ __forceinline__ void ball_sum(L &&load, F &&term)
{
  using B = Ball<D2>;
  const int base = (threadIdx.x % kBallX) + (threadIdx.x / kBallX) * B::sx;
#pragma unroll
  for(int z = 0; z < B::sz; z++)
#pragma unroll
    for(int dj = -B::r; dj <= B::r; dj++)
#pragma unroll
      for(int di = -B::r; di <= B::r; di++)
        if(B::used(z, dj, di))
        {
          const auto v = load(base + (z * B::sy + dj + B::r) * B::sx + di + B::r);
#pragma unroll
          for(int o = 0; o < kBallZ; o++)
            if(B::in(z - B::r - o, dj, di))
              term(o, B::index(z - B::r - o, dj, di), v);
        }
}

// call f(std::integral_constant<int, D2>) for the compiled ball d2
template <typename F> inline void ball_dispatch(int d2, F &&f)
{
  switch(d2)
  {
  case 1: f(std::integral_constant<int, 1>()); break;
  case 2: f(std::integral_constant<int, 2>()); break;
  case 3: f(std::integral_constant<int, 3>()); break;
  case 4: f(std::integral_constant<int, 4>()); break;
  case 5: f(std::integral_constant<int, 5>()); break;
  case 6: f(std::integral_constant<int, 6>()); break;
  case 8: f(std::integral_constant<int, 8>()); break;
  case 9: f(std::integral_constant<int, 9>()); break;
  default: throw Error{ICARAT_ERR_STATE, "no compiled ball of this radius"};
  }
}

} // namespace icarat_b200
