// Backward 3x3x3 convolutions of the U-net on the tensor cores with FP32
// accuracy.
//
// Both gradients multiply BF16 data (activations or weights) by the FP32
// output gradient.  Its 24-bit significand is exactly three BF16 values
// (high, middle, low: each the rounded rest of the one before), so three
// BF16 products per term with FP32 sums replace an FP32 product.  (Below
// magnitudes of about 2^-109 the low part meets the smallest BF16 value,
// 2^-133, and what is under that is lost.)  The tensor
// core's own running sum is not used for long chains (it does not round to
// nearest): a chain ends after at most 9 products and is added to FP32
// registers.
//
// Operands are read channel-last, [voxel][channel] in rows of 16 channels (32
// bytes): a tap is then a shift by whole rows and ldmatrix delivers either
// orientation.  k_split turns the masked gradient into its three parts and
// the bias gradient's partial sums on the way, k_channel_last the activations.
// A block stages tiles of 16 x 4 x 4 voxels (with a halo of one where taps
// shift) by cp.async; the two 16-byte halves of a row swap with bit 2 of the
// row number, which keeps ldmatrix free of bank conflicts at every shift.
//
//   k_wgrad_mma  D (16 input x 16 output channels, 9 taps of one dz per warp)
//                += x^T dy over the voxels; blocks split the voxels, 4 warps
//                per dz the tile's planes, and fixed-order sums join them.
//   k_dgrad_mma  D (16 voxels x 16 or 32 input channels) += dy W over taps
//                and chunks of 16 output channels.
//
// Measured on a B200, before (FP32 FMA kernels) and now, with the split and
// the channel-last copies: layer 48 -> 16 at 104 x 56 x 56 voxels, weight
// gradient 1505 -> 275 us, data gradient 788 -> 160 us, split 49; 64 -> 64 at
// 26 x 14 x 14, 616 -> 48 and 326 -> 45 us.  Error against 64 bits over all
// layer shapes: 0.8e-7 to 3.4e-7 of the gradient's norm, 1.4e-7 to 6.5e-7
// before.  The large levels are bound by staging (about half their time is
// copies into shared memory), the small ones by too few blocks.
//
// mma.sync m16n8k16: the contraction runs over voxels with 27 shifted views
// of one operand (wgrad), or must leave the accumulator every 9 products
// (dgrad); both want the sums in registers.
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>

#include "internal.cuh"

namespace icarat_b200
{

namespace
{

typedef __nv_bfloat16 bf16;

constexpr int kTX = 16, kTY = 4, kTZ = 4, kTile = kTX * kTY * kTZ;
constexpr int kHX = kTX + 2, kHY = kTY + 2, kHZ = kTZ + 2, kHalo = kHX * kHY * kHZ;
constexpr int kRow = 32; // bytes of 16 channels

struct Vol
{
  int X, Y, Z;
  long V;
};

__device__ __forceinline__ uint32_t saddr(const void *p)
{
  return (uint32_t)__cvta_generic_to_shared(p);
}

// byte offset of 16-byte half c of row r
__device__ __forceinline__ uint32_t row_at(int r, int c)
{
  return (uint32_t)(r * kRow + ((c ^ (r >> 2)) & 1) * 16);
}

__device__ __forceinline__ void copy16(uint32_t dst, const void *src, bool valid)
{
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n)
               : "memory");
}

__device__ __forceinline__ void ldsm(uint32_t (&r)[4], uint32_t at)
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(at)
               : "memory");
}
__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], uint32_t at)
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(at)
               : "memory");
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                    uint32_t b1)
{
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, "
               "{%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// rows of a 16 x 4 x 4 tile at (x0, y0, z0), `halo` voxels around it, of the
// 16 channels at c0 of src[voxel][C]; rows outside the grid are 0
__device__ __forceinline__ void stage_tile(uint32_t dst, const bf16 *src, int C, int c0,
                                           const Vol &v, int x0, int y0, int z0, int halo)
{
  const int hx = kTX + 2 * halo, hy = kTY + 2 * halo, hz = kTZ + 2 * halo;
  for(int q = threadIdx.x; q < 2 * hx * hy * hz; q += blockDim.x)
  {
    const int r = q >> 1, c = q & 1;
    const int x = x0 - halo + r % hx, y = y0 - halo + r / hx % hy, z = z0 - halo + r / (hx * hy);
    const bool in = x >= 0 && x < v.X && y >= 0 && y < v.Y && z >= 0 && z < v.Z;
    const long n = in ? x + (long)y * v.X + (long)z * v.X * v.Y : 0;
    copy16(dst + row_at(r, c), src + n * C + c0 + 8 * c, in);
  }
}

// out[v][c] = x[c][v] for c < cin, 0 up to Cp (a multiple of 16)
__global__ void k_channel_last(long V, const bf16 *__restrict__ x, int cin, int Cp,
                               bf16 *__restrict__ out)
{
  const long v = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int c0 = 8 * blockIdx.y;
  if(v >= V)
    return;
  __align__(16) bf16 r[8];
#pragma unroll
  for(int q = 0; q < 8; q++)
    r[q] = c0 + q < cin ? x[(long)(c0 + q) * V + v] : __float2bfloat16_rn(0.0f);
  *reinterpret_cast<uint4 *>(out + v * Cp + c0) = *reinterpret_cast<const uint4 *>(r);
}

// g = dy where ymask > 0, else 0: its three BF16 parts channel-last, and each
// block's sums per channel
__global__ void __launch_bounds__(256)
    k_split(long V, const float *__restrict__ dy, const bf16 *__restrict__ ymask, int C,
            bf16 *__restrict__ hi, bf16 *__restrict__ mid, bf16 *__restrict__ lo,
            double *__restrict__ part)
{
  __shared__ double sh[8 * 32];
  const long v = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int c0 = 8 * blockIdx.y;
  __align__(16) bf16 h[8], m[8], l[8];
  double s[8];
#pragma unroll
  for(int q = 0; q < 8; q++)
  {
    float g = 0.0f;
    if(v < V)
    {
      const long id = (long)(c0 + q) * V + v;
      g = __bfloat162float(ymask[id]) > 0.0f ? dy[id] : 0.0f;
    }
    s[q] = g;
    // the top of the FP32 range rounds past BF16's: truncate there; no rest
    // of an infinity or a NaN
    const bool finite = fabsf(g) <= 3.402823466e38f;
    h[q] = fabsf(g) < 3.3e38f || !finite ? __float2bfloat16_rn(g) : __float2bfloat16_rz(g);
    const float r1 = finite ? g - __bfloat162float(h[q]) : 0.0f;
    m[q] = __float2bfloat16_rn(r1);
    l[q] = __float2bfloat16_rn(r1 - __bfloat162float(m[q]));
  }
  if(v < V)
  {
    *reinterpret_cast<uint4 *>(hi + v * C + c0) = *reinterpret_cast<const uint4 *>(h);
    *reinterpret_cast<uint4 *>(mid + v * C + c0) = *reinterpret_cast<const uint4 *>(m);
    *reinterpret_cast<uint4 *>(lo + v * C + c0) = *reinterpret_cast<const uint4 *>(l);
  }
  block_sum<8>(s, sh);
  if(threadIdx.x == 0)
#pragma unroll
    for(int q = 0; q < 8; q++)
      part[(long)blockIdx.x * C + c0 + q] = s[q];
}

// out[c] = sum of part[b][c] (fixed order), one warp per value
__global__ void k_sum_parts(int blocks, int C, const double *__restrict__ part,
                            float *__restrict__ out)
{
  const int c = blockIdx.x, lane = threadIdx.x;
  double s = 0.0;
  for(int b = lane; b < blocks; b += 32)
    s += part[(long)b * C + c];
  for(int o = 16; o > 0; o >>= 1)
    s += __shfl_down_sync(0xffffffffu, s, o);
  if(lane == 0)
    out[c] = (float)s;
}

constexpr int kWThreads = 384; // 3 dz x 4 planes of the tile
constexpr uint32_t kWStage = kHalo * kRow + 3 * kTile * kRow;

// part[split][co][ci][tap], ci < cin
__global__ void __launch_bounds__(kWThreads)
    k_wgrad_mma(Vol v, const bf16 *__restrict__ x, int cin, int Cp, const bf16 *__restrict__ hi,
                const bf16 *__restrict__ mid, const bf16 *__restrict__ lo, int cout,
                float *__restrict__ part)
{
  extern __shared__ __align__(128) unsigned char wg_raw[];
  const uint32_t base = saddr(wg_raw);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int dz = w % 3, zp = w / 3;
  const int co_tiles = cout / 16;
  const int ci0 = (int)blockIdx.y / co_tiles * 16, co0 = (int)blockIdx.y % co_tiles * 16;
  const int ntx = (v.X + kTX - 1) / kTX, nty = (v.Y + kTY - 1) / kTY, ntz = (v.Z + kTZ - 1) / kTZ;
  const int tiles = ntx * nty * ntz;
  auto stage = [&](int tile, int buf) {
    if(tile < tiles)
    {
      const int x0 = tile % ntx * kTX, y0 = tile / ntx % nty * kTY, z0 = tile / (ntx * nty) * kTZ;
      const uint32_t d = base + buf * kWStage;
      stage_tile(d, x, Cp, ci0, v, x0, y0, z0, 1);
      stage_tile(d + kHalo * kRow, hi, cout, co0, v, x0, y0, z0, 0);
      stage_tile(d + (kHalo + kTile) * kRow, mid, cout, co0, v, x0, y0, z0, 0);
      stage_tile(d + (kHalo + 2 * kTile) * kRow, lo, cout, co0, v, x0, y0, z0, 0);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  float acc[9][2][4];
#pragma unroll
  for(int k = 0; k < 9; k++)
#pragma unroll
    for(int n = 0; n < 2; n++)
#pragma unroll
      for(int q = 0; q < 4; q++)
        acc[k][n][q] = 0.0f;
  // ldmatrix rows of this lane (trans): A voxels (lane / 16, lane % 8) and
  // channel half lane / 8 % 2; B voxels lane / 8 % 2, half lane / 16
  const int ar = (lane >> 4) * 8 + (lane & 7), ac = (lane >> 3) & 1;
  const int br = ((lane >> 3) & 1) * 8 + (lane & 7), bc = lane >> 4;
  stage(blockIdx.x, 0);
  int buf = 0;
  for(int tile = blockIdx.x; tile < tiles; tile += gridDim.x, buf ^= 1)
  {
    stage(tile + gridDim.x, buf ^ 1);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    const uint32_t xs = base + buf * kWStage, ds = xs + kHalo * kRow;
#pragma unroll 1
    for(int yr = 0; yr < kTY; yr++)
    {
      uint32_t b[3][4];
#pragma unroll
      for(int p = 0; p < 3; p++)
        ldsm_t(b[p], ds + p * kTile * kRow + row_at((zp * kTY + yr) * kTX + br, bc));
#pragma unroll
      for(int dy = 0; dy < 3; dy++)
#pragma unroll
        for(int dx = 0; dx < 3; dx++)
        {
          uint32_t a[4];
          ldsm_t(a, xs + row_at(((zp + dz) * kHY + yr + dy) * kHX + dx + ar, ac));
#pragma unroll
          for(int n = 0; n < 2; n++)
          {
            float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for(int p = 2; p >= 0; p--) // low part first
              mma(d, a, b[p][2 * n], b[p][2 * n + 1]);
#pragma unroll
            for(int q = 0; q < 4; q++)
              acc[dy * 3 + dx][n][q] += d[q];
          }
        }
    }
    __syncthreads(); // the buffer is staged again by the next round
  }
  // planes 1 .. 3 join plane 0 in order
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  float *red = reinterpret_cast<float *>(wg_raw);
  for(int s = 1; s < 4; s++)
  {
    __syncthreads();
    if(zp == s)
#pragma unroll
      for(int k = 0; k < 9; k++)
#pragma unroll
        for(int n = 0; n < 2; n++)
#pragma unroll
          for(int q = 0; q < 4; q++)
            red[((dz * 72) + k * 8 + n * 4 + q) * 32 + lane] = acc[k][n][q];
    __syncthreads();
    if(zp == 0)
#pragma unroll
      for(int k = 0; k < 9; k++)
#pragma unroll
        for(int n = 0; n < 2; n++)
#pragma unroll
          for(int q = 0; q < 4; q++)
            acc[k][n][q] += red[((dz * 72) + k * 8 + n * 4 + q) * 32 + lane];
  }
  if(zp == 0)
  {
    float *out = part + (long)blockIdx.x * cout * cin * 27;
#pragma unroll
    for(int k = 0; k < 9; k++)
#pragma unroll
      for(int n = 0; n < 2; n++)
#pragma unroll
        for(int q = 0; q < 4; q++)
        {
          const int ci = ci0 + (lane >> 2) + 8 * (q >> 1);
          const int co = co0 + 8 * n + 2 * (lane & 3) + (q & 1);
          if(ci < cin)
            out[((long)co * cin + ci) * 27 + dz * 9 + k] = acc[k][n][q];
        }
  }
}

// wpk[chunk of 16 co][tap][ci][16 co] = wt[ci][co][tap] (the transposed,
// flipped weights)
__global__ void k_dgrad_pack(const bf16 *__restrict__ wt, int cin, int cout,
                             bf16 *__restrict__ wpk)
{
  const long n = (long)cin * cout * 27;
  for(long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
      i += (long)gridDim.x * blockDim.x)
  {
    const int k = (int)(i % 16), ci = (int)(i / 16 % cin);
    const int tap = (int)(i / (16L * cin) % 27), ch = (int)(i / (16L * cin * 27));
    wpk[i] = wt[((long)ci * cout + 16 * ch + k) * 27 + tap];
  }
}

constexpr int kDThreads = 256;

// dx[ci][v] = sum over co, taps of wt[ci][co][tap] g[co][v + tap]; NT n-tiles of
// 8 input channels per block
template <int NT>
__global__ void __launch_bounds__(kDThreads)
    k_dgrad_mma(Vol v, const bf16 *__restrict__ hi, const bf16 *__restrict__ mid,
                const bf16 *__restrict__ lo, int cout, const bf16 *__restrict__ wpk, int cin,
                float *__restrict__ dx)
{
  extern __shared__ __align__(128) unsigned char dg_raw[];
  const uint32_t gs = saddr(dg_raw), ws = gs + 3 * kHalo * kRow;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntx = (v.X + kTX - 1) / kTX, nty = (v.Y + kTY - 1) / kTY;
  const int x0 = (int)blockIdx.x % ntx * kTX, y0 = (int)blockIdx.x / ntx % nty * kTY,
            z0 = (int)blockIdx.x / (ntx * nty) * kTZ;
  const int ci0 = blockIdx.y * 8 * NT;
  float acc[2][NT][4];
#pragma unroll
  for(int m = 0; m < 2; m++)
#pragma unroll
    for(int n = 0; n < NT; n++)
#pragma unroll
      for(int q = 0; q < 4; q++)
        acc[m][n][q] = 0.0f;
  const int ar = lane & 15, ac = lane >> 4;
  const int br = (lane >> 4) * 8 + (lane & 7), bc = (lane >> 3) & 1;
  const bf16 *parts[3] = {hi, mid, lo};
  for(int ch = 0; ch < cout / 16; ch++)
  {
    if(ch > 0)
      __syncthreads();
#pragma unroll
    for(int p = 0; p < 3; p++)
      stage_tile(gs + p * kHalo * kRow, parts[p], cout, 16 * ch, v, x0, y0, z0, 1);
    for(int q = threadIdx.x; q < 27 * 8 * NT * 2; q += kDThreads)
    {
      const int r = q >> 1, c = q & 1; // row: tap, input channel
      const bf16 *src = wpk + (((long)ch * 27 + r / (8 * NT)) * cin + ci0 + r % (8 * NT)) * 16;
      copy16(ws + row_at(r, c), src + 8 * c, true);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
#pragma unroll 1
    for(int dzy = 0; dzy < 9; dzy++)
    {
      const int dz = dzy / 3, dy = dzy % 3;
      float d[2][NT][4];
#pragma unroll
      for(int m = 0; m < 2; m++)
#pragma unroll
        for(int n = 0; n < NT; n++)
#pragma unroll
          for(int q = 0; q < 4; q++)
            d[m][n][q] = 0.0f;
#pragma unroll
      for(int dxx = 0; dxx < 3; dxx++)
      {
        uint32_t b[NT / 2][4];
#pragma unroll
        for(int n = 0; n < NT / 2; n++)
          ldsm(b[n], ws + row_at((dzy * 3 + dxx) * 8 * NT + 16 * n + br, bc));
#pragma unroll
        for(int m = 0; m < 2; m++)
        {
          const int mt = 2 * w + m, zp = mt / kTY, yr = mt % kTY;
          const int r = ((zp + dz) * kHY + yr + dy) * kHX + dxx + ar;
#pragma unroll
          for(int p = 2; p >= 0; p--) // low part first
          {
            uint32_t a[4];
            ldsm(a, gs + p * kHalo * kRow + row_at(r, ac));
#pragma unroll
            for(int n = 0; n < NT; n++)
              mma(d[m][n], a, b[n / 2][2 * (n & 1)], b[n / 2][2 * (n & 1) + 1]);
          }
        }
      }
#pragma unroll
      for(int m = 0; m < 2; m++)
#pragma unroll
        for(int n = 0; n < NT; n++)
#pragma unroll
          for(int q = 0; q < 4; q++)
            acc[m][n][q] += d[m][n][q];
    }
  }
#pragma unroll
  for(int m = 0; m < 2; m++)
  {
    const int mt = 2 * w + m, y = y0 + mt % kTY, z = z0 + mt / kTY;
    if(y >= v.Y || z >= v.Z)
      continue;
#pragma unroll
    for(int n = 0; n < NT; n++)
#pragma unroll
      for(int q = 0; q < 4; q++)
      {
        const int x = x0 + (lane >> 2) + 8 * (q >> 1);
        const int ci = ci0 + 8 * n + 2 * (lane & 3) + (q & 1);
        if(x < v.X)
          dx[(long)ci * v.V + x + (long)y * v.X + (long)z * v.X * v.Y] = acc[m][n][q];
      }
  }
}

int vol_tiles(const Vol &v)
{
  return ((v.X + kTX - 1) / kTX) * ((v.Y + kTY - 1) / kTY) * ((v.Z + kTZ - 1) / kTZ);
}

// the kernel's shared-memory limit, raised once per device (by two threads at
// once to the same value)
typedef std::atomic<bool> OnceFlags[kMaxDevices];
template <typename K> void allow_smem(K kernel, size_t n, OnceFlags &done)
{
  std::atomic<bool> &d = done[device_slot()];
  if(!d.load())
  {
    ICK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n));
    d.store(true);
  }
}

} // namespace

void sum_parts(int blocks, int C, const double *part, float *out, cudaStream_t st)
{
  note_launch();
  k_sum_parts<<<C, 32, 0, st>>>(blocks, C, part, out);
  ICK(cudaGetLastError());
}

int conv3_split_blocks(long V) { return (int)((V + 255) / 256); }

// Voxel splits of a layer's weight gradient: about kWgradBlocks blocks over its
// channel tiles (two for each of the B200's 148 SMs), at least two tiles each.
// A constant and not the device's SM count: it fixes the order of the sums.
constexpr int kWgradBlocks = 2 * 148;
int conv3_wgrad_splits(int X, int Y, int Z, int cin, int cout)
{
  const Vol v{X, Y, Z, (long)X * Y * Z};
  const int ch = ((cin + 15) / 16) * (cout / 16), tiles = vol_tiles(v);
  return std::max(1, std::min((kWgradBlocks + ch - 1) / ch, (tiles + 1) / 2));
}

// parts of the masked gradient (three arrays of C V at g3, channel-last) and
// the bias gradient
void conv3_split(long V, const float *dy, const uint16_t *ymask, int C, uint16_t *g3,
                 double *part, float *db, cudaStream_t st)
{
  const int blocks = conv3_split_blocks(V);
  bf16 *g = reinterpret_cast<bf16 *>(g3);
  note_launch();
  k_split<<<dim3(blocks, C / 8), 256, 0, st>>>(V, dy, reinterpret_cast<const bf16 *>(ymask), C, g,
                                               g + C * V, g + 2 * C * V, part);
  ICK(cudaGetLastError());
  sum_parts(blocks, C, part, db, st);
}

// part[split][cout][cin][27] of the weight gradient; xcl: scratch of V times
// cin rounded up to 16
void conv3_wgrad(int X, int Y, int Z, const uint16_t *x, int cin, const uint16_t *g3, int cout,
                 uint16_t *xcl, float *part, int splits, cudaStream_t st)
{
  const Vol v{X, Y, Z, (long)X * Y * Z};
  const int Cp = (cin + 15) / 16 * 16;
  static OnceFlags done;
  allow_smem(k_wgrad_mma, 2 * kWStage, done);
  const bf16 *g = reinterpret_cast<const bf16 *>(g3);
  note_launch(2);
  k_channel_last<<<dim3((unsigned)((v.V + 255) / 256), Cp / 8), 256, 0, st>>>(
      v.V, reinterpret_cast<const bf16 *>(x), cin, Cp, reinterpret_cast<bf16 *>(xcl));
  k_wgrad_mma<<<dim3(splits, Cp / 16 * (cout / 16)), kWThreads, 2 * kWStage, st>>>(
      v, reinterpret_cast<const bf16 *>(xcl), cin, Cp, g, g + cout * v.V, g + 2 * cout * v.V, cout,
      part);
  ICK(cudaGetLastError());
}

void conv3_dgrad_pack(const uint16_t *wt, int cin, int cout, uint16_t *wpk, cudaStream_t st)
{
  const long n = (long)cin * cout * 27;
  note_launch();
  k_dgrad_pack<<<(unsigned)std::min(1024L, (n + 255) / 256), 256, 0, st>>>(
      reinterpret_cast<const bf16 *>(wt), cin, cout, reinterpret_cast<bf16 *>(wpk));
  ICK(cudaGetLastError());
}

// the data gradient (cin a multiple of 16) from the parts of the gradient
void conv3_dgrad(int X, int Y, int Z, const uint16_t *g3, int cout, const uint16_t *wpk, int cin,
                 float *dx, cudaStream_t st)
{
  IREQUIRE(cin % 16 == 0 && cout % 16 == 0, ICARAT_ERR_ARG,
           "the data gradient needs channels in steps of 16");
  const Vol v{X, Y, Z, (long)X * Y * Z};
  const bf16 *g = reinterpret_cast<const bf16 *>(g3);
  const bf16 *wp = reinterpret_cast<const bf16 *>(wpk);
  auto launch = [&](auto kernel, int nt, OnceFlags &done) {
    const size_t smem = 3 * kHalo * kRow + 27 * 8 * (size_t)nt * kRow;
    allow_smem(kernel, smem, done);
    note_launch();
    kernel<<<dim3(vol_tiles(v), cin / (8 * nt)), kDThreads, smem, st>>>(
        v, g, g + cout * v.V, g + 2 * cout * v.V, cout, wp, cin, dx);
  };
  static OnceFlags done2, done4;
  if(cin % 32 == 0)
    launch(k_dgrad_mma<4>, 4, done4);
  else
    launch(k_dgrad_mma<2>, 2, done2);
  ICK(cudaGetLastError());
}

} // namespace icarat_b200
