// Learned block preconditioner: a small 3D U-Net over one 8^3 pressure block
// plus a one-cell halo, trained on the GPU with these kernels.
//
// The reference has no learned solver; this is a build-only component. The
// network (channels 16/32/64, 3x3x3 convolutions, ReLU, 2x average pooling,
// nearest upsampling with 1x1 reductions and additive skips, 141,937
// parameters) is:
//   e1a = relu(conv3(x, 2->16, valid))        10^3 -> 8^3
//   s1  = relu(conv3(e1a, 16->16))            8^3
//   e2a = relu(conv3(pool(s1), 16->32))       4^3
//   s2  = relu(conv3(e2a, 32->32))            4^3
//   bt  = relu(conv3(pool(s2), 32->64))       2^3
//   u2  = relu(up(conv1(bt, 64->32)) + s2)    4^3
//   d2  = relu(conv3(u2, 32->32))
//   u1  = relu(up(conv1(d2, 32->16)) + s1)    8^3
//   d1  = relu(conv3(u1, 16->16))
//   y   = conv1(d1, 16->1)                    8^3
// conv1(up(x)) is evaluated as up(conv1(x)) (identical for a pointwise linear
// map and nearest upsampling). Parameters are FP32, flattened layer by layer as
// weight [Cout][Cin][27 taps (dz,dy,dx)] then bias [Cout]. Training activations
// are FP32 [batch][channel][z][y][x]. Every reduction (weight gradients, loss)
// runs in a fixed order, so a training step is bitwise reproducible.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "../../include/fluidity_b200.h"
#include "fl_internal.cuh"
#include "fl_kernels.h"
#include "fl_unet.h"

namespace fl {
namespace {

constexpr int kT = 256;

// ---------------------------------------------------------------- forward

// The FP32 3x3x3 convolutions, forward and data gradient. Both are
//   out[b][o][cell] = f(sum_i sum_tap W[o][i][tap] in[b][i][cell + tap - 1]),
// the data gradient with i over the layer's output channels and
// W[o][i][tap] = w[i][o][26 - tap]. Bound by latency: at 45 items an SM holds 8 to 16
// warps, which issue in 30-36% of cycles and wait for what they stage first. A
// thread owns four x-adjacent cells and kCo output channels, so one input row (a
// 16- and an 8-byte shared load) serves 3 taps x 4 cells x kCo channels in packed
// FMAs (channel pairs). A training step of 45 items takes 392 us; with one output per
// thread and an input and a weight load per FMA it took 1821, with one group of 128
// threads per CTA here and at most one CTA per SM in the weight gradients 629, with
// one stream and plain launches 549.
// One CTA per item, slab of kZ output planes and 16 output channels, two groups
// of 128 threads each taking half of the input channels; the slab's zero-padded
// input (rows padded to a multiple of four words, planes so that the eight lanes of
// a 16-byte access touch all banks) and the 16 channels' weights ([input
// channel][tap][channel]) are staged in shared memory. Sums run over input
// channels, then taps in ascending order.
template <int S>
struct ConvTile {
  static constexpr int kZ = S == 8 ? 2 : 4;   // output planes per CTA
  static constexpr int kCo = S == 8 ? 4 : 2;  // output channels per thread
  static constexpr int kRow = S == 8 ? 12 : 8;
  static constexpr int kPlane = S == 8 ? 10 * 12 : 6 * 8 + 4;
  static constexpr int kChannel = (kZ + 2) * kPlane;
  // (at least what the exchange of the two groups' sums needs)
  static constexpr size_t smem(int cin) {
    const size_t staged = sizeof(float) * cin * (kChannel + 27 * kConvW), sums = sizeof(float) * 128 * 4 * kCo;
    return staged > sums ? staged : sums;
  }
  static constexpr int kConvW = 20;  // words per (channel, tap): 16 weights, padded against store conflicts
};

constexpr int kConvThreads = 256;

template <int S, bool VALID, bool DATA>
__global__ void __launch_bounds__(kConvThreads) k_conv3(const float* __restrict__ in, int cin, const float* __restrict__ w,
                                               const float* __restrict__ bias, int cout, float* __restrict__ out,
                                               int relu, const float* __restrict__ act) {
  grid_dependency_wait(in, w, bias, act);
  using T = ConvTile<S>;
  constexpr int E = S + 2, S3 = S * S * S, EIN = VALID ? E : S, EIN3 = EIN * EIN * EIN, OFF = VALID ? 0 : 1;
  constexpr int kSlabs = S / T::kZ, kCells = (T::kZ + 2) * E * E;
  extern __shared__ __align__(16) float conv_smem[];
  float* tile = conv_smem;
  float* wt = tile + cin * T::kChannel;
  const int t = threadIdx.x, lane = t & 31, warp = (t >> 5) & 3, half = t >> 7;
  const int b = blockIdx.x / kSlabs, z0 = (blockIdx.x % kSlabs) * T::kZ, co0 = blockIdx.y * 16;
  const float* src = in + (size_t)b * cin * EIN3;
#pragma unroll 4
  for (int i = t; i < cin * kCells; i += kConvThreads) {
    const int ci = i / kCells, r = i % kCells;
    const int pz = r / (E * E), py = (r / E) % E, px = r % E;
    const int z = z0 + pz - OFF, y = py - OFF, x = px - OFF;
    float v = 0.0f;
    if (VALID || (z >= 0 && z < S && y >= 0 && y < S && x >= 0 && x < S)) v = src[ci * EIN3 + (z * EIN + y) * EIN + x];
    tile[ci * T::kChannel + pz * T::kPlane + py * T::kRow + px] = v;
  }
  if (DATA) {  // in channel i = a layer output, the 16 layer inputs co0 .. co0 + 15 contiguous in w[i]
#pragma unroll 4
    for (int e = t; e < cin * 16 * 27; e += kConvThreads) {
      const int i = e / (16 * 27), r = e % (16 * 27), o = r / 27, tap = r % 27;
      wt[(i * 27 + 26 - tap) * T::kConvW + o] = w[((size_t)i * cout + co0 + o) * 27 + tap];
    }
  } else {
#pragma unroll 4
    for (int e = t; e < 16 * cin * 27; e += kConvThreads) {
      const int o = e / (cin * 27), r = e % (cin * 27);
      wt[r * T::kConvW + o] = w[(size_t)(co0 + o) * cin * 27 + r];
    }
  }
  __syncthreads();
  // S = 8: lanes (y, x half, z), warp = channel quad; S = 4: lanes (y, z, channel pair of the warp's quad)
  const int y = S == 8 ? lane & 7 : lane & 3, z = S == 8 ? lane >> 4 : (lane >> 2) & 3;
  const int x0 = S == 8 ? 4 * ((lane >> 3) & 1) : 0;
  const int co = 4 * warp + (S == 8 ? 0 : 2 * (lane >> 4));
  float2 acc[4][T::kCo / 2];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int h = 0; h < T::kCo / 2; ++h)
      acc[c][h] = DATA || half != 0
                      ? make_float2(0.0f, 0.0f)
                      : make_float2(__ldg(&bias[co0 + co + 2 * h]), __ldg(&bias[co0 + co + 2 * h + 1]));
  for (int ci = half * (cin / 2); ci < (half + 1) * (cin / 2); ++ci) {
    const float* base = tile + ci * T::kChannel + z * T::kPlane + y * T::kRow + x0;
    const float* wc = wt + ci * 27 * T::kConvW + co;
#pragma unroll
    for (int dz = 0; dz < 3; ++dz)
#pragma unroll
      for (int dy = 0; dy < 3; ++dy) {
        const float4 a = *reinterpret_cast<const float4*>(base + dz * T::kPlane + dy * T::kRow);
        const float2 e = *reinterpret_cast<const float2*>(base + dz * T::kPlane + dy * T::kRow + 4);
        const float v[6] = {a.x, a.y, a.z, a.w, e.x, e.y};
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
          const float* wp = wc + ((dz * 3 + dy) * 3 + dx) * T::kConvW;
          float2 wv[T::kCo / 2];
          if constexpr (T::kCo == 4) {
            const float4 q = *reinterpret_cast<const float4*>(wp);
            wv[0] = make_float2(q.x, q.y);
            wv[1] = make_float2(q.z, q.w);
          } else {
            wv[0] = *reinterpret_cast<const float2*>(wp);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = 0; h < T::kCo / 2; ++h)
              acc[c][h] = __ffma2_rn(make_float2(v[c + dx], v[c + dx]), wv[h], acc[c][h]);
        }
      }
  }
  // the second group's sums, added by the first (through the tile's shared memory)
  __syncthreads();
  float2* other = reinterpret_cast<float2*>(tile) + (t & 127);
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int h = 0; h < T::kCo / 2; ++h)
      if (half != 0) other[(c * (T::kCo / 2) + h) * 128] = acc[c][h];
  __syncthreads();
  if (half != 0) return;
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int h = 0; h < T::kCo / 2; ++h) acc[c][h] = __fadd2_rn(acc[c][h], other[(c * (T::kCo / 2) + h) * 128]);
#pragma unroll
  for (int k = 0; k < T::kCo; ++k) {
    const size_t o = ((size_t)b * cout + co0 + co + k) * S3 + ((z0 + z) * S + y) * S + x0;
    float r[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) r[c] = (k & 1) ? acc[c][k >> 1].y : acc[c][k >> 1].x;
    if (DATA && act != nullptr) {
      const float4 m = *reinterpret_cast<const float4*>(act + o);
      r[0] = m.x > 0.0f ? r[0] : 0.0f;
      r[1] = m.y > 0.0f ? r[1] : 0.0f;
      r[2] = m.z > 0.0f ? r[2] : 0.0f;
      r[3] = m.w > 0.0f ? r[3] : 0.0f;
    } else if (!DATA && relu) {
#pragma unroll
      for (int c = 0; c < 4; ++c) r[c] = fmaxf(r[c], 0.0f);
    }
    *reinterpret_cast<float4*>(out + o) = make_float4(r[0], r[1], r[2], r[3]);
  }
}

// The 2^3 layer: an output cell sees all eight input cells, each through one
// tap, so only 8 of its 27 taps are formed. Lanes hold 32 items, a warp one
// (z, y) row of two cells and four output channels: the weights of a tap are
// then one broadcast 16-byte load for the warp. One CTA of 8 warps per 32 items
// and 8 output channels.
constexpr int kConv2Items = 33;  // words per (channel, cell): 32 items, padded
constexpr int kConv2W = 12;      // words per (channel, tap): 8 weights, padded
constexpr size_t conv2_smem(int cin) { return sizeof(float) * cin * (8 * kConv2Items + 27 * kConv2W); }

template <bool DATA>
__global__ void __launch_bounds__(256) k_conv3_2(const float* __restrict__ in, int cin, const float* __restrict__ w,
                                                 const float* __restrict__ bias, int cout, int batch,
                                                 float* __restrict__ out, int relu, const float* __restrict__ act) {
  grid_dependency_wait(in, w, bias, act);
  extern __shared__ __align__(16) float conv_smem[];
  float* wt = conv_smem;
  float* tile = wt + cin * 27 * kConv2W;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int b0 = blockIdx.x * 32, co0 = blockIdx.y * 8;
  const int items = min(32, batch - b0);
  for (int e = t; e < 32 * cin * 8; e += 256) {
    const int b = e / (cin * 8), r = e % (cin * 8);
    tile[r * kConv2Items + b] = b < items ? in[(size_t)(b0 + b) * cin * 8 + r] : 0.0f;
  }
  for (int e = t; e < cin * 8 * 27; e += 256) {
    if (DATA) {
      const int i = e / (8 * 27), r = e % (8 * 27), o = r / 27, tap = r % 27;
      wt[(i * 27 + 26 - tap) * kConv2W + o] = w[((size_t)i * cout + co0 + o) * 27 + tap];
    } else {
      const int o = e / (cin * 27), r = e % (cin * 27);
      wt[r * kConv2W + o] = w[(size_t)(co0 + o) * cin * 27 + r];
    }
  }
  __syncthreads();
  const int z = (warp >> 1) & 1, y = warp & 1, co = 4 * (warp >> 2);
  float2 acc[2][2];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      acc[c][h] = DATA ? make_float2(0.0f, 0.0f)
                       : make_float2(__ldg(&bias[co0 + co + 2 * h]), __ldg(&bias[co0 + co + 2 * h + 1]));
  for (int ci = 0; ci < cin; ++ci) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {  // input row (z', y'): taps z' - z + 1 and y' - y + 1
      const int tap = ((r >> 1) - z + 1) * 9 + ((r & 1) - y + 1) * 3;
      const float* v = tile + (ci * 8 + 2 * r) * kConv2Items + lane;
      const float2 v0 = make_float2(v[0], v[0]), v1 = make_float2(v[kConv2Items], v[kConv2Items]);
      const float* wp = wt + (ci * 27 + tap) * kConv2W + co;
      float2 wv[3][2];
#pragma unroll
      for (int dx = 0; dx < 3; ++dx) {
        const float4 q = *reinterpret_cast<const float4*>(wp + dx * kConv2W);
        wv[dx][0] = make_float2(q.x, q.y);
        wv[dx][1] = make_float2(q.z, q.w);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        acc[0][h] = __ffma2_rn(v1, wv[2][h], __ffma2_rn(v0, wv[1][h], acc[0][h]));
        acc[1][h] = __ffma2_rn(v1, wv[1][h], __ffma2_rn(v0, wv[0][h], acc[1][h]));
      }
    }
  }
  if (lane >= items) return;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const size_t o = ((size_t)(b0 + lane) * cout + co0 + co + k) * 8 + z * 4 + y * 2;
    float r[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      r[c] = (k & 1) ? acc[c][k >> 1].y : acc[c][k >> 1].x;
      if (DATA && act != nullptr && !(act[o + c] > 0.0f)) r[c] = 0.0f;
      if (!DATA && relu) r[c] = fmaxf(r[c], 0.0f);
    }
    *reinterpret_cast<float2*>(out + o) = make_float2(r[0], r[1]);
  }
}

// out[b][co][cell] = bias[co] + sum_ci w[co][ci] in[b][ci][cell].
__global__ void k_conv1_fwd(const float* __restrict__ in, int cin, const float* __restrict__ w,
                            const float* __restrict__ bias, int cout, int s3, long long total,
                            float* __restrict__ out) {
  grid_dependency_wait(in, w, bias);
  for (long long i = blockIdx.x * (long long)kT + threadIdx.x; i < total; i += (long long)gridDim.x * kT) {
    const int cell = (int)(i % s3);
    const int co = (int)((i / s3) % cout);
    const long long b = i / ((long long)s3 * cout);
    float acc = bias[co];
    const float* src = in + (size_t)b * cin * s3 + cell;
    for (int ci = 0; ci < cin; ++ci) acc = fmaf(__ldg(&w[co * cin + ci]), src[(size_t)ci * s3], acc);
    out[i] = acc;
  }
}

// 2x average pooling: out [B][C][(S/2)^3] from in [B][C][S^3].
__global__ void k_pool(const float* __restrict__ in, int S, long long total, float* __restrict__ out) {
  grid_dependency_wait(in);
  const int H = S / 2, H3 = H * H * H, S3 = S * S * S;
  for (long long i = blockIdx.x * (long long)kT + threadIdx.x; i < total; i += (long long)gridDim.x * kT) {
    const int c = (int)(i % H3);
    const long long bc = i / H3;
    const int z = c / (H * H), y = (c / H) % H, x = c % H;
    const float* src = in + bc * S3 + ((2 * z) * S + 2 * y) * S + 2 * x;
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += src[((k >> 2) * S + ((k >> 1) & 1)) * S + (k & 1)];
    out[i] = s * 0.125f;
  }
}

// out = relu(up(conv1(in)) + skip): a thread forms one output channel of one of the
// H^3 coarse cells and adds it to the cell's eight children at resolution 2H, which
// are loaded first. Bound by its launch and one round trip; as two kernels with the
// coarse sums between them a training step took 302 us instead of 299 (64 items,
// tensor cores) and 408 instead of 404 (45, FP32).
__global__ void k_up_conv1_relu(const float* __restrict__ in, int cin, const float* __restrict__ w,
                                const float* __restrict__ bias, const float* __restrict__ skip, int cout, int H,
                                long long total, float* __restrict__ out) {
  grid_dependency_wait(in, w, bias, skip);
  const int S = 2 * H, H3 = H * H * H;
  for (long long i = blockIdx.x * (long long)kT + threadIdx.x; i < total; i += (long long)gridDim.x * kT) {
    const int cell = (int)(i % H3), co = (int)((i / H3) % cout);
    const long long b = i / ((long long)H3 * cout);
    const int x = cell % H, y = (cell / H) % H, z = cell / (H * H);
    const long long fine = (b * cout + co) * 8 * H3 + ((long long)(2 * z) * S + 2 * y) * S + 2 * x;
    float2 child[4];  // pairs along x
#pragma unroll
    for (int k = 0; k < 4; ++k)
      child[k] = *reinterpret_cast<const float2*>(skip + fine + (k >> 1) * S * S + (k & 1) * S);
    float acc = bias[co];
    const float* src = in + (size_t)b * cin * H3 + cell;
#pragma unroll 8
    for (int ci = 0; ci < cin; ++ci) acc = fmaf(__ldg(&w[co * cin + ci]), src[(size_t)ci * H3], acc);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      *reinterpret_cast<float2*>(out + fine + (k >> 1) * S * S + (k & 1) * S) =
          make_float2(fmaxf(acc + child[k].x, 0.0f), fmaxf(acc + child[k].y, 0.0f));
  }
}

// ---------------------------------------------------------------- backward

// Weight and bias gradient of a 3x3x3 layer:
//   dw[co][ci][tap] = sum_b sum_o g[b][co][o] in[b][ci][o + tap - pad], db[co] = sum_b sum_o g[b][co][o].
// A thread owns one input channel, one (dz, dy) and eight output channels: per
// cell one input value (three kept for the dx taps) and two broadcast 16-byte
// loads of g (staged [cell][channel]) feed 12 packed FMAs.
// Work units (an item's slab of two planes at 8^3, an item at 4^3, four items
// at 2^3) are dealt to gridDim.x CTAs in order and each CTA writes one partial
// row; k_wgrad_sum adds the rows in order, so the result is reproducible.
// With two input channels (the first layer) kSplit threads share a role, each
// taking every kSplit-th row of cells into a partial row of its own.
template <int S, bool VALID, int CIN>
struct WgradTile {
  static constexpr int kSplit = CIN == 2 ? 8 : 1;
  static constexpr int kThreads = CIN * 18 * kSplit;  // channels x 9 x 2 octets of output channels
  static constexpr int kZ = S == 8 ? 2 : S;
  static constexpr int kItems = S == 2 ? 4 : 1;
  static constexpr int kSlabs = S / kZ;
  static constexpr int kCh = CIN + 1;                                 // words per cell: odd or whole-warp reads
  static constexpr int kRow = (S + 2) * kCh + (CIN == 16 && S == 8 ? 6 : 0);  // 16 mod 32: half-warps on two rows
  static constexpr int kPlane = (S + 2) * kRow + (CIN == 16 && S == 8 ? 16 : 0);
  static constexpr int kItem = (kZ + 2) * kPlane;
  static constexpr int kG = 20;  // words per cell of g: 16 channels, padded
  static constexpr size_t kSmem = sizeof(float) * (kItems * (kItem + kZ * S * S * kG) + 4);
};

template <int S, bool VALID, int CIN>
__global__ void __launch_bounds__(WgradTile<S, VALID, CIN>::kThreads)
    k_conv3_wgrad(const float* __restrict__ in, const float* __restrict__ g, int cout, int batch, int units,
                  float* __restrict__ part) {
  grid_dependency_wait(in, g);
  using T = WgradTile<S, VALID, CIN>;
  constexpr int E = S + 2, S3 = S * S * S, EIN = VALID ? E : S, EIN3 = EIN * EIN * EIN, OFF = VALID ? 0 : 1;
  constexpr int kInCells = (T::kZ + 2) * E * E, kOutCells = T::kZ * S * S;
  extern __shared__ __align__(16) float wg_smem[];
  float* gt = wg_smem;                                // [item][cell][16, padded]
  float* it = gt + T::kItems * kOutCells * T::kG;     // [item][z][y][x][channel]
  const int t = threadIdx.x, co0 = blockIdx.y * 16;
  const int ci = t % CIN, rest = t / CIN, dzy = rest % 9, oct = (rest / 9) & 1, split = rest / 18;
  const int dz = dzy / 3, dy = dzy % 3;
  float2 acc[3][4], bsum[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    bsum[h] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int dx = 0; dx < 3; ++dx) acc[dx][h] = make_float2(0.0f, 0.0f);
  }
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    const int b0 = u / T::kSlabs * T::kItems, z0 = (u % T::kSlabs) * T::kZ;
    __syncthreads();  // the previous unit's reads
    for (int i = t; i < T::kItems * CIN * kInCells; i += T::kThreads) {
      const int k = i / (CIN * kInCells), r = i % (CIN * kInCells), c = r / kInCells, cell = r % kInCells;
      const int pz = cell / (E * E), py = (cell / E) % E, px = cell % E;
      const int z = z0 + pz - OFF, y = py - OFF, x = px - OFF;
      float v = 0.0f;
      if (b0 + k < batch && (VALID || (z >= 0 && z < S && y >= 0 && y < S && x >= 0 && x < S)))
        v = in[((size_t)(b0 + k) * CIN + c) * EIN3 + (z * EIN + y) * EIN + x];
      it[k * T::kItem + pz * T::kPlane + py * T::kRow + px * T::kCh + c] = v;
    }
    for (int i = t; i < T::kItems * 16 * kOutCells; i += T::kThreads) {
      const int k = i / (16 * kOutCells), r = i % (16 * kOutCells), o = r / kOutCells, cell = r % kOutCells;
      gt[(k * kOutCells + cell) * T::kG + o] =
          b0 + k < batch ? g[((size_t)(b0 + k) * cout + co0 + o) * S3 + z0 * S * S + cell] : 0.0f;
    }
    __syncthreads();
    for (int row = split; row < T::kItems * T::kZ * S; row += T::kSplit) {
      const int k = row / (T::kZ * S), z = (row / S) % T::kZ, y = row % S;
      const float* v = it + k * T::kItem + (z + dz) * T::kPlane + (y + dy) * T::kRow + ci;
      const float* gp = gt + (size_t)row * S * T::kG + 8 * oct;
      float v0 = v[0], v1 = v[T::kCh];
#pragma unroll
      for (int x = 0; x < S; ++x) {
        const float v2 = v[(x + 2) * T::kCh];
        const float4 ga = *reinterpret_cast<const float4*>(gp + x * T::kG);
        const float4 gb = *reinterpret_cast<const float4*>(gp + x * T::kG + 4);
        const float2 gv[4] = {make_float2(ga.x, ga.y), make_float2(ga.z, ga.w), make_float2(gb.x, gb.y),
                              make_float2(gb.z, gb.w)};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          acc[0][h] = __ffma2_rn(make_float2(v0, v0), gv[h], acc[0][h]);
          acc[1][h] = __ffma2_rn(make_float2(v1, v1), gv[h], acc[1][h]);
          acc[2][h] = __ffma2_rn(make_float2(v2, v2), gv[h], acc[2][h]);
          if (dzy == 0) bsum[h] = __fadd2_rn(bsum[h], gv[h]);
        }
        v0 = v1;
        v1 = v2;
      }
    }
  }
  const int nw = cout * CIN * 27;
  float* row = part + ((size_t)blockIdx.x * T::kSplit + split) * (nw + cout);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int o = co0 + 8 * oct + k;
#pragma unroll
    for (int dx = 0; dx < 3; ++dx)
      row[((size_t)o * CIN + ci) * 27 + dzy * 3 + dx] = (k & 1) ? acc[dx][k >> 1].y : acc[dx][k >> 1].x;
    if (dzy == 0 && ci == 0) row[nw + o] = (k & 1) ? bsum[k >> 1].y : bsum[k >> 1].x;
  }
}

// dw, db = the partial rows added in order: 32 values per CTA, eight warps taking
// every eighth row, then the eight sums in order.
__global__ void __launch_bounds__(kT) k_wgrad_sum(const float* __restrict__ part, int rows, int nw, int cout,
                                                  float* __restrict__ dw, float* __restrict__ db) {
  grid_dependency_wait(part);
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + lane, n = nw + cout;
  float s = 0.0f;
  if (e < n) {
#pragma unroll 8
    for (int r = warp; r < rows; r += 8) s += part[(size_t)r * n + e];
  }
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && e < n) {
    float v = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) v += red[k][lane];
    if (e < nw)
      dw[e] = v;
    else
      db[e - nw] = v;
  }
}

// dw[co][ci] = sum g[b][co][o] in[b][ci][o]; db[co] likewise (ci == 0 CTA). One CTA of NT
// threads per (ci, co): 1024 for the output layer, whose 16 CTAs each reduce a whole plane.
template <int NT>
__global__ void __launch_bounds__(NT) k_conv1_bwd_weight(const float* __restrict__ in, int cin,
                                                         const float* __restrict__ g, int cout, int s3, int batch,
                                                         float* __restrict__ dw, float* __restrict__ db) {
  grid_dependency_wait(in, g);
  __shared__ float red[2 * (NT / 32)];
  const int ci = blockIdx.x, co = blockIdx.y;
  float a = 0.0f, bs = 0.0f;
  for (int idx = threadIdx.x; idx < batch * s3; idx += NT) {
    const int b = idx / s3, o = idx % s3;
    const float gv = g[((size_t)b * cout + co) * s3 + o];
    a = fmaf(gv, in[((size_t)b * cin + ci) * s3 + o], a);
    bs += gv;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    bs += __shfl_xor_sync(0xffffffffu, bs, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5] = a;
    red[NT / 32 + (threadIdx.x >> 5)] = bs;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.0f, t = 0.0f;
    for (int k = 0; k < NT / 32; ++k) {
      s += red[k];
      t += red[NT / 32 + k];
    }
    dw[co * cin + ci] = s;
    if (ci == 0) db[co] = t;
  }
}

// din[b][ci][o] = (sum_co w[co][ci] g[b][co][o]) * (act > 0).
__global__ void k_conv1_bwd_data(const float* __restrict__ g, int cout, const float* __restrict__ w, int cin, int s3,
                                 long long total, const float* __restrict__ act, float* __restrict__ din) {
  grid_dependency_wait(g, w, act);
  for (long long i = blockIdx.x * (long long)kT + threadIdx.x; i < total; i += (long long)gridDim.x * kT) {
    const int o = (int)(i % s3);
    const int ci = (int)((i / s3) % cin);
    const long long b = i / ((long long)s3 * cin);
    float acc = 0.0f;
    if (act == nullptr || act[i] > 0.0f) {
      const float* src = g + (size_t)b * cout * s3 + o;
      for (int co = 0; co < cout; ++co) acc = fmaf(__ldg(&w[co * cin + ci]), src[(size_t)co * s3], acc);
    }
    din[i] = acc;
  }
}

// out[b][c][coarse] = sum of the 8 children of g at resolution S.
__global__ void k_up_back(const float* __restrict__ g, int S, long long total, float* __restrict__ out) {
  grid_dependency_wait(g);
  const int H = S / 2, H3 = H * H * H, S3 = S * S * S;
  for (long long i = blockIdx.x * (long long)kT + threadIdx.x; i < total; i += (long long)gridDim.x * kT) {
    const int c = (int)(i % H3);
    const long long bc = i / H3;
    const int z = c / (H * H), y = (c / H) % H, x = c % H;
    const float* src = g + bc * S3 + ((2 * z) * S + 2 * y) * S + 2 * x;
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += src[((k >> 2) * S + ((k >> 1) & 1)) * S + (k & 1)];
    out[i] = s;
  }
}

// out = (ga + gp[parent] / 8) * (act > 0) at resolution S.
__global__ void k_pool_back_add_mask(const float* __restrict__ ga, const float* __restrict__ gp,
                                     const float* __restrict__ act, int S, long long total, float* __restrict__ out) {
  grid_dependency_wait(ga, gp, act);
  const int H = S / 2, S3 = S * S * S, H3 = H * H * H;
  for (long long i = blockIdx.x * (long long)kT + threadIdx.x; i < total; i += (long long)gridDim.x * kT) {
    const int c = (int)(i % S3);
    const long long bc = i / S3;
    const int z = c / (S * S), y = (c / S) % S, x = c % S;
    const float v = ga[i] + 0.125f * gp[bc * H3 + ((z >> 1) * H + (y >> 1)) * H + (x >> 1)];
    out[i] = act[i] > 0.0f ? v : 0.0f;
  }
}

// Masked squared error in one CTA (fixed order). relative == 0:
//   loss = sum m (y - t)^2 / max(1, sum m), grad = 2 m (y - t) / max(1, sum m);
// relative == 1 (every item weighs the same whatever its scale):
//   loss = (1/V) sum_items [sum m (y - t)^2 / sum m t^2] over the V items with
//   sum m t^2 > 0 (items without target energy add nothing), grad likewise.
__global__ void __launch_bounds__(1024) k_masked_mse(const float* __restrict__ y, const float* __restrict__ t,
                                                     const float* __restrict__ m, int batch, int relative,
                                                     float* __restrict__ loss, float* __restrict__ grad) {
  __shared__ double red[2 * 32];
  __shared__ double item_den[1024];
  const int n = batch * 512;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  // per-item denominators (one warp per item, items in order)
  for (int b = warp; b < batch; b += nwarps) {
    double s = 0.0, c = 0.0;
    for (int k = lane; k < 512; k += 32) {
      const double tv = t[b * 512 + k];
      s += m[b * 512 + k] * tv * tv;
      c += m[b * 512 + k];
    }
    s = warp_sum(s);
    c = warp_sum(c);
    if (lane == 0) item_den[b] = relative ? s : c;
  }
  __syncthreads();
  double global_den = 0.0;
  int valid = 0;
  for (int b = 0; b < batch; ++b) {
    global_den += item_den[b];
    valid += item_den[b] > 0.0;
  }
  global_den = global_den > 1.0 ? global_den : 1.0;
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int b = i >> 9;
    const double den = relative ? item_den[b] * valid : global_den;
    const double d = (double)y[i] - (double)t[i];
    const double w = relative && !(item_den[b] > 0.0) ? 0.0 : m[i] / den;
    acc += w * d * d;
    if (grad) grad[i] = (float)(2.0 * w * d);
  }
  acc = warp_sum(acc);
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0 && loss) {
    double total = 0.0;
    for (int k = 0; k < nwarps; ++k) total += red[k];
    *loss = (float)total;
  }
}

// Block-residual loss. For item b the input window holds r / s (channel 0) and the
// cell mask (channel 1: fluid 1, air 0, solid -1) on the block plus a one-cell
// halo; y is the network's correction on the block's 8^3 cells. With A_b the
// level-0 pressure operator restricted to the block's fluid cells (unit
// conductance to fluid and air neighbours, none to solid ones, the block's
// neighbours held at zero):
//   rho = r_b - A_b y,  loss = (1/V) sum_items |rho|^2 / D_b,
//   d loss / d y = -(2 / (V D_b)) A_b rho   (A_b is symmetric),
// with D_b = max(|r_b|^2, 1) (the window is scaled to max |r| = 1, so a block
// whose residual is mostly in its halo does not weigh more than the rest),
// over the V items whose block holds residual. The zero correction scores at
// most 1; a network that inverts A_b on its block scores 0.
//
// Bound by latency: an item is 12 KB. One cluster of 8 CTAs x 16 warps, four warps
// per item (four cells per thread, a barrier of their own), so 32 items are in
// flight at once; V and the loss are summed over the cluster through distributed
// shared memory in item order, so no scratch memory and no second launch is
// needed and the call stays bitwise reproducible. One item takes 15 us, 64 16 and
// 1024 114; with a warp per item 23, 25 and 131, with a CTA per item 15, 26 and
// 260, and with one CTA taking all items in turn 12, 210 and 3230.
constexpr int kLossCtas = 8, kLossWarps = 16, kLossItemWarps = 4, kLossMaxItems = 1024;
constexpr int kLossFlags = 1024;  // bytes: 1000 window flags, padded
constexpr size_t kLossItemBytes = kLossFlags + sizeof(float) * 512;

__global__ void __cluster_dims__(kLossCtas, 1, 1) __launch_bounds__(kLossWarps * 32)
    k_block_residual_loss(const float* __restrict__ y, const float* __restrict__ x, int batch,
                          float* __restrict__ loss, float* __restrict__ grad) {
  constexpr int kMine = kLossMaxItems / kLossCtas;
  constexpr int kGroups = kLossWarps / kLossItemWarps, kThreads = 32 * kLossItemWarps, kCells = 512 / kThreads;
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ double den[kMine], num[kMine];
  __shared__ double parts[kLossWarps];
  __shared__ int valid_cta;
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = warp / kLossItemWarps, t = threadIdx.x % kThreads;  // the item's warps, the thread among theirs
  unsigned char* flag = dyn + group * kLossItemBytes;  // bit 0 fluid, bit 1 not solid
  float* vec = reinterpret_cast<float*>(flag + kLossFlags);
  if (threadIdx.x == 0) valid_cta = 0;
  for (int k = threadIdx.x; k < kMine; k += kLossWarps * 32) num[k] = 0.0;
  __syncthreads();
  auto sync = [&] { asm volatile("barrier.sync %0, %1;" ::"r"(1 + group), "n"(kThreads) : "memory"); };
  // over the item's threads, the warps' sums in order (parts may be written again after the next sync)
  auto item_sum = [&](double v) {
    v = warp_sum(v);
    if (lane == 0) parts[warp] = v;
    sync();
    v = parts[group * kLossItemWarps];
#pragma unroll
    for (int w = 1; w < kLossItemWarps; ++w) v += parts[group * kLossItemWarps + w];
    return v;
  };
  auto window = [](int l) { return ((l >> 6) + 1) * 100 + (((l >> 3) & 7) + 1) * 10 + (l & 7) + 1; };
  // pass 1: |r_b|^2 per item and the number of items with residual (item b: CTA b % 8, slot b / 8)
  for (int slot = group; slot * kLossCtas + rank < batch; slot += kGroups) {
    const float* xb = x + (size_t)(slot * kLossCtas + rank) * 2000;
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
      const int w = window(t + kThreads * k);
      const float m = xb[1000 + w], r = xb[w];
      if (m == 1.0f) v += (double)r * (double)r;
    }
    v = item_sum(v);
    if (t == 0) {
      den[slot] = v;
      if (v > 0.0) atomicAdd(&valid_cta, 1);
    }
    sync();  // the next item's sum overwrites the parts
  }
  cluster.sync();
  int valid = 0;
#pragma unroll
  for (int c = 0; c < kLossCtas; ++c) valid += *cluster.map_shared_rank(&valid_cta, c);
  // pass 2: residual after the correction, the loss and its gradient
  for (int slot = group; slot * kLossCtas + rank < batch; slot += kGroups) {
    const size_t b = (size_t)slot * kLossCtas + rank;
    const float* xb = x + b * 2000;
    float yv[kCells], rv[kCells];
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
      yv[k] = y[b * 512 + t + kThreads * k];
      rv[k] = xb[window(t + kThreads * k)];
    }
#pragma unroll 8
    for (int k = 0; k < 2 * kCells; ++k) {
      const int i = t + kThreads * k;
      if (i < 1000) {
        const float m = xb[1000 + i];
        flag[i] = (unsigned char)((m == 1.0f ? 1 : 0) | (m >= 0.0f ? 2 : 0));
      }
    }
    sync();
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
      const int l = t + kThreads * k;
      if (!(flag[window(l)] & 1)) yv[k] = 0.0f;
      vec[l] = yv[k];
    }
    sync();
    const int dw[6] = {-1, 1, -10, 10, -100, 100}, dl[6] = {-1, 1, -8, 8, -64, 64};
    // the sum of the block's fluid neighbours of cell l and (diag) its open faces
    auto neighbours = [&](int l, float* diag) {
      const int w = window(l), c[3] = {l & 7, (l >> 3) & 7, l >> 6};
      float off = 0.0f, d = 0.0f;
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const unsigned f = flag[w + dw[q]];
        d += (f & 2) ? 1.0f : 0.0f;
        const bool in = (q & 1) ? c[q >> 1] < 7 : c[q >> 1] > 0;
        if (in && (f & 1)) off += vec[l + dl[q]];
      }
      *diag = d;
      return off;
    };
    float rho[kCells], dg[kCells];
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
      const int l = t + kThreads * k;
      const float off = neighbours(l, &dg[k]);
      rho[k] = (flag[window(l)] & 1) ? rv[k] - (dg[k] * yv[k] - off) : 0.0f;
    }
    sync();
#pragma unroll
    for (int k = 0; k < kCells; ++k) vec[t + kThreads * k] = rho[k];
    sync();
    const double d = den[slot];
    const double scale = d > 0.0 ? 1.0 / (valid * fmax(d, 1.0)) : 0.0;
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
      const int l = t + kThreads * k;
      acc += scale * (double)rho[k] * (double)rho[k];
      if (grad != nullptr) {
        float arho = 0.0f;
        if (flag[window(l)] & 1) {
          float dd;
          const float off = neighbours(l, &dd);
          arho = dg[k] * rho[k] - off;
        }
        grad[b * 512 + l] = (float)(-2.0 * scale * (double)arho);
      }
    }
    acc = item_sum(acc);
    if (t == 0) num[slot] = acc;
    sync();  // the next item overwrites flag and vec
  }
  cluster.sync();
  if (rank == 0 && warp == 0 && loss != nullptr) {
    double total = 0.0;
    for (int b = lane; b < batch; b += 32) total += cluster.map_shared_rank(num, b % kLossCtas)[b / kLossCtas];
    total = warp_sum(total);
    if (lane == 0) *loss = (float)total;
  }
  cluster.sync();  // the other CTAs' shared memory is read until here
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, long long n, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
  for (long long i = blockIdx.x * (long long)kT + threadIdx.x; i < n; i += (long long)gridDim.x * kT) {
    const float gi = g[i];
    const float mi = fmaf(b1, m[i], (1.0f - b1) * gi);
    const float vi = fmaf(b2, v[i], (1.0f - b2) * gi * gi);
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// He-uniform weights from a counter-based SplitMix64 stream, zero biases.
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void k_init_params(float* p, UNetLayout L, unsigned long long seed) {
  const long long n = L.total;
  for (long long i = blockIdx.x * (long long)kT + threadIdx.x; i < n; i += (long long)gridDim.x * kT) {
    int l = 0;
    while (l + 1 < kUNetLayers && i >= L.offset[l + 1]) ++l;
    const long long local = i - L.offset[l];
    const long long nw = (long long)L.cout[l] * L.cin[l] * L.taps[l];
    if (local >= nw) {
      p[i] = 0.0f;
      continue;
    }
    const float bound = sqrtf(6.0f / (float)(L.cin[l] * L.taps[l]));
    const unsigned long long r = splitmix64(seed * 0x100000001B3ull + (unsigned long long)i);
    const float u = (float)((r >> 40) * (1.0 / 16777216.0));  // [0, 1)
    p[i] = (2.0f * u - 1.0f) * bound;
  }
}

unsigned grid_for(long long n) {
  long long b = (n + kT - 1) / kT;
  return (unsigned)(b < 1 ? 1 : (b > 4096 ? 4096 : b));
}

template <int S, bool VALID>
void conv3_fwd(const float* in, int cin, const float* w, const float* bias, int cout, float* out, int batch, int relu,
               cudaStream_t s) {
  ++g_kernel_launches;
  if constexpr (S == 2)
    launch_dep(k_conv3_2<false>, dim3((batch + 31) / 32, cout / 8), 256, conv2_smem(cin), s, in, cin, w, bias, cout,
               batch, out, relu, nullptr);
  else
    launch_dep(k_conv3<S, VALID, false>, dim3(batch * (S / ConvTile<S>::kZ), cout / 16), kConvThreads,
               ConvTile<S>::smem(cin), s, in, cin, w, bias, cout, out, relu, nullptr);
}

// g has the layer's cout channels, din its cin: the roles of k_conv3's cin and cout.
template <int S>
void conv3_bwd_data(const float* g, int cout, const float* w, int cin, const float* act, float* din, int batch,
                    cudaStream_t s) {
  ++g_kernel_launches;
  if constexpr (S == 2)
    launch_dep(k_conv3_2<true>, dim3((batch + 31) / 32, cin / 8), 256, conv2_smem(cout), s, g, cout, w, nullptr, cin,
               batch, din, 0, act);
  else
    launch_dep(k_conv3<S, false, true>, dim3(batch * (S / ConvTile<S>::kZ), cin / 16), kConvThreads,
               ConvTile<S>::smem(cout), s, g, cout, w, nullptr, cin, din, 0, act);
}

template <int S, bool VALID, int CIN>
void wgrad(const float* in, const float* g, int cout, int batch, float* part, float* dw, float* db, cudaStream_t s) {
  using T = WgradTile<S, VALID, CIN>;
  const int nw = cout * CIN * 27;
  const int units = (batch + T::kItems - 1) / T::kItems * T::kSlabs;
  // two CTAs per SM where the units and the partial rows' space allow it
  const int ctas = (int)std::min<long long>({(long long)units, 2 * 148, kWgradPart / ((long long)T::kSplit * (nw + cout))});
  ++g_kernel_launches;
  launch_dep(k_conv3_wgrad<S, VALID, CIN>, dim3(ctas, cout / 16), T::kThreads, T::kSmem, s, in, g, cout, batch, units,
             part);
  wgrad_sum(part, ctas * T::kSplit, nw, cout, dw, db, s);
}

// The network's layers: 2 input channels (first layer) or 16 at 8^3, 16 or 32 at 4^3, 32 at 2^3.
template <int S, bool VALID>
void conv3_bwd_weight(const float* in, int cin, const float* g, int cout, int batch, float* part, float* dw, float* db,
                      cudaStream_t s) {
  if constexpr (VALID)
    wgrad<S, true, 2>(in, g, cout, batch, part, dw, db, s);
  else if constexpr (S == 8)
    wgrad<S, false, 16>(in, g, cout, batch, part, dw, db, s);
  else if (S == 4 && cin == 16)
    wgrad<S, false, 16>(in, g, cout, batch, part, dw, db, s);
  else
    wgrad<S, false, 32>(in, g, cout, batch, part, dw, db, s);
}

// A 3x3x3 layer in the FP32 kernels (tc == nullptr) or on the tensor cores;
// the first tensor-core failure is kept in `e` and the remaining layers skip.
template <int S, bool VALID>
void fwd3(UNetTcTrain* tc, cudaError_t& e, int layer, const float* in, int cin, const float* w, const float* bias,
          int cout, float* out, int batch, int relu, cudaStream_t s) {
  if (tc == nullptr) return conv3_fwd<S, VALID>(in, cin, w, bias, cout, out, batch, relu, s);
  if (e == cudaSuccess) e = conv3_fwd_tc(*tc, layer, in, bias, out, batch, s);
}
template <int S>
void bwd3_data(UNetTcTrain* tc, cudaError_t& e, int layer, const float* g, int cout, const float* w, int cin,
               const float* act, float* din, int batch, cudaStream_t s) {
  if (tc == nullptr) return conv3_bwd_data<S>(g, cout, w, cin, act, din, batch, s);
  if (e == cudaSuccess) e = conv3_bwd_data_tc(*tc, layer, g, act, din, batch, s);
}
template <int S, bool VALID>
void bwd3_weight(UNetTcTrain* tc, cudaError_t& e, int layer, const float* in, int cin, const float* g, int cout,
                 int batch, float* part, float* dw, float* db, cudaStream_t s) {
  if (tc == nullptr) return conv3_bwd_weight<S, VALID>(in, cin, g, cout, batch, part, dw, db, s);
  if (e == cudaSuccess) e = conv3_bwd_weight_tc(layer, in, g, batch, part, dw, db, s);
}

}  // namespace

void wgrad_sum(const float* part, int rows, int nw, int cout, float* dw, float* db, cudaStream_t s) {
  ++g_kernel_launches;
  launch_dep(k_wgrad_sum, (nw + cout + 31) / 32, kT, 0, s, part, rows, nw, cout, dw, db);
}

UNetLayout unet_layout() {
  static const int kCin[kUNetLayers] = {2, 16, 16, 32, 32, 64, 32, 32, 16, 16};
  static const int kCout[kUNetLayers] = {16, 16, 32, 32, 64, 32, 32, 16, 16, 1};
  static const int kTaps[kUNetLayers] = {27, 27, 27, 27, 27, 1, 27, 1, 27, 1};
  UNetLayout L{};
  long long off = 0;
  for (int l = 0; l < kUNetLayers; ++l) {
    L.cin[l] = kCin[l];
    L.cout[l] = kCout[l];
    L.taps[l] = kTaps[l];
    L.offset[l] = off;
    L.bias[l] = off + (long long)kCout[l] * kCin[l] * kTaps[l];
    off = L.bias[l] + kCout[l];
  }
  L.total = off;
  return L;
}

UNetCache unet_cache_layout(int batch) {
  UNetCache C{};
  long long off = 0;
  auto take = [&](long long per_item) {
    const long long o = off;
    off += per_item * batch;
    return o;
  };
  C.x = take(2 * 1000);
  C.e1a = take(16 * 512);
  C.s1 = take(16 * 512);
  C.p1 = take(16 * 64);
  C.e2a = take(32 * 64);
  C.s2 = take(32 * 64);
  C.p2 = take(32 * 8);
  C.bt = take(64 * 8);
  C.u2 = take(32 * 64);
  C.d2 = take(32 * 64);
  C.u1 = take(16 * 512);
  C.d1 = take(16 * 512);
  C.y = take(512);
  C.activations = off;
  // backward scratch
  C.g8a = take(16 * 512);
  C.g8b = take(16 * 512);
  C.g8c = take(16 * 512);
  C.g4a = take(32 * 64);
  C.g4b = take(32 * 64);
  C.g4c = take(32 * 64);
  C.g2a = take(64 * 8);
  C.g2b = take(64 * 8);
  off = (off + 3) / 4 * 4;
  C.part = off;  // partial rows of the weight gradients
  off += kWgradPart;
  C.total = off;
  return C;
}

void configure_unet_kernels() {
  static OncePerDevice configured;
  once_on_device(configured, [] {
    auto allow = [](auto* kernel, size_t bytes) {
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    allow(k_conv3<8, true, false>, ConvTile<8>::smem(2));
    allow(k_conv3<8, false, false>, ConvTile<8>::smem(16));
    allow(k_conv3<8, false, true>, ConvTile<8>::smem(16));
    allow(k_conv3<4, false, false>, ConvTile<4>::smem(32));
    allow(k_conv3<4, false, true>, ConvTile<4>::smem(32));
    allow(k_conv3_2<false>, conv2_smem(32));
    allow(k_conv3_2<true>, conv2_smem(64));
    allow(k_conv3_wgrad<8, true, 2>, WgradTile<8, true, 2>::kSmem);
    allow(k_conv3_wgrad<8, false, 16>, WgradTile<8, false, 16>::kSmem);
    allow(k_conv3_wgrad<4, false, 16>, WgradTile<4, false, 16>::kSmem);
    allow(k_conv3_wgrad<4, false, 32>, WgradTile<4, false, 32>::kSmem);
    allow(k_conv3_wgrad<2, false, 32>, WgradTile<2, false, 32>::kSmem);
  });
}

// Forward pass of `batch` items; every activation is kept in `cache` (layout unet_cache_layout).
cudaError_t unet_forward(const float* P, const float* x, int batch, float* cache, float* y, cudaStream_t s,
                         UNetTcTrain* tc) {
  configure_unet_kernels();
  const UNetLayout L = unet_layout();
  const UNetCache C = unet_cache_layout(batch);
  float* A = cache;
  const long long B = batch;
  if (x != A + C.x) cudaMemcpyAsync(A + C.x, x, sizeof(float) * 2000 * B, cudaMemcpyDeviceToDevice, s);
  auto W = [&](int l) { return P + L.offset[l]; };
  auto Bi = [&](int l) { return P + L.bias[l]; };
  cudaError_t tce = tc != nullptr ? unet_tc_train_pack(*tc, P, false, s) : cudaSuccess;
  fwd3<8, true>(tc, tce, 0, A + C.x, 2, W(0), Bi(0), 16, A + C.e1a, batch, 1, s);
  fwd3<8, false>(tc, tce, 1, A + C.e1a, 16, W(1), Bi(1), 16, A + C.s1, batch, 1, s);
  g_kernel_launches += 1;
  launch_dep(k_pool, grid_for(B * 16 * 64), kT, 0, s, A + C.s1, 8, B * 16 * 64, A + C.p1);
  fwd3<4, false>(tc, tce, 2, A + C.p1, 16, W(2), Bi(2), 32, A + C.e2a, batch, 1, s);
  fwd3<4, false>(tc, tce, 3, A + C.e2a, 32, W(3), Bi(3), 32, A + C.s2, batch, 1, s);
  g_kernel_launches += 1;
  launch_dep(k_pool, grid_for(B * 32 * 8), kT, 0, s, A + C.s2, 4, B * 32 * 8, A + C.p2);
  fwd3<2, false>(tc, tce, 4, A + C.p2, 32, W(4), Bi(4), 64, A + C.bt, batch, 1, s);
  g_kernel_launches += 3;
  launch_dep(k_up_conv1_relu, grid_for(B * 32 * 8), kT, 0, s, A + C.bt, 64, W(5), Bi(5), A + C.s2, 32, 2, B * 32 * 8,
             A + C.u2);
  fwd3<4, false>(tc, tce, 6, A + C.u2, 32, W(6), Bi(6), 32, A + C.d2, batch, 1, s);
  launch_dep(k_up_conv1_relu, grid_for(B * 16 * 64), kT, 0, s, A + C.d2, 32, W(7), Bi(7), A + C.s1, 16, 4, B * 16 * 64,
             A + C.u1);
  fwd3<8, false>(tc, tce, 8, A + C.u1, 16, W(8), Bi(8), 16, A + C.d1, batch, 1, s);
  launch_dep(k_conv1_fwd, grid_for(B * 512), kT, 0, s, A + C.d1, 16, W(9), Bi(9), 1, 512, B * 512, A + C.y);
  if (y != nullptr && y != A + C.y)
    cudaMemcpyAsync(y, A + C.y, sizeof(float) * 512 * B, cudaMemcpyDeviceToDevice, s);
  if (tce != cudaSuccess) return tce;
  return cudaGetLastError();
}

cudaError_t unet_side_create(UNetSide* side) {
  cudaError_t e = cudaStreamCreateWithFlags(&side->s, cudaStreamNonBlocking);
  cudaEvent_t* events[] = {&side->fork[0], &side->fork[1], &side->fork[2], &side->fork[3],
                           &side->fork[4], &side->fork[5], &side->read,    &side->join};
  for (cudaEvent_t* v : events)
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(v, cudaEventDisableTiming);
  if (e != cudaSuccess) unet_side_destroy(side);
  return e;
}

void unet_side_destroy(UNetSide* side) {
  for (cudaEvent_t v : side->fork)
    if (v != nullptr) cudaEventDestroy(v);
  if (side->read != nullptr) cudaEventDestroy(side->read);
  if (side->join != nullptr) cudaEventDestroy(side->join);
  if (side->s != nullptr) cudaStreamDestroy(side->s);
  *side = UNetSide{};
}

// Gradient of sum(gy * y) with respect to the parameters, from the cache of the last forward.
// A layer's kernels fill a part of the chip at training batches, and the weight gradients
// (over half of the time) feed nothing: they run on the side stream, each forked off once
// its output gradient is there, beside the chain of data gradients on `s`; `s` joins them
// at the end. The chain reuses the first half's gradient buffers only after the side
// stream has read them (`read`). A training step of 64 items on the tensor cores 335 ->
// 301 us, of 45 in FP32 448 -> 407.
cudaError_t unet_backward(const float* P, float* cache, const float* gy, int batch, float* G, cudaStream_t s,
                          const UNetSide& side, UNetTcTrain* tc) {
  configure_unet_kernels();
  cudaError_t tce = tc != nullptr ? unet_tc_train_pack(*tc, P, true, s) : cudaSuccess;
  const UNetLayout L = unet_layout();
  const UNetCache C = unet_cache_layout(batch);
  float* A = cache;
  const long long B = batch;
  auto W = [&](int l) { return P + L.offset[l]; };
  auto GW = [&](int l) { return G + L.offset[l]; };
  auto GB = [&](int l) { return G + L.bias[l]; };
  const cudaStream_t w = side.s;
  auto fork = [&](int k) {  // the side stream goes on from here
    cudaEventRecord(side.fork[k], s);
    cudaStreamWaitEvent(w, side.fork[k], 0);
  };
  // out layer (16 -> 1)
  g_kernel_launches += 2;
  launch_dep(k_conv1_bwd_data, grid_for(B * 16 * 512), kT, 0, s, gy, 1, W(9), 16, 512, B * 16 * 512, A + C.d1,
             A + C.g8a);
  fork(0);
  launch_dep(k_conv1_bwd_weight<1024>, dim3(16, 1), 1024, 0, w, A + C.d1, 16, gy, 1, 512, batch, GW(9), GB(9));
  // d1 (conv3 16->16 on u1); gu1 pre-activation -> g8b
  bwd3_weight<8, false>(tc, tce, 8, A + C.u1, 16, A + C.g8a, 16, batch, A + C.part, GW(8), GB(8), w);
  bwd3_data<8>(tc, tce, 8, A + C.g8a, 16, W(8), 16, A + C.u1, A + C.g8b, batch, s);
  // u1 = relu(up(conv1(d2, 32->16)) + s1)
  g_kernel_launches += 3;
  launch_dep(k_up_back, grid_for(B * 16 * 64), kT, 0, s, A + C.g8b, 8, B * 16 * 64, A + C.g4c);
  launch_dep(k_conv1_bwd_data, grid_for(B * 32 * 64), kT, 0, s, A + C.g4c, 16, W(7), 32, 64, B * 32 * 64, A + C.d2,
             A + C.g4a);
  fork(1);
  launch_dep(k_conv1_bwd_weight<kT>, dim3(32, 16), kT, 0, w, A + C.d2, 32, A + C.g4c, 16, 64, batch, GW(7), GB(7));
  // d2 (conv3 32->32 on u2); gu2 pre-activation -> g4b
  bwd3_weight<4, false>(tc, tce, 6, A + C.u2, 32, A + C.g4a, 32, batch, A + C.part, GW(6), GB(6), w);
  bwd3_data<4>(tc, tce, 6, A + C.g4a, 32, W(6), 32, A + C.u2, A + C.g4b, batch, s);
  // u2 = relu(up(conv1(bt, 64->32)) + s2)
  g_kernel_launches += 3;
  launch_dep(k_up_back, grid_for(B * 32 * 8), kT, 0, s, A + C.g4b, 4, B * 32 * 8, A + C.g2b);
  launch_dep(k_conv1_bwd_data, grid_for(B * 64 * 8), kT, 0, s, A + C.g2b, 32, W(5), 64, 8, B * 64 * 8, A + C.bt,
             A + C.g2a);
  fork(2);
  launch_dep(k_conv1_bwd_weight<kT>, dim3(64, 32), kT, 0, w, A + C.bt, 64, A + C.g2b, 32, 8, batch, GW(5), GB(5));
  cudaEventRecord(side.read, w);
  // bt (conv3 32->64 on p2) -> gp2 (g2b, 32 channels)
  bwd3_weight<2, false>(tc, tce, 4, A + C.p2, 32, A + C.g2a, 64, batch, A + C.part, GW(4), GB(4), w);
  cudaStreamWaitEvent(s, side.read, 0);  // g2b, g4c, g4a and g8a are written again from here
  bwd3_data<2>(tc, tce, 4, A + C.g2a, 64, W(4), 32, nullptr, A + C.g2b, batch, s);
  // s2 gradient: (gu2 + pool_back(gp2)) * (s2 > 0) -> g4a
  g_kernel_launches += 1;
  launch_dep(k_pool_back_add_mask, grid_for(B * 32 * 64), kT, 0, s, A + C.g4b, A + C.g2b, A + C.s2, 4, B * 32 * 64,
             A + C.g4a);
  // e2b (conv3 32->32 on e2a) -> ge2a (g4c)
  bwd3_data<4>(tc, tce, 3, A + C.g4a, 32, W(3), 32, A + C.e2a, A + C.g4c, batch, s);
  fork(3);
  bwd3_weight<4, false>(tc, tce, 3, A + C.e2a, 32, A + C.g4a, 32, batch, A + C.part, GW(3), GB(3), w);
  // e2a (conv3 16->32 on p1) -> gp1 (g4b, 16 channels)
  bwd3_weight<4, false>(tc, tce, 2, A + C.p1, 16, A + C.g4c, 32, batch, A + C.part, GW(2), GB(2), w);
  bwd3_data<4>(tc, tce, 2, A + C.g4c, 32, W(2), 16, nullptr, A + C.g4b, batch, s);
  // s1 gradient: (gu1 + pool_back(gp1)) * (s1 > 0) -> g8a
  g_kernel_launches += 1;
  launch_dep(k_pool_back_add_mask, grid_for(B * 16 * 512), kT, 0, s, A + C.g8b, A + C.g4b, A + C.s1, 8, B * 16 * 512,
             A + C.g8a);
  // e1b (conv3 16->16 on e1a) -> ge1a (g8c)
  fork(4);
  bwd3_weight<8, false>(tc, tce, 1, A + C.e1a, 16, A + C.g8a, 16, batch, A + C.part, GW(1), GB(1), w);
  bwd3_data<8>(tc, tce, 1, A + C.g8a, 16, W(1), 16, A + C.e1a, A + C.g8c, batch, s);
  // e1a (valid conv3 2->16 on x)
  fork(5);
  bwd3_weight<8, true>(tc, tce, 0, A + C.x, 2, A + C.g8c, 16, batch, A + C.part, GW(0), GB(0), w);
  cudaEventRecord(side.join, w);
  cudaStreamWaitEvent(s, side.join, 0);
  if (tce != cudaSuccess) return tce;
  return cudaGetLastError();
}

cudaError_t unet_masked_mse(const float* y, const float* t, const float* m, int batch, int relative, float* loss,
                            float* grad, cudaStream_t s) {
  ++g_kernel_launches;
  k_masked_mse<<<1, 1024, 0, s>>>(y, t, m, batch, relative, loss, grad);
  return cudaGetLastError();
}

cudaError_t unet_block_residual_loss(const float* y, const float* x, int batch, float* loss, float* grad,
                                     cudaStream_t s) {
  ++g_kernel_launches;
  constexpr size_t smem = kLossWarps / kLossItemWarps * kLossItemBytes;  // 12 KB
  k_block_residual_loss<<<kLossCtas, kLossWarps * 32, smem, s>>>(y, x, batch, loss, grad);
  return cudaGetLastError();
}

cudaError_t adam_step(float* p, const float* g, float* m, float* v, long long n, int step, float lr, float b1,
                      float b2, float eps, cudaStream_t s) {
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  ++g_kernel_launches;
  k_adam<<<grid_for(n), kT, 0, s>>>(p, g, m, v, n, lr, b1, b2, eps, c1, c2);
  return cudaGetLastError();
}

cudaError_t unet_init_params(float* p, unsigned long long seed, cudaStream_t s) {
  const UNetLayout L = unet_layout();
  ++g_kernel_launches;
  k_init_params<<<grid_for(L.total), kT, 0, s>>>(p, L, seed);
  return cudaGetLastError();
}


// ---------------------------------------------------------------- solver <-> network

namespace {

// Input item of block b: its 8^3 cells plus a one-cell halo (10^3, z-major),
// channel 0 = residual / s, channel 1 = cell mask (fluid 1, air 0, solid -1),
// s = max |residual| over the window (0 -> all-zero input). Missing blocks
// read as air (inactive, inside the lattice) or solid (outside it).
__global__ void __launch_bounds__(512) k_unet_gather(GridView g, const float* __restrict__ r_rb,
                                                     const unsigned char* __restrict__ type,
                                                     const int* __restrict__ blocks, float* __restrict__ inputs,
                                                     float* __restrict__ scale) {
  __shared__ float red[16];
  const int item = blockIdx.x;
  const int b = blocks ? blocks[item] : item;
  float rv[2], mv[2], mx = 0.0f;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int i = threadIdx.x + 512 * k;
    rv[k] = 0.0f;
    mv[k] = 0.0f;
    if (i < 1000) {
      const int hz = i / 100 - 1, hy = (i / 10) % 10 - 1, hx = i % 10 - 1;
      const int ox = hx < 0 ? -1 : (hx > 7 ? 1 : 0), oy = hy < 0 ? -1 : (hy > 7 ? 1 : 0),
                oz = hz < 0 ? -1 : (hz > 7 ? 1 : 0);
      const int nb = (ox | oy | oz) ? g.nbr27[b * 27 + nbr_index(ox, oy, oz)] : b;
      if (nb >= 0) {
        const int l = ((hz - 8 * oz) * 8 + (hy - 8 * oy)) * 8 + (hx - 8 * ox);
        rv[k] = r_rb[nb * 512 + rb_of(l)];
        const int t = type[nb * 512 + l];
        mv[k] = t == 1 ? 1.0f : (t == 0 ? -1.0f : 0.0f);
      } else {
        mv[k] = nb == -1 ? 0.0f : -1.0f;
      }
      mx = fmaxf(mx, fabsf(rv[k]));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  float sc = 0.0f;
#pragma unroll
  for (int k = 0; k < 16; ++k) sc = fmaxf(sc, red[k]);
  float* out = inputs + (size_t)item * 2000;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int i = threadIdx.x + 512 * k;
    if (i < 1000) {
      out[i] = sc > 0.0f ? rv[k] / sc : 0.0f;
      out[1000 + i] = mv[k];
    }
  }
  if (threadIdx.x == 0) scale[item] = sc;
}

// Target item: (p_star - p_k) / s on fluid cells (natural order), mask = fluid.
__global__ void __launch_bounds__(512) k_unet_targets(GridView g, const double* __restrict__ p_star,
                                                      const double* __restrict__ p_k,
                                                      const unsigned char* __restrict__ type,
                                                      const int* __restrict__ blocks, const float* __restrict__ scale,
                                                      float* __restrict__ targets, float* __restrict__ masks) {
  const int item = blockIdx.x, l = threadIdx.x;
  const int b = blocks ? blocks[item] : item;
  const bool fluid = type[b * 512 + l] == 1;
  const float sc = scale[item];
  const int i = b * 512 + rb_of(l);
  targets[(size_t)item * 512 + l] = fluid && sc > 0.0f ? (float)((p_star[i] - p_k[i]) / (double)sc) : 0.0f;
  masks[(size_t)item * 512 + l] = fluid ? 1.0f : 0.0f;
}

// z = s * y on fluid cells, 0 elsewhere; RB: level-0 solver layout, else natural.
template <typename T, bool RB>
__global__ void __launch_bounds__(512) k_unet_scatter(int nb, const float* __restrict__ y,
                                                      const float* __restrict__ scale,
                                                      const unsigned char* __restrict__ type, T* __restrict__ z) {
  const int b = blockIdx.x, l = threadIdx.x;
  const float v = type[b * 512 + l] == 1 ? scale[b] * y[(size_t)b * 512 + l] : 0.0f;
  st_T(&z[b * 512 + (RB ? rb_of(l) : l)], v);
}

__global__ void __launch_bounds__(512) k_block_has_fluid(const unsigned char* __restrict__ type, int* flags) {
  const int b = blockIdx.x;
  const int any = __syncthreads_or(type[b * 512 + threadIdx.x] == 1);
  if (threadIdx.x == 0) flags[b] = any;
}

}  // namespace

cudaError_t unet_gather(const GridView& g, const float* r_rb, const unsigned char* type, const int* blocks, int count,
                        float* inputs, float* scale, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  ++g_kernel_launches;
  k_unet_gather<<<count, 512, 0, s>>>(g, r_rb, type, blocks, inputs, scale);
  return cudaGetLastError();
}

cudaError_t unet_targets(const GridView& g, const double* p_star, const double* p_k, const unsigned char* type,
                         const int* blocks, int count, const float* scale, float* targets, float* masks,
                         cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  ++g_kernel_launches;
  k_unet_targets<<<count, 512, 0, s>>>(g, p_star, p_k, type, blocks, scale, targets, masks);
  return cudaGetLastError();
}

template <typename T>
cudaError_t unet_scatter(int nb, const float* y, const float* scale, const unsigned char* type, T* z, bool rb,
                         cudaStream_t s) {
  if (nb <= 0) return cudaSuccess;
  ++g_kernel_launches;
  if (rb)
    k_unet_scatter<T, true><<<nb, 512, 0, s>>>(nb, y, scale, type, z);
  else
    k_unet_scatter<T, false><<<nb, 512, 0, s>>>(nb, y, scale, type, z);
  return cudaGetLastError();
}
template cudaError_t unet_scatter<float>(int, const float*, const float*, const unsigned char*, float*, bool,
                                         cudaStream_t);
template cudaError_t unet_scatter<__nv_bfloat16>(int, const float*, const float*, const unsigned char*,
                                                 __nv_bfloat16*, bool, cudaStream_t);

cudaError_t unet_block_has_fluid(int nb, const unsigned char* type, int* flags, cudaStream_t s) {
  if (nb <= 0) return cudaSuccess;
  ++g_kernel_launches;
  k_block_has_fluid<<<nb, 512, 0, s>>>(type, flags);
  return cudaGetLastError();
}

}  // namespace fl

// ---------------------------------------------------------------- C-ABI

struct fl_unet {
  int device = 0;
  int max_batch = 0;
  float* cache = nullptr;
  fl::UNetSide side;
  fl::UNetTcTrain* tc = nullptr;  // set: the 3x3x3 training convolutions run on the tensor cores
};

namespace {
int unet_code(cudaError_t e) {
  if (e == cudaSuccess) return FL_OK;
  cudaGetLastError();
  return FL_INTERNAL;
}

int unet_device_ready() {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
    cudaGetLastError();
    return FL_FAILED_PRECONDITION;
  }
  return FL_OK;
}
}  // namespace

extern "C" {

int64_t fl_unet_param_count(void) { return fl::unet_layout().total; }

int fl_unet_create(int max_batch, fl_unet** out) {
  if (out == nullptr || max_batch <= 0 || max_batch > (1 << 16)) return FL_INVALID_ARGUMENT;
  *out = nullptr;
  int st = unet_device_ready();
  if (st != FL_OK) return st;
  fl_unet* u = new fl_unet();
  cudaGetDevice(&u->device);
  u->max_batch = max_batch;
  const size_t bytes = sizeof(float) * (size_t)fl::unet_cache_layout(max_batch).total;
  if (cudaMalloc(&u->cache, bytes) != cudaSuccess) {
    cudaGetLastError();
    delete u;
    return FL_RESOURCE_EXHAUSTED;
  }
  if (fl::unet_side_create(&u->side) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(u->cache);
    delete u;
    return FL_RESOURCE_EXHAUSTED;
  }
  cudaMemset(u->cache, 0, bytes);
  *out = u;
  return FL_OK;
}

int fl_unet_destroy(fl_unet* u) {
  if (u == nullptr) return FL_OK;
  if (u->tc != nullptr) {
    fl::unet_tc_train_destroy(u->tc);
    delete u->tc;
  }
  cudaFree(u->cache);
  fl::unet_side_destroy(&u->side);
  delete u;
  return FL_OK;
}

int fl_unet_set_tensor_cores(fl_unet* u, int enable) {
  if (u == nullptr || (enable != 0 && enable != 1)) return FL_INVALID_ARGUMENT;
  if (!enable) {
    if (u->tc != nullptr) {
      fl::unet_tc_train_destroy(u->tc);
      delete u->tc;
      u->tc = nullptr;
    }
    return FL_OK;
  }
  if (u->tc != nullptr) return FL_OK;
  if (u->max_batch > fl::kUNetTcMaxBatch) return FL_OUT_OF_RANGE;
  int st = fl::check_device();
  if (st != FL_OK) return st;
  auto* t = new fl::UNetTcTrain();
  if (fl::unet_tc_train_create(t) != cudaSuccess) {
    cudaGetLastError();
    delete t;
    return FL_RESOURCE_EXHAUSTED;
  }
  u->tc = t;
  return FL_OK;
}

int fl_unet_init_params(float* params, uint64_t seed, void* stream) {
  if (params == nullptr) return FL_INVALID_ARGUMENT;
  int st = unet_device_ready();
  if (st != FL_OK) return st;
  return unet_code(fl::unet_init_params(params, seed, static_cast<cudaStream_t>(stream)));
}

int fl_unet_forward(fl_unet* u, const float* params, const float* input, int batch, float* output, void* stream) {
  if (u == nullptr || params == nullptr || input == nullptr || batch < 0) return FL_INVALID_ARGUMENT;
  if (batch > u->max_batch) return FL_RESOURCE_EXHAUSTED;
  if (batch == 0) return FL_OK;
  return unet_code(
      fl::unet_forward(params, input, batch, u->cache, output, static_cast<cudaStream_t>(stream), u->tc));
}

int fl_unet_backward(fl_unet* u, const float* params, const float* grad_output, int batch, float* grad_params,
                     void* stream) {
  if (u == nullptr || params == nullptr || grad_output == nullptr || grad_params == nullptr || batch <= 0)
    return FL_INVALID_ARGUMENT;
  if (batch > u->max_batch) return FL_RESOURCE_EXHAUSTED;
  return unet_code(fl::unet_backward(params, u->cache, grad_output, batch, grad_params,
                                     static_cast<cudaStream_t>(stream), u->side, u->tc));
}

int fl_unet_masked_mse(const float* output, const float* target, const float* mask, int batch, int relative,
                       float* loss, float* grad_output, void* stream) {
  if (output == nullptr || target == nullptr || mask == nullptr || batch <= 0 || batch > 1024 ||
      (relative != 0 && relative != 1))
    return FL_INVALID_ARGUMENT;
  return unet_code(fl::unet_masked_mse(output, target, mask, batch, relative, loss, grad_output,
                                       static_cast<cudaStream_t>(stream)));
}

int fl_unet_block_residual_loss(const float* output, const float* input, int batch, float* loss, float* grad_output,
                                void* stream) {
  if (output == nullptr || input == nullptr || batch <= 0 || batch > 1024) return FL_INVALID_ARGUMENT;
  return unet_code(fl::unet_block_residual_loss(output, input, batch, loss, grad_output,
                                                static_cast<cudaStream_t>(stream)));
}

int fl_adam_step(float* params, const float* grads, float* m, float* v, uint64_t count, int step, float lr,
                 float beta1, float beta2, float eps, void* stream) {
  if (params == nullptr || grads == nullptr || m == nullptr || v == nullptr || step < 1 || !(lr > 0.0f) ||
      !(beta1 >= 0.0f && beta1 < 1.0f) || !(beta2 >= 0.0f && beta2 < 1.0f) || !(eps > 0.0f))
    return FL_INVALID_ARGUMENT;
  if (count == 0) return FL_OK;
  return unet_code(fl::adam_step(params, grads, m, v, (long long)count, step, lr, beta1, beta2, eps,
                                 static_cast<cudaStream_t>(stream)));
}

}  // extern "C"
