// Training convolutions of the learned preconditioner on tensor cores.
//
// Each 3x3x3 convolution of training (forward, data gradient, weight gradient)
// is an implicit GEMM of BF16 operands with FP32 accumulation: the operands are
// rounded from the FP32 master values while they are staged in shared memory
// channels-last, and a tap is a constant shift of the rows that ldmatrix reads,
// so no im2col operand is ever written.
//
//   forward     Y[o][co]  = sum_tap sum_ci X[o + tap][ci] W[tap][co][ci]
//   data grad   D[o][ci]  = sum_tap sum_co G[o + tap][co] Wf[tap][ci][co]   (Wf: ci/co swapped, taps reversed)
//   weight grad dW[co][tap][ci] = sum_o G[co][o] X[o + tap][ci]             (bias gradient summed in FP32)
//
// A batch of 64 items is 5 GFLOP in all, 3 us at the BF16 rate, and a layer has
// at most 64 output channels and 32k rows: every layer is bound by staging its
// operands and by launch latency, so warp-level MMAs (m16n8k16), which read
// their operands from where they were staged and need no tensor-memory
// allocation or epilogue copy, are enough to take the matrix work off the
// critical path. A training step of 64 items takes 291 us; with im2col operands
// written to memory and library GEMMs between them (92 + 20 launches) it took 664,
// with up to 32 channels per CTA and several items per weight-gradient unit (so 8
// to 64 CTAs a layer) 494, without programmatic launches 429, with the weight
// gradients on the data gradients' stream 335. Under the profiler the kernels of 64
// items issue in 7-19% of cycles with the tensor pipe active in 2-7%; at 256 the
// convolutions in 32-47% (tensor 8-19%), but the weight gradients, at most one CTA an
// SM, still in 8-17%: four times the matrix work does not bound them either.
// Bias, ReLU and the ReLU mask are applied in the epilogue. Sums and every
// result are FP32, as are the parameters and Adam's state; every reduction has a
// fixed order. The FP32 kernels of fl_unet.cu remain the exact path.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "fl_internal.cuh"
#include "fl_kernels.h"
#include "fl_unet.h"

namespace fl {
namespace {

constexpr int kConvThreads = 256;
constexpr int kWgradThreads = 288;  // a warp per (dz, dy)

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm4(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4_t(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// D += A B, m16n8k16, BF16 operands, FP32 accumulators.
__device__ __forceinline__ void mma16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ----------------------------------------------------------------- packed weights

// The seven 3x3x3 layers' BF16 weights, forward [tap][cout][cin] and, for the
// data gradients (every layer but the first), [tap][cin][cout] with the taps
// reversed. The first layer's two channels are padded to 32 taps.
struct PackLayer {
  int layer, cin, cout;
  int fwd, data;  // element offsets
};
constexpr int kPackLayers = 7;
struct PackTable {
  PackLayer l[kPackLayers];
  int total;
};
__host__ __device__ constexpr PackTable pack_table() {
  PackTable t{};
  const int layer[kPackLayers] = {0, 1, 2, 3, 4, 6, 8};
  const int cin[kPackLayers] = {2, 16, 16, 32, 32, 32, 16};
  const int cout[kPackLayers] = {16, 16, 32, 32, 64, 32, 16};
  int off = 0;
  for (int k = 0; k < kPackLayers; ++k) {
    t.l[k] = PackLayer{layer[k], cin[k], cout[k], 0, 0};
    t.l[k].fwd = off;
    off += (k == 0 ? 32 : 27) * cin[k] * cout[k];
  }
  for (int k = 1; k < kPackLayers; ++k) {
    t.l[k].data = off;
    off += 27 * cin[k] * cout[k];
  }
  t.total = off;
  return t;
}
__host__ __device__ constexpr int pack_index(int layer) {
  const PackTable t = pack_table();
  for (int k = 0; k < kPackLayers; ++k)
    if (t.l[k].layer == layer) return k;
  return -1;
}

// Element e of the forward (data = 0) or data-gradient half of the table.
__global__ void k_pack(const float* __restrict__ params, UNetLayout L, int data, __nv_bfloat16* __restrict__ out) {
  grid_dependency_wait(params);
  constexpr PackTable T = pack_table();
  const int first = data ? T.l[1].data : 0, end = data ? T.total : T.l[1].data;
  const int e = first + blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= end) return;
  int k = data ? 1 : 0;
  while (k + 1 < kPackLayers && e >= (data ? T.l[k + 1].data : T.l[k + 1].fwd)) ++k;
  const int cin = T.l[k].cin, cout = T.l[k].cout;
  const int r = e - (data ? T.l[k].data : T.l[k].fwd), tap = r / (cin * cout), m = r % (cin * cout);
  const float* w = params + L.offset[T.l[k].layer];
  float v = 0.0f;
  if (data) {
    const int ci = m / cout, co = m % cout;
    v = w[((size_t)co * cin + ci) * 27 + 26 - tap];
  } else if (tap < 27) {
    const int co = m / cin, ci = m % cin;
    v = w[((size_t)co * cin + ci) * 27 + tap];
  }
  out[e] = __float2bfloat16_rn(v);
}

// ----------------------------------------------------------------- staging

// Shape of one CTA's input: kItems items of kZ output planes, zero-padded by one
// cell all round, a cell's CIN channels contiguous (16 bytes of padding keep the
// eight rows of an ldmatrix in different banks; two channels are one word).
template <int S, int CIN, int ITEMS, int Z>
struct Tile {
  static constexpr int E = S + 2, kItems = ITEMS, kZ = Z;
  static constexpr int kPos = (Z + 2) * E * E;            // positions of one item
  static constexpr int kRow = CIN == 2 ? 2 : CIN + 8;     // BF16 per position
  static constexpr int kCells = ITEMS * Z * S * S;        // output cells
  static constexpr size_t kBytes = sizeof(__nv_bfloat16) * kRow * ITEMS * kPos;
  // first position (tap 0) of output cell m
  static __device__ __forceinline__ int pos(int m) {
    const int item = m / (Z * S * S), c = m % (Z * S * S);
    return item * kPos + (c / (S * S)) * E * E + ((c / S) % S) * E + c % S;
  }
};

template <int S, bool VALID, int CIN, int ITEMS, int Z, int THREADS>
__device__ __forceinline__ void stage(const float* __restrict__ in, int b0, int z0, int batch, __nv_bfloat16* tile) {
  using T = Tile<S, CIN, ITEMS, Z>;
  constexpr int EIN = VALID ? S + 2 : S, EIN3 = EIN * EIN * EIN, OFF = VALID ? 0 : 1, HC = CIN / 2;
#pragma unroll 4
  for (int i = threadIdx.x; i < ITEMS * T::kPos * HC; i += THREADS) {
    const int p = i % (ITEMS * T::kPos), c = i / (ITEMS * T::kPos), item = p / T::kPos, r = p % T::kPos;
    const int z = z0 + r / (T::E * T::E) - OFF, y = (r / T::E) % T::E - OFF, x = r % T::E - OFF;
    float v0 = 0.0f, v1 = 0.0f;
    if (b0 + item < batch && (VALID || (z >= 0 && z < S && y >= 0 && y < S && x >= 0 && x < S))) {
      const float* src = in + ((size_t)(b0 + item) * CIN + 2 * c) * EIN3 + (z * EIN + y) * EIN + x;
      v0 = src[0];
      v1 = src[EIN3];
    }
    *reinterpret_cast<__nv_bfloat162*>(tile + p * T::kRow + 2 * c) = __floats2bfloat162_rn(v0, v1);
  }
}

// ----------------------------------------------------------------- forward and data gradient

template <int S>
struct ConvShape {
  static constexpr int kItems = S == 2 ? 4 : 1, kZ = S == 8 ? 4 : S;
  static constexpr int kCo = S == 2 ? 32 : 16;  // output channels of one CTA
  static constexpr int kWm = S == 8 ? 8 : (S == 4 ? 4 : 2), kWn = 8 / kWm;  // warps over rows and channels
  static constexpr int kMw = S == 8 ? 2 : 1;                               // 16-row tiles per warp
};
template <int S, int CIN>
constexpr size_t conv_smem() {
  using T = Tile<S, CIN, ConvShape<S>::kItems, ConvShape<S>::kZ>;
  constexpr int kCo = ConvShape<S>::kCo;
  return T::kBytes + sizeof(__nv_bfloat16) * (CIN == 2 ? 32 * kCo * 2 : 27 * kCo * (CIN + 8));
}

// One CTA: kItems items' slab of kZ planes, kCo of the COUT channels. The epilogue adds
// the bias and applies the ReLU (forward), or the ReLU mask of `act` (data gradient).
template <int S, bool VALID, int CIN, int COUT, bool DATA>
__global__ void __launch_bounds__(kConvThreads)
    k_conv_mma(const float* __restrict__ in, const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias,
               float* __restrict__ out, int batch, int relu, const float* __restrict__ act) {
  grid_dependency_wait(in, w, bias, act);
  using C = ConvShape<S>;
  using T = Tile<S, CIN, C::kItems, C::kZ>;
  constexpr int kSlabs = S / C::kZ, S3 = S * S * S, kNw = C::kCo / 8 / C::kWn;
  const int co0 = blockIdx.y * C::kCo;
  constexpr int kW = CIN + 8;  // BF16 per (tap, output channel) row
  extern __shared__ __align__(16) unsigned char conv_bytes[];
  __nv_bfloat16* tile = reinterpret_cast<__nv_bfloat16*>(conv_bytes);
  __nv_bfloat16* wt = reinterpret_cast<__nv_bfloat16*>(conv_bytes + T::kBytes);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, wm = warp % C::kWm, wn = warp / C::kWm;
  const int b0 = blockIdx.x / kSlabs * C::kItems, z0 = (blockIdx.x % kSlabs) * C::kZ;
  if constexpr (CIN == 2) {
    static_assert(CIN != 2 || COUT == C::kCo, "the first layer's channels are one CTA's");
    for (int i = t; i < 32 * COUT * 2 / 8; i += kConvThreads)
      reinterpret_cast<uint4*>(wt)[i] = reinterpret_cast<const uint4*>(w)[i];
  } else {
    constexpr int kChunks = CIN / 8;
#pragma unroll 4
    for (int i = t; i < 27 * C::kCo * kChunks; i += kConvThreads) {
      const int row = i / kChunks, tap = row / C::kCo, o = row % C::kCo;
      *reinterpret_cast<uint4*>(wt + row * kW + (i % kChunks) * 8) =
          reinterpret_cast<const uint4*>(w)[(tap * COUT + co0 + o) * kChunks + i % kChunks];
    }
  }
  stage<S, VALID, CIN, C::kItems, C::kZ, kConvThreads>(in, b0, z0, batch, tile);
  __syncthreads();
  float acc[C::kMw][kNw][4];
#pragma unroll
  for (int m = 0; m < C::kMw; ++m)
#pragma unroll
    for (int n = 0; n < kNw; ++n)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[m][n][k] = 0.0f;
  if constexpr (CIN == 2) {
    // k = (tap, channel): a lane's word is one tap of one cell
    const unsigned* t32 = reinterpret_cast<const unsigned*>(tile);
    const unsigned* w32 = reinterpret_cast<const unsigned*>(wt);
    const int g = lane >> 2, q = lane & 3;
    int p[C::kMw][2];
#pragma unroll
    for (int m = 0; m < C::kMw; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) p[m][h] = T::pos((wm * C::kMw + m) * 16 + g + 8 * h);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int tap0 = 8 * s + q, tap1 = tap0 + 4;
      // (taps 27 .. 31 have zero weights: read tap 26's cell)
      const int u0 = min(tap0, 26), u1 = min(tap1, 26);
      const int o0 = (u0 / 9) * T::E * T::E + ((u0 / 3) % 3) * T::E + u0 % 3;
      const int o1 = (u1 / 9) * T::E * T::E + ((u1 / 3) % 3) * T::E + u1 % 3;
#pragma unroll
      for (int m = 0; m < C::kMw; ++m) {
        const unsigned a[4] = {t32[p[m][0] + o0], t32[p[m][1] + o0], t32[p[m][0] + o1], t32[p[m][1] + o1]};
#pragma unroll
        for (int n = 0; n < kNw; ++n) {
          const int co = (wn * kNw + n) * 8 + g;
          mma16816(acc[m][n], a, w32[tap0 * COUT + co], w32[tap1 * COUT + co]);
        }
      }
    }
  } else {
    unsigned arow[C::kMw];
#pragma unroll
    for (int m = 0; m < C::kMw; ++m)
      arow[m] = smem_addr(tile + T::pos((wm * C::kMw + m) * 16 + (lane & 15)) * T::kRow + (lane >> 4) * 8);
    // rows of the weights: n tile pairs (x4) or, for a single tile, its two k halves twice
    const unsigned brow =
        smem_addr(wt + (wn * kNw * 8 + (lane & 7) + (kNw > 1 ? (lane >> 4) * 8 : 0)) * kW + ((lane >> 3) & 1) * 8);
#pragma unroll 3
    for (int tap = 0; tap < 27; ++tap) {
      const int off = (tap / 9) * T::E * T::E + ((tap / 3) % 3) * T::E + tap % 3;
#pragma unroll
      for (int c = 0; c < CIN / 16; ++c) {
        unsigned b[(kNw + 1) / 2][4];
#pragma unroll
        for (int n = 0; n < (kNw + 1) / 2; ++n) ldsm4(b[n], brow + 2 * ((tap * C::kCo + 16 * n) * kW + 16 * c));
#pragma unroll
        for (int m = 0; m < C::kMw; ++m) {
          unsigned a[4];
          ldsm4(a, arow[m] + 2 * (off * T::kRow + 16 * c));
#pragma unroll
          for (int n = 0; n < kNw; ++n) mma16816(acc[m][n], a, b[n / 2][2 * (n & 1)], b[n / 2][2 * (n & 1) + 1]);
        }
      }
    }
  }
  const int g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int m = 0; m < C::kMw; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int cell = (wm * C::kMw + m) * 16 + g + 8 * h;
      const int item = cell / (C::kZ * S * S), r = z0 * S * S + cell % (C::kZ * S * S);
      if (b0 + item >= batch) continue;
#pragma unroll
      for (int n = 0; n < kNw; ++n)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int co = co0 + (wn * kNw + n) * 8 + 2 * q + k;
          const size_t o = ((size_t)(b0 + item) * COUT + co) * S3 + r;
          float v = acc[m][n][2 * h + k];
          if (DATA) {
            if (act != nullptr && !(act[o] > 0.0f)) v = 0.0f;
          } else {
            v += bias[co];
            if (relu) v = fmaxf(v, 0.0f);
          }
          out[o] = v;
        }
    }
}

// ----------------------------------------------------------------- weight gradient

template <int S, int CIN, int COUT>
struct WgradShape {
  static constexpr int kItems = S == 2 ? 4 : 1, kZ = S == 8 ? 4 : S;
  static constexpr int kCo = 16;  // output channels of one CTA
  using T = Tile<S, CIN, kItems, kZ>;
  static constexpr int kG = T::kCells + 8;  // BF16 per row of g
  static constexpr size_t kSmem = T::kBytes + sizeof(__nv_bfloat16) * kCo * kG;
};

// Work units (kItems items' slab of kZ planes) are dealt to gridDim.x CTAs in
// order; a warp owns one (dz, dy), its three dx and every input channel, so the
// gradient rows it loads serve all of them; each CTA writes one partial row
// (weights, then biases), added in order by wgrad_sum.
template <int S, bool VALID, int CIN, int COUT>
__global__ void __launch_bounds__(kWgradThreads)
    k_wgrad_mma(const float* __restrict__ in, const float* __restrict__ g, int batch, int units,
                float* __restrict__ part) {
  grid_dependency_wait(in, g);
  using W = WgradShape<S, CIN, COUT>;
  using T = typename W::T;
  constexpr int kSlabs = S / W::kZ, S3 = S * S * S, kM = W::kCo / 16, kN = CIN == 2 ? 1 : CIN / 8;
  constexpr int kDx = CIN == 2 ? 1 : 3;  // (two channels: the three dx share one 8-column tile)
  constexpr int kSteps = T::kCells / 16;
  extern __shared__ __align__(16) unsigned char wg_bytes[];
  __shared__ float db[W::kCo];
  __nv_bfloat16* tile = reinterpret_cast<__nv_bfloat16*>(wg_bytes);
  __nv_bfloat16* gt = reinterpret_cast<__nv_bfloat16*>(wg_bytes + T::kBytes);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, dz = warp / 3, dy = warp % 3;
  const int co0 = blockIdx.y * W::kCo;
  if (t < W::kCo) db[t] = 0.0f;
  float acc[kDx][kM][kN][4];
#pragma unroll
  for (int d = 0; d < kDx; ++d)
#pragma unroll
    for (int m = 0; m < kM; ++m)
#pragma unroll
      for (int n = 0; n < kN; ++n)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[d][m][n][k] = 0.0f;
  const int off = dz * T::E * T::E + dy * T::E;
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    const int b0 = u / kSlabs * W::kItems, z0 = (u % kSlabs) * W::kZ;
    __syncthreads();  // the previous unit's reads (and db's zeros)
    stage<S, VALID, CIN, W::kItems, W::kZ, kWgradThreads>(in, b0, z0, batch, tile);
    for (int o = warp; o < W::kCo; o += kWgradThreads / 32) {  // one warp per row of g: its FP32 sum too
      float sum = 0.0f;
      for (int c = 2 * lane; c < T::kCells; c += 64) {
        const int item = c / (W::kZ * S * S), r = z0 * S * S + c % (W::kZ * S * S);
        float2 v = make_float2(0.0f, 0.0f);
        if (b0 + item < batch)
          v = *reinterpret_cast<const float2*>(g + ((size_t)(b0 + item) * COUT + co0 + o) * S3 + r);
        sum += v.x + v.y;
        *reinterpret_cast<__nv_bfloat162*>(gt + o * W::kG + c) = __floats2bfloat162_rn(v.x, v.y);
      }
#pragma unroll
      for (int k = 16; k > 0; k >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, k);
      if (lane == 0) db[o] += sum;
    }
    __syncthreads();
    const unsigned arow = smem_addr(gt + (lane & 15) * W::kG + (lane >> 4) * 8);
#pragma unroll 2
    for (int s = 0; s < kSteps; ++s) {
      unsigned a[kM][4];
#pragma unroll
      for (int m = 0; m < kM; ++m) ldsm4(a[m], arow + 2 * (16 * m * W::kG + 16 * s));
      if constexpr (CIN == 2) {
        // column n of the tile is (dx = n / 2, channel n & 1); dx = 3 is not a tap and is dropped
        const int n = lane >> 2, q = lane & 3, dx = min(n >> 1, 2);
        const unsigned short* h = reinterpret_cast<const unsigned short*>(tile);
        unsigned b[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int m0 = 16 * s + 8 * k + 2 * q;
          const unsigned lo = h[2 * (T::pos(m0) + off + dx) + (n & 1)];
          const unsigned hi = h[2 * (T::pos(m0 + 1) + off + dx) + (n & 1)];
          b[k] = lo | (hi << 16);
        }
#pragma unroll
        for (int m = 0; m < kM; ++m) mma16816(acc[0][m][0], a[m], b[0], b[1]);
      } else {
        const int cell = 16 * s + (lane & 7) + ((lane >> 3) & 1) * 8;
        const unsigned brow = smem_addr(tile + (T::pos(cell) + off) * T::kRow + (lane >> 4) * 8);
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
#pragma unroll
          for (int n = 0; n < kN / 2; ++n) {
            unsigned b[4];
            ldsm4_t(b, brow + 2 * (dx * T::kRow + 16 * n));
#pragma unroll
            for (int m = 0; m < kM; ++m) {
              mma16816(acc[dx][m][2 * n], a[m], b[0], b[1]);
              mma16816(acc[dx][m][2 * n + 1], a[m], b[2], b[3]);
            }
          }
      }
    }
  }
  __syncthreads();  // db complete
  constexpr int kNw = COUT * CIN * 27;
  float* row = part + (size_t)blockIdx.x * (kNw + COUT);
  const int gr = lane >> 2, q = lane & 3;
#pragma unroll
  for (int d = 0; d < kDx; ++d)
#pragma unroll
    for (int m = 0; m < kM; ++m)
#pragma unroll
      for (int n = 0; n < kN; ++n)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int co = co0 + 16 * m + gr + 8 * (k >> 1), col = 8 * n + 2 * q + (k & 1);
          const int ci = CIN == 2 ? col & 1 : col, dx = CIN == 2 ? col >> 1 : d;
          if (dx < 3) row[((size_t)co * CIN + ci) * 27 + warp * 3 + dx] = acc[d][m][n][k];
        }
  if (t < W::kCo) row[kNw + co0 + t] = db[t];
}

template <int S, bool VALID, int CIN, int COUT>
cudaError_t conv(const UNetTcTrain& t, int layer, bool data, const float* in, const float* bias, float* out, int batch,
                 int relu, const float* act, cudaStream_t s) {
  using C = ConvShape<S>;
  constexpr size_t smem = conv_smem<S, CIN>();
  const PackLayer p = pack_table().l[pack_index(layer)];
  const dim3 grid((unsigned)((batch + C::kItems - 1) / C::kItems * (S / C::kZ)), COUT / C::kCo);
  ++g_kernel_launches;
  static OncePerDevice configured[2];
  if constexpr (VALID) {
    launch_dep(k_conv_mma<S, VALID, CIN, COUT, false>, grid, kConvThreads, smem, s, in, t.w + p.fwd, bias, out, batch,
               relu, nullptr);
  } else {
    auto* kernel = data ? k_conv_mma<S, VALID, CIN, COUT, true> : k_conv_mma<S, VALID, CIN, COUT, false>;
    once_on_device(configured[data],
                   [&] { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); });
    launch_dep(kernel, grid, kConvThreads, smem, s, in, t.w + (data ? p.data : p.fwd), bias, out, batch, relu, act);
  }
  return cudaGetLastError();
}

template <int S, bool VALID, int CIN, int COUT>
cudaError_t wgrad(const float* in, const float* g, int batch, float* part, float* dw, float* db, cudaStream_t s) {
  using W = WgradShape<S, CIN, COUT>;
  constexpr int nw = COUT * CIN * 27;
  const int units = (batch + W::kItems - 1) / W::kItems * (S / W::kZ);
  const int ctas = (int)std::min<long long>({(long long)units, 148, kWgradPart / (nw + COUT)});
  static OncePerDevice configured;
  once_on_device(configured, [] {
    cudaFuncSetAttribute(k_wgrad_mma<S, VALID, CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)W::kSmem);
  });
  ++g_kernel_launches;
  launch_dep(k_wgrad_mma<S, VALID, CIN, COUT>, dim3(ctas, COUT / W::kCo), kWgradThreads, W::kSmem, s, in, g,
             batch, units, part);
  wgrad_sum(part, ctas, nw, COUT, dw, db, s);
  return cudaGetLastError();
}

}  // namespace

cudaError_t unet_tc_train_create(UNetTcTrain* t) {
  *t = UNetTcTrain{};
  if (cudaMalloc(&t->w, sizeof(__nv_bfloat16) * pack_table().total) != cudaSuccess) {
    cudaGetLastError();
    return cudaErrorMemoryAllocation;
  }
  return cudaSuccess;
}

void unet_tc_train_destroy(UNetTcTrain* t) {
  cudaFree(t->w);
  *t = UNetTcTrain{};
}

cudaError_t unet_tc_train_pack(const UNetTcTrain& t, const float* params, bool data, cudaStream_t s) {
  constexpr PackTable T = pack_table();
  const int n = data ? T.total - T.l[1].data : T.l[1].data;
  ++g_kernel_launches;
  launch_dep(k_pack, (n + 255) / 256, 256, 0, s, params, unet_layout(), data ? 1 : 0, t.w);
  return cudaGetLastError();
}

cudaError_t conv3_fwd_tc(const UNetTcTrain& t, int layer, const float* in, const float* bias, float* out, int batch,
                         cudaStream_t s) {
  switch (layer) {
    case 0: return conv<8, true, 2, 16>(t, layer, false, in, bias, out, batch, 1, nullptr, s);
    case 1:
    case 8: return conv<8, false, 16, 16>(t, layer, false, in, bias, out, batch, 1, nullptr, s);
    case 2: return conv<4, false, 16, 32>(t, layer, false, in, bias, out, batch, 1, nullptr, s);
    case 3:
    case 6: return conv<4, false, 32, 32>(t, layer, false, in, bias, out, batch, 1, nullptr, s);
    case 4: return conv<2, false, 32, 64>(t, layer, false, in, bias, out, batch, 1, nullptr, s);
  }
  return cudaErrorInvalidValue;
}

cudaError_t conv3_bwd_data_tc(const UNetTcTrain& t, int layer, const float* g, const float* act, float* din, int batch,
                              cudaStream_t s) {
  switch (layer) {
    case 1:
    case 8: return conv<8, false, 16, 16>(t, layer, true, g, nullptr, din, batch, 0, act, s);
    case 2: return conv<4, false, 32, 16>(t, layer, true, g, nullptr, din, batch, 0, act, s);
    case 3:
    case 6: return conv<4, false, 32, 32>(t, layer, true, g, nullptr, din, batch, 0, act, s);
    case 4: return conv<2, false, 64, 32>(t, layer, true, g, nullptr, din, batch, 0, act, s);
  }
  return cudaErrorInvalidValue;
}

cudaError_t conv3_bwd_weight_tc(int layer, const float* in, const float* g, int batch, float* part, float* dw, float* db,
                                cudaStream_t s) {
  switch (layer) {
    case 0: return wgrad<8, true, 2, 16>(in, g, batch, part, dw, db, s);
    case 1:
    case 8: return wgrad<8, false, 16, 16>(in, g, batch, part, dw, db, s);
    case 2: return wgrad<4, false, 16, 32>(in, g, batch, part, dw, db, s);
    case 3:
    case 6: return wgrad<4, false, 32, 32>(in, g, batch, part, dw, db, s);
    case 4: return wgrad<2, false, 32, 64>(in, g, batch, part, dw, db, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace fl
