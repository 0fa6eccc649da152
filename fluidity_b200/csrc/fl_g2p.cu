// APIC grid-to-particle transfer with fused advection.
//
// Semantics follow GatherMac3D / GatherMacVelocityComponentFromSlots
// (native/src/transfers_3d.cc:199-261; native/src/mac_gather_3d_internal.h:15-69):
//   v_a          = sum_n w_n u_n
//   increment_a  = v_a - sum_n w_n u_old_n
//   C_a (fitted) = 4 * sum_n w_n u_n (x_n - x_p)/h  /  h
//   grad_a       = sum_n grad(w_n) u_n
// The step mode keeps (v, C) and advects x += dt v with a clamp to the
// non-solid box (the reference's contact-constrained update,
// liquid_boundary_transfer_3d.cu:544, is out of scope; a plain clamp stands in).
//
// B200 design: one CTA per non-empty 8^3 block. The CTA stages the block's
// 11x10x10 halo tile of each face component in shared memory (coalesced from
// the owned-face arrays of the 27 neighbouring blocks), then its threads stride
// over the block's contiguous particle range, gather all 81 samples from
// shared memory and keep C in registers.
#include "fl_internal.cuh"
#include "fl_kernels.h"

namespace fl {

constexpr int kG2PThreads = 256;

__device__ __forceinline__ int tile_ext0(int a) { return a == 0 ? 11 : 10; }
__device__ __forceinline__ int tile_ext1(int a) { return a == 1 ? 11 : 10; }

// Entry n of the block's three halo tiles in the owned-face arrays (its component
// in *a), or -1 where no active block owns the face.
__device__ __forceinline__ long long tile_source(const GridView& g, int b, int n, int* a) {
  *a = n / kTileFaces;
  const int idx = n % kTileFaces;
  const int e0 = tile_ext0(*a), e1 = tile_ext1(*a);
  const int nx = idx % e0 - 1, ny = (idx / e0) % e1 - 1, nz = idx / (e0 * e1) - 1;
  const int dx = nx < 0 ? -1 : (nx > 7 ? 1 : 0), dy = ny < 0 ? -1 : (ny > 7 ? 1 : 0),
            dz = nz < 0 ? -1 : (nz > 7 ? 1 : 0);
  const int nb = g.nbr27[b * 27 + nbr_index(dx, dy, dz)];
  return nb < 0 ? -1 : (long long)nb * kBlockCells + ((nz - 8 * dz) * 8 + (ny - 8 * dy)) * 8 + (nx - 8 * dx);
}

__device__ void load_tile(const GridView& g, int b, const float* const u[3], float* tile, int t) {
  for (int n = t; n < 3 * kTileFaces; n += kG2PThreads) {
    int a;
    const long long src = tile_source(g, b, n, &a);
    tile[n] = src >= 0 ? u[a][src] : 0.0f;
  }
}

// Four CTAs per SM (at most 64 registers): with the packed sums below and no
// cap the step kernel runs at less than half the speed (2.29 vs 0.95 ms at the
// 256^3 splash).
constexpr int kG2PMinBlocks = 4;

__global__ void __launch_bounds__(kG2PThreads, kG2PMinBlocks)
    k_g2p(GridView g, ParticlesView p, const int* cell_start, const float* u0, const float* u1, const float* u2,
          G2PParams prm, DeviceReport* rep) {
  __shared__ float tile[3 * kTileFaces];
  __shared__ unsigned int next_blocks;  // neighbouring blocks the advected particles land in
  const int b = blockIdx.x, t = threadIdx.x;
  if (b == 0 && t == 0 && rep != nullptr) rep->compiled_architecture = compiled_arch();
  const int pbeg = cell_start[b * kBlockCells], pend = cell_start[(b + 1) * kBlockCells];
  if (pbeg == pend) return;
  if (t == 0) next_blocks = 0u;
  const float* un[3] = {u0, u1, u2};
  load_tile(g, b, un, tile, t);
  __syncthreads();
  const int bc[3] = {g.coord[3 * b] * 8, g.coord[3 * b + 1] * 8, g.coord[3 * b + 2] * 8};
  const float four_inv_h = 4.0f * g.inv_h;  // fitted slopes 4 sum w u r / h (one multiply instead of a division)
  // Position of particle q (read through the cell order in fl_step); the
  // next particle's is loaded one iteration ahead, so its two dependent loads
  // overlap the current particle's work.
  auto load_x = [&](int q, float out[3]) {
    const int src = prm.order != nullptr ? (int)prm.order[q] : -1;
#pragma unroll
    for (int d = 0; d < 3; ++d) out[d] = src >= 0 ? prm.x_in[d][src] : p.x[d][q];
  };
  float xnext[3] = {0.0f, 0.0f, 0.0f};
  if (pbeg + t < pend) load_x(pbeg + t, xnext);
  for (int q = pbeg + t; q < pend; q += kG2PThreads) {
    float xw[3] = {xnext[0], xnext[1], xnext[2]}, X[3];
    if (q + kG2PThreads < pend) load_x(q + kG2PThreads, xnext);
    int cell[3];
    bool inside = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      X[d] = lattice_coord(g, xw[d], d);
      cell[d] = __float2int_rd(X[d]);
      inside = inside && cell[d] >= bc[d] && cell[d] < bc[d] + 8;
    }
    if (!inside) {  // the sort binned this particle elsewhere: never index the tile
      report_error(rep, kInternal, (unsigned long long)q);
      continue;
    }
    float vel[3], fit[9];
    // The cell-centred factors of each axis (shift 1/2) serve the two components
    // transverse to it, so they are formed once per particle; only the normal
    // axis's face-centred factors are formed per component.
    int firstC[3];
    float wC[3][3], wrC[3][3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float fst = floorf(X[d] - 1.0f);
      firstC[d] = (int)fst;
      const float a0 = fst + 0.5f;
      const float dl = X[d] - (a0 + 0.5f);
      const float dr = fabsf(X[d] - (a0 + 1.5f));
      const float c = X[d] - (a0 + 1.0f);
      wC[d][0] = 0.5f * dr * dr;
      wC[d][1] = 0.75f - c * c;
      wC[d][2] = 0.5f * dl * dl;
#pragma unroll
      for (int s = 0; s < 3; ++s) wrC[d][s] = wC[d][s] * ((a0 + (float)s) - X[d]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      // Axis factors: first node, weights, and weights times offset/h.
      int first[3];
      float w[3][3], wr[3][3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if (d != a) {
          first[d] = firstC[d];
#pragma unroll
          for (int s = 0; s < 3; ++s) w[d][s] = wC[d][s], wr[d][s] = wrC[d][s];
          continue;
        }
        const float fst = floorf(X[d] - 0.5f);
        first[d] = (int)fst;
        const float dl = X[d] - (fst + 0.5f);
        const float dr = fabsf(X[d] - (fst + 1.5f));
        const float c = X[d] - (fst + 1.0f);
        w[d][0] = 0.5f * dr * dr;
        w[d][1] = 0.75f - c * c;
        w[d][2] = 0.5f * dl * dl;
#pragma unroll
        for (int s = 0; s < 3; ++s) wr[d][s] = w[d][s] * ((fst + (float)s) - X[d]);
      }
      const int e0 = tile_ext0(a), e1 = tile_ext1(a);
      const int n0 = ((first[2] - bc[2] + 1) * e1 + (first[1] - bc[1] + 1)) * e0 + (first[0] - bc[0] + 1);
      const float* ta = tile + a * kTileFaces + n0;
      // The 27-node sums factor by axis: contract x (weights w0 and w0*r0), then
      // y, then z. Every output is the same sum of w-products times node values as
      // the direct 27-term form, with about half the FP32 operations.
      float pic, m0, m1, m2;
      {
        // The pairs (U0, U1), (V0, V1), (pic, m0) and (m1, m2) are each
        // updated by one packed FP32 FMA: every lane performs the scalar
        // form's operations in the same order, so the results are bitwise equal.
        const float2 wA[3] = {make_float2(w[0][0], wr[0][0]), make_float2(w[0][1], wr[0][1]),
                              make_float2(w[0][2], wr[0][2])};
        float2 pm0 = make_float2(0.0f, 0.0f), m12 = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int kz = 0; kz < 3; ++kz) {
          float2 V01 = make_float2(0.0f, 0.0f);
          float V2 = 0.0f;
#pragma unroll
          for (int ky = 0; ky < 3; ++ky) {
            const int row = (kz * e1 + ky) * e0;
            const float u0 = ta[row], u1 = ta[row + 1], u2 = ta[row + 2];
            float2 U01 = __fmul2_rn(wA[0], make_float2(u0, u0));
            U01 = __ffma2_rn(wA[1], make_float2(u1, u1), U01);
            U01 = __ffma2_rn(wA[2], make_float2(u2, u2), U01);
            V01 = __ffma2_rn(make_float2(w[1][ky], w[1][ky]), U01, V01);
            V2 = fmaf(wr[1][ky], U01.x, V2);
          }
          pm0 = __ffma2_rn(make_float2(w[2][kz], w[2][kz]), V01, pm0);
          m12 = __ffma2_rn(make_float2(w[2][kz], wr[2][kz]), make_float2(V2, V01.x), m12);
        }
        pic = pm0.x;
        m0 = pm0.y;
        m1 = m12.x;
        m2 = m12.y;
      }
      vel[a] = pic;
      fit[3 * a] = four_inv_h * m0;
      fit[3 * a + 1] = four_inv_h * m1;
      fit[3 * a + 2] = four_inv_h * m2;
    }
    bool finite = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) finite = finite && isfinite(vel[a]);
    if (!finite) report_error(rep, kOutOfRange, (unsigned long long)q);
    int off[3];
    bool near = true, valid = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      p.v[d][q] = vel[d];
      float nx = xw[d] + prm.dt * vel[d];
      nx = fminf(fmaxf(nx, prm.clamp_lo[d]), prm.clamp_hi[d]);
      p.x[d][q] = nx;
      // the next step's block of this particle (the cell rule of the sort)
      const float Xn = lattice_coord(g, nx, d);
      valid = valid && isfinite(Xn) && fabsf(Xn) < 1.0e9f;
      const int nb_d = floor_div8(valid ? __float2int_rd(Xn) : 0);
      off[d] = nb_d - bc[d] / 8;
      near = near && off[d] >= -1 && off[d] <= 1;
      valid = valid && nb_d - g.blo[d] >= 0 && nb_d - g.blo[d] < g.bdim[d];
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) p.c[k][q] = fit[k];
    // Particles that leave the lattice are reported by the next sort; here they mark nothing.
    if (prm.occ_next != nullptr) {
      // one shared-memory OR per warp for the neighbouring blocks
      const unsigned bit = valid && near ? 1u << nbr_index(off[0], off[1], off[2]) : 0u;
      const unsigned active = __activemask();
      const unsigned bits = __reduce_or_sync(active, bit);
      if (bits != 0u && (threadIdx.x & 31) == __ffs(active) - 1) atomicOr(&next_blocks, bits);
      if (valid && !near) {
        const int bx = bc[0] / 8 + off[0] - g.blo[0], by = bc[1] / 8 + off[1] - g.blo[1],
                  bz = bc[2] / 8 + off[2] - g.blo[2];
        prm.occ_next[((size_t)bz * g.bdim[1] + by) * g.bdim[0] + bx] = 1;
      }
    }
  }
  if (prm.occ_next != nullptr) {
    __syncthreads();
    if (t < 27 && ((next_blocks >> t) & 1u)) {
      const int bx = bc[0] / 8 + t % 3 - 1 - g.blo[0], by = bc[1] / 8 + (t / 3) % 3 - 1 - g.blo[1],
                bz = bc[2] / 8 + t / 9 - 1 - g.blo[2];
      prm.occ_next[((size_t)bz * g.bdim[1] + by) * g.bdim[0] + bx] = 1;
    }
  }
}

// The full gather (24 values per particle: velocity, increment over the old
// faces, fitted slopes, gradients). Bound by instruction issue: 81 x 2 node
// values and about 330 FMAs a particle, contracted axis by axis in packed pairs
// (u and old share their weights and lie side by side in the tile: one 8-byte load
// is the pair that dw0 u + w0 old's FMA takes, without moves; two tiles of their
// own cost 6% of the whole call below). A particle's
// record is 96 contiguous bytes, so a warp's 32 records are staged in shared
// memory (rows of 25 words: no conflicts) and stored as 24 contiguous 128-byte
// lines; a lane storing its own record touches 32 lines per instruction. The
// 120 x 104 x 88 transfers, whose gather this is, went from 616 to 534 us with the
// staged records, to 500 with the pairs and to 484 with the tile's lookups in batches.
constexpr int kFullRow = 25;
// Tile entries of a thread in flight at once, lookups before values: the 13 entries are two
// dependent round trips each, and with three CTAs an SM one entry after another left blocks
// of few particles behind the kernel that shared the step's four (17 a block, no old field: 56 ->
// 60 us at 1.9k blocks; now 53, and 240 instead of 248 at 512 a block with one).
constexpr int kFullBatch = 7;
constexpr size_t kFullSmem = sizeof(float) * (6 * kTileFaces + kG2PThreads * kFullRow);

__global__ void __launch_bounds__(kG2PThreads, 3)
    k_g2p_full(GridView g, ParticlesView p, const int* cell_start, const float* u0, const float* u1, const float* u2,
               const float* o0, const float* o1, const float* o2, float* full_out, DeviceReport* rep) {
  extern __shared__ float full_smem[];
  float2* tile = reinterpret_cast<float2*>(full_smem);  // (new, old) face velocities
  const int b = blockIdx.x, t = threadIdx.x, lane = t & 31;
  float* rows = full_smem + 6 * kTileFaces + (t - lane) * kFullRow;  // the warp's staged records
  if (b == 0 && t == 0 && rep != nullptr) rep->compiled_architecture = compiled_arch();
  const int pbeg = cell_start[b * kBlockCells], pend = cell_start[(b + 1) * kBlockCells];
  if (pbeg == pend) return;
#pragma unroll 1
  for (int n0 = t; n0 < 3 * kTileFaces; n0 += kFullBatch * kG2PThreads) {
    int src[kFullBatch];  // at most 2^21 blocks of 512 faces
#pragma unroll
    for (int k = 0; k < kFullBatch; ++k) {
      const int n = n0 + k * kG2PThreads;
      int a;
      src[k] = n < 3 * kTileFaces ? (int)tile_source(g, b, n, &a) : -1;
    }
    float2 v[kFullBatch];
#pragma unroll
    for (int k = 0; k < kFullBatch; ++k) {
      const int a = (n0 + k * kG2PThreads) / kTileFaces;
      const float* fresh = a == 0 ? u0 : (a == 1 ? u1 : u2);
      const float* old = a == 0 ? o0 : (a == 1 ? o1 : o2);
      v[k] = make_float2(src[k] >= 0 ? fresh[src[k]] : 0.0f, src[k] >= 0 && o0 != nullptr ? old[src[k]] : 0.0f);
    }
#pragma unroll
    for (int k = 0; k < kFullBatch; ++k)
      if (n0 + k * kG2PThreads < 3 * kTileFaces) tile[n0 + k * kG2PThreads] = v[k];
  }
  __syncthreads();
  const int bc[3] = {g.coord[3 * b] * 8, g.coord[3 * b + 1] * 8, g.coord[3 * b + 2] * 8};
  const float four_inv_h = 4.0f * g.inv_h;
  float xnext[3] = {0.0f, 0.0f, 0.0f};
  if (pbeg + t < pend) {
#pragma unroll
    for (int d = 0; d < 3; ++d) xnext[d] = p.x[d][pbeg + t];
  }
  for (int q0 = pbeg + t - lane; q0 < pend; q0 += kG2PThreads) {  // uniform over the warp
    const int q = q0 + lane;
    float X[3];
    int cell[3];
    bool inside = q < pend;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      X[d] = lattice_coord(g, xnext[d], d);
      if (q + kG2PThreads < pend) xnext[d] = p.x[d][q + kG2PThreads];
      cell[d] = __float2int_rd(X[d]);
      inside = inside && cell[d] >= bc[d] && cell[d] < bc[d] + 8;
    }
    if (q < pend && !inside) report_error(rep, kInternal, (unsigned long long)q);  // the sort binned it elsewhere
    if (inside) {
      float* row = rows + lane * kFullRow;
      bool finite = true;
#pragma unroll 1
      for (int a = 0; a < 3; ++a) {
        // Axis factors: first node, weights, derivatives and weights times offset/h.
        int first[3];
        float w[3][3], dw[3][3], wr[3][3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float shift = d == a ? 0.0f : 0.5f;
          const float fst = floorf(X[d] - shift - 0.5f);
          first[d] = (int)fst;
          const float a0 = fst + shift;
          const float dl = X[d] - (a0 + 0.5f);
          const float dr = fabsf(X[d] - (a0 + 1.5f));
          const float c = X[d] - (a0 + 1.0f);
          w[d][0] = 0.5f * dr * dr;
          w[d][1] = 0.75f - c * c;
          w[d][2] = 0.5f * dl * dl;
          dw[d][0] = -dr;
          dw[d][1] = -2.0f * c;
          dw[d][2] = dl;
#pragma unroll
          for (int s = 0; s < 3; ++s) wr[d][s] = w[d][s] * ((a0 + (float)s) - X[d]);
        }
        const int e0 = tile_ext0(a), e1 = tile_ext1(a);
        const int n0 = ((first[2] - bc[2] + 1) * e1 + (first[1] - bc[1] + 1)) * e0 + (first[0] - bc[0] + 1);
        const float2* ta = tile + a * kTileFaces + n0;
        float2 pm0 = make_float2(0.0f, 0.0f), m1g1 = pm0, m2g2 = pm0, g0old = pm0;
#pragma unroll
        for (int kz = 0; kz < 3; ++kz) {
          float2 V01 = make_float2(0.0f, 0.0f), V24 = V01, V35 = V01;
#pragma unroll
          for (int ky = 0; ky < 3; ++ky) {
            const int at = (kz * e1 + ky) * e0;
            float2 U01, Uo;
#pragma unroll
            for (int kx = 0; kx < 3; ++kx) {
              const float2 node = ta[at + kx];  // one 8-byte load, and the pair that Uo's FMA takes
              const float u = node.x;
              const float2 wx = make_float2(w[0][kx], wr[0][kx]), dx = make_float2(dw[0][kx], w[0][kx]);
              U01 = kx == 0 ? __fmul2_rn(wx, make_float2(u, u)) : __ffma2_rn(wx, make_float2(u, u), U01);
              Uo = kx == 0 ? __fmul2_rn(dx, node) : __ffma2_rn(dx, node, Uo);
            }
            const float2 wy = make_float2(w[1][ky], w[1][ky]);
            V01 = __ffma2_rn(wy, U01, V01);
            V35 = __ffma2_rn(wy, Uo, V35);
            V24 = __ffma2_rn(make_float2(wr[1][ky], dw[1][ky]), make_float2(U01.x, U01.x), V24);
          }
          const float2 wz = make_float2(w[2][kz], w[2][kz]);
          pm0 = __ffma2_rn(wz, V01, pm0);
          m1g1 = __ffma2_rn(wz, V24, m1g1);
          g0old = __ffma2_rn(wz, V35, g0old);
          m2g2 = __ffma2_rn(make_float2(wr[2][kz], dw[2][kz]), make_float2(V01.x, V01.x), m2g2);
        }
        finite = finite && isfinite(pm0.x);
        row[a] = pm0.x;
        row[3 + a] = pm0.x - g0old.y;
        row[6 + 3 * a] = four_inv_h * pm0.y;
        row[7 + 3 * a] = four_inv_h * m1g1.x;
        row[8 + 3 * a] = four_inv_h * m2g2.x;
        row[15 + 3 * a] = g0old.x * g.inv_h;
        row[16 + 3 * a] = m1g1.y * g.inv_h;
        row[17 + 3 * a] = m2g2.y * g.inv_h;
      }
      if (!finite) report_error(rep, kOutOfRange, (unsigned long long)q);
    }
    const unsigned have = __ballot_sync(0xffffffffu, inside);  // records of other particles stay as they are
    __syncwarp();
    float* out = full_out + 24 * (size_t)q0;
#pragma unroll
    for (int k = 0; k < 24; ++k) {
      const int e = lane + 32 * k, r = e / 24;
      if ((have >> r) & 1u) out[e] = rows[r * kFullRow + e % 24];
    }
    __syncwarp();
  }
}

cudaError_t launch_g2p(const GridView& g, const ParticlesView& p, const int* cell_start, const float* const u[3],
                       const float* const u_old[3], const G2PParams& prm, float* full_out, DeviceReport* rep,
                       cudaStream_t s) {
  if (g.nb == 0 || p.count == 0) return cudaSuccess;
  ++g_kernel_launches;
  if (full_out != nullptr) {
    static OncePerDevice configured;
    once_on_device(configured, [] {
      cudaFuncSetAttribute(k_g2p_full, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFullSmem);
    });
    k_g2p_full<<<g.nb, kG2PThreads, kFullSmem, s>>>(g, p, cell_start, u[0], u[1], u[2], u_old ? u_old[0] : nullptr,
                                                    u_old ? u_old[1] : nullptr, u_old ? u_old[2] : nullptr, full_out,
                                                    rep);
  } else {
    k_g2p<<<g.nb, kG2PThreads, 0, s>>>(g, p, cell_start, u[0], u[1], u[2], prm, rep);
  }
  return cudaGetLastError();
}

}  // namespace fl
