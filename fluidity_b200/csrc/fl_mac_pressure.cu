// Reference-shaped integrated MAC pressure projection on the GPU.
//
// Replaces ProjectMacPressure3D / CudaProjectMacPressure3D
// (native/include/fluidity/host/mac_pressure_3d.h:14-102,
// native/include/fluidity/host/cuda_mac_pressure_3d.h:19-20) for the bounded
// owned-face systems those operators take (1-4096 pressure cells, at most
// 24576 faces): general fluid volumes, target divergences, compliance (bulk
// modulus), wall fluxes, apertures, mobilities, pressure-gradient distances,
// internal pressure jumps, Dirichlet exterior pressures and sealed faces. The
// arithmetic follows the integrated system of native/src/
// mac_pressure_3d_arithmetic.h (FreezeCell :110-146, FreezeLinkFromIncidence
// :174-245, AssembleIntegratedRhsInto :263-313 with compensated sums,
// SelectGaugesInto :328-399, ApplyOriginalPressureOperatorInto :404-436,
// CorrectFacesAndAccumulatePhysicalDefectInto :440-503), the warm start of
// InitializeMacPressure3D (mac_pressure_3d_multigrid.cc:401-419) and the
// evaluation and identity check of mac_pressure_workspace_3d.cc:399-461.
//
// B200 layout. Such a system is a few hundred KB and its solve a chain of some
// hundred dependent sums, so it is bound by the latency of a CG iteration. One
// cluster of 8 CTAs x 512 threads does all of it in a single launch, in FP64,
// with one cell per thread: a thread keeps its cell's row (six conductances and
// the addresses of the six neighbours), residual, preconditioned residual and
// pressure in registers; only the search direction is shared, through
// distributed shared memory. A sum over all cells is warp shuffles, one remote
// store per warp and CTA, and a cluster barrier, after which every warp adds the
// 128 warp sums itself in a fixed order: three cluster barriers per iteration.
// The 3375-cell dam break to the reference's gate takes 175 us; one CTA of 1024
// threads with the vectors in its shared memory took 643 us.
// Before the solve: per-face coefficients, then per cell the right-hand side and
// the diagonal summed over its incident faces in increasing face order (the
// order of the reference's face loop, so the compensated sums are the
// reference's sums) and the gauge balance of every unanchored component; after
// it the evaluation (corrected face velocities, residuals, physical defects, the
// residual/defect identity). The host does only index
// work: face endpoints by binary search, per-cell face lists, connected
// components and gauges. This file is compiled with -fmad=false so that no
// product is fused into a sum, as in the reference's FP64 arithmetic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <chrono>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/fluidity_b200.h"
#include "fl_internal.cuh"
#include "fl_kernels.h"

namespace fl {
namespace {

constexpr int kMpCtas = 8, kMpThreads = 512;  // one cluster
constexpr int kMpAll = kMpCtas * kMpThreads;
constexpr int kMpWarps = kMpAll / 32;
constexpr uint64_t kMpMaxCells = 4096;   // mac_pressure_3d_arithmetic.h:19
static_assert(kMpMaxCells <= (uint64_t)kMpAll, "one cell per thread");
constexpr uint64_t kMpMaxFaces = 24576;  // mac_pressure_3d_arithmetic.h:20
constexpr int kMpMaxIterations = 65536;

enum { kLinkSealed = 0, kLinkInternal = 1, kLinkDirichlet = 2 };

struct MpStatus {
  int status;
  int iterations;
  int arch;
  double true_residual_l2, max_volume_scaled_residual, max_defect, rhs_l2;
};

// Device view of one system. Per-cell face lists hold (face << 1) | side,
// side 1 when the cell is the face's head; unanchored components list their
// cells and their faces that do not join two cells of the same component,
// with the sign of the face's wall flux in the component's balance.
struct MpSystem {
  int nc, nf, ncomp;
  double h, dt, rel_tol;
  int max_iterations;
  const double* cell_values;  // nc x 5
  const double* face_values;  // nf x 6
  const int* face_kind;
  const int* tail;
  const int* head;
  const int* cell_ent;  // 6 nc
  const int* root;       // component root (smallest ordinal) per cell
  const unsigned char* pinned;
  const int* comp_cell_off;  // ncomp + 1 (unanchored components only)
  const int* comp_cells;
  const int* comp_face_off;
  const int* comp_faces;  // (face << 1) | (1 when the component holds the head)
  // work and results
  double *scale, *cond, *wall_face;  // nf
  double *rhs, *p, *residual, *defect;  // nc
  double* corrected_u;                                    // nf
  MpStatus* out;
};

// Neumaier-compensated sum (CompensatedSum, mac_pressure_3d_arithmetic.h:57-74).
struct NSum {
  double sum = 0.0, corr = 0.0;
  __device__ void add(double t) {
    const double next = sum + t;
    if (fabs(sum) >= fabs(t))
      corr += (sum - next) + t;
    else
      corr += (t - next) + sum;
    sum = next;
  }
  __device__ double total() const { return sum + corr; }
};
struct Row {
  NSum flux, absolute;
  __device__ void add(double t) {
    flux.add(t);
    absolute.add(fabs(t));
  }
};

__device__ __forceinline__ unsigned mp_map(unsigned a, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ double mp_ld(unsigned a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void mp_st(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
// Cluster barrier; orders the cluster's shared and global memory accesses.
__device__ __forceinline__ void mp_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// Sums (and, for the last N - kSums values, maxima) of v[N] over the cluster,
// returned to every thread: `slots` holds N doubles per warp of the cluster, is
// written by every CTA and may be written again only after a further barrier.
template <int N, int kSums>
__device__ void mp_reduce(double (&v)[N], double* slots, unsigned rank) {
  const int lane = threadIdx.x & 31, warp = (int)rank * (kMpThreads / 32) + (threadIdx.x >> 5);
#pragma unroll
  for (int n = 0; n < N; ++n) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, v[n], o);
      v[n] = n < kSums ? v[n] + w : fmax(v[n], w);
    }
  }
  if (lane < kMpCtas) {
    const unsigned to = mp_map((unsigned)__cvta_generic_to_shared(slots + warp * N), (unsigned)lane);
#pragma unroll
    for (int n = 0; n < N; ++n) mp_st(to + 8u * n, v[n]);
  }
  mp_sync();
#pragma unroll
  for (int n = 0; n < N; ++n) {
    double s = slots[lane * N + n];
#pragma unroll
    for (int k = 1; k < kMpWarps / 32; ++k) {
      const double w = slots[(lane + 32 * k) * N + n];
      s = n < kSums ? s + w : fmax(s, w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, s, o);
      s = n < kSums ? s + w : fmax(s, w);
    }
    v[n] = s;
  }
}

// One cell's row: its compliance, then per incident face (increasing face
// order) the conductance (0: no flux), the address of the other cell's entry of
// the shared vector, whether there is such a cell (its value is zero otherwise)
// and the side this cell is on.
struct MpRow {
  double compliance, c[6];
  unsigned other[6], has, head;  // bit k: face k has another cell; this cell is face k's head
};
// (A x)_i for x_i = xi: the flux is c (x_tail - x_head) as in the face loop.
__device__ __forceinline__ double mp_apply(const MpRow& r, double xi) {
  double out = r.compliance * xi, xo[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) xo[k] = (r.has >> k) & 1u ? mp_ld(r.other[k]) : 0.0;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    if (r.c[k] == 0.0) continue;
    if ((r.head >> k) & 1u)
      out -= r.c[k] * (xo[k] - xi);
    else
      out += r.c[k] * (xi - xo[k]);
  }
  return out;
}

__device__ double corrected_velocity(const MpSystem& S, const double* p, int f) {
  const double* v = S.face_values + 6 * f;
  double u = v[3];
  if (v[0] > 0.0) {
    const int kind = S.face_kind[f];
    const double ext = kind == kLinkDirichlet ? v[5] : 0.0;
    const double jump = kind == kLinkInternal ? v[5] : 0.0;
    const int t = S.tail[f], hd = S.head[f];
    const double pt = t >= 0 ? p[t] : ext, ph = hd >= 0 ? p[hd] : ext;
    u += S.scale[f] * (pt - ph + jump);
  }
  return u;
}

__global__ void __cluster_dims__(kMpCtas, 1, 1) __launch_bounds__(kMpThreads, 1) k_mac_pressure(MpSystem S) {
  __shared__ double vec[kMpThreads];  // the shared vector: this CTA's cells
  __shared__ double slots_a[kMpWarps], slots_b[2 * kMpWarps], slots_c[5 * kMpWarps];
  unsigned rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int t = (int)rank * kMpThreads + threadIdx.x;  // this thread's cell
  const int nc = S.nc, nf = S.nf;
  const bool mine = t < nc;
  if (t == 0) S.out->arch = compiled_arch();
  const double full_area = S.h * S.h;
  // Face coefficients (FreezeLinkFromIncidence).
  for (int f = t; f < nf; f += kMpAll) {
    const double* v = S.face_values + 6 * f;
    double sc = 0.0, c = 0.0;
    if (v[0] > 0.0) {
      sc = (S.dt * v[1]) / v[2];
      c = v[0] * sc;
    }
    S.scale[f] = sc;
    S.cond[f] = c;
    S.wall_face[f] = (full_area - v[0]) * v[4];
  }
  mp_sync();
  // Right-hand side and diagonal (AssembleIntegratedRhsInto): the cell's own
  // terms, then its six faces in increasing face order; each face entry resolved
  // for the operator row. Every cell lists exactly its six incident faces (the
  // host checks the face set), so cell i's entries are 6i .. 6i + 5.
  MpRow row{};
  double dg = 0.0, rhs = 0.0, rhs_abs = 0.0, start = 0.0;
  bool pinned = false;
  const unsigned vec_a = (unsigned)__cvta_generic_to_shared(vec);
  if (mine) {
    const double* v = S.cell_values + 5 * t;
    row.compliance = v[2] == 0.0 ? 0.0 : v[0] / (v[2] * S.dt);
    Row sum;
    sum.add(v[0] * v[1]);
    sum.add(v[4]);
    sum.add(row.compliance * v[3]);
    dg = row.compliance;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int ent = S.cell_ent[6 * t + k], f = ent >> 1;
      const bool is_head = ent & 1;
      const int other = is_head ? S.tail[f] : S.head[f];
      const double c = S.cond[f];
      row.c[k] = c;
      if (other >= 0) {
        row.other[k] = mp_map(vec_a + 8u * (unsigned)(other % kMpThreads), (unsigned)(other / kMpThreads));
        row.has |= 1u << k;
      }
      row.head |= is_head ? 1u << k : 0u;
      const double* fv = S.face_values + 6 * f;
      const double fluid_flux = fv[0] * fv[3];
      const double sgn = is_head ? 1.0 : -1.0;
      sum.add(sgn * fluid_flux);
      sum.add(sgn * S.wall_face[f]);
      const int kind = S.face_kind[f];
      if (kind == kLinkInternal)
        sum.add(sgn * (c * fv[5]));
      else if (kind == kLinkDirichlet)
        sum.add(c * fv[5]);
      dg += c;
    }
    rhs = sum.flux.total();
    rhs_abs = sum.absolute.total();
    S.rhs[t] = rhs;
    pinned = S.pinned[t] != 0;
    // Warm start: the previous pressure, less the pin's on unanchored components.
    const int rt = S.root[t];
    start = v[3] - (S.pinned[rt] ? S.cell_values[5 * rt + 3] : 0.0);
  }
  // Gauge balance of each unanchored component (SelectGaugesInto): its cells'
  // source and wall terms, then the wall flux of its faces, in order.
  double unbalanced = 0.0;
  for (int k = t; k < S.ncomp; k += kMpAll) {
    Row bal;
    for (int e = S.comp_cell_off[k]; e < S.comp_cell_off[k + 1]; ++e) {
      const double* v = S.cell_values + 5 * S.comp_cells[e];
      bal.add(v[0] * v[1]);
      bal.add(v[4]);
    }
    for (int e = S.comp_face_off[k]; e < S.comp_face_off[k + 1]; ++e) {
      const int f = S.comp_faces[e] >> 1;
      bal.add((S.comp_faces[e] & 1) ? S.wall_face[f] : -1.0 * S.wall_face[f]);
    }
    if (fabs(bal.flux.total()) > 32.0 * DBL_EPSILON * bal.absolute.total()) unbalanced = 1.0;
  }
  double P = start, D = 0.0;
  vec[threadIdx.x] = P;
  double first[2] = {rhs * rhs, unbalanced};
  mp_reduce<2, 1>(first, slots_b, rank);
  if (first[1] != 0.0) {  // the same for every thread of the cluster
    if (t == 0) {
      S.out->status = FL_FAILED_PRECONDITION;
      S.out->iterations = 0;
      S.out->true_residual_l2 = S.out->max_volume_scaled_residual = S.out->max_defect = S.out->rhs_l2 = 0.0;
    }
    return;
  }
  const double bnorm = sqrt(first[0]);
  // ||b - Ap||_2 <= rel_tol ||b||_2, or the reference's gate 2e-6 + 2e-6 ||b||_2
  const double limit = S.rel_tol > 0.0 ? S.rel_tol * bnorm : 2e-6 + 2e-6 * bnorm;
  // Jacobi-preconditioned CG; the pinned rows stay at their warm start.
  const bool solved = mine && !pinned, scaled = solved && dg != 0.0;
  double R = solved ? rhs - mp_apply(row, P) : 0.0;
  double Z = scaled ? R / dg : 0.0;
  double sums[2] = {R * R, R * Z};
  mp_sync();  // every CTA has read slots_b and its neighbours' starts
  mp_reduce<2, 2>(sums, slots_b, rank);
  double rr = sums[0], rz = sums[1], rz_prev = 0.0;
  int it = 0;
  double status = FL_OK;
  for (; it < S.max_iterations; ++it) {
    if (sqrt(rr) <= limit) break;
    const double beta = it == 0 ? 0.0 : rz / rz_prev;
    D = it == 0 ? Z : Z + beta * D;
    vec[threadIdx.x] = D;
    mp_sync();
    const double Q = solved ? mp_apply(row, D) : 0.0;
    double dq[1] = {D * Q};
    mp_reduce<1, 1>(dq, slots_a, rank);  // its barrier also ends the reads of vec
    if (!(dq[0] > 0.0)) {
      status = FL_ABORTED;
      break;
    }
    const double alpha = rz / dq[0];
    P += alpha * D;
    R = R - alpha * Q;
    Z = scaled ? R / dg : 0.0;
    double next[2] = {R * R, R * Z};
    mp_reduce<2, 2>(next, slots_b, rank);
    rz_prev = rz;
    rr = next[0];
    rz = next[1];
  }
  // Evaluation: corrected faces, residuals b - Ap, physical defects and the
  // identity V d + r = 0 within 64 ulp of the terms' magnitudes.
  if (mine) S.p[t] = P;
  mp_sync();
  for (int f = t; f < nf; f += kMpAll) {
    const double u = corrected_velocity(S, S.p, f);
    if (!isfinite(u)) status = fmax(status, (double)FL_OUT_OF_RANGE);
    S.corrected_u[f] = u;
  }
  mp_sync();
  double l2 = 0.0, maxr = 0.0, maxd = 0.0;
  if (mine) {
    const double* v = S.cell_values + 5 * t;
    Row op, ph;
    op.add(row.compliance * P);
    ph.add(-v[0] * v[1]);
    ph.add(-v[4]);
    if (row.compliance > 0.0) ph.add(row.compliance * (P - v[3]));
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int ent = S.cell_ent[6 * t + k], f = ent >> 1;
      const bool is_head = ent & 1;
      if (row.c[k] != 0.0) {
        const int tl = S.tail[f], hd = S.head[f];
        const double pt = tl >= 0 ? S.p[tl] : 0.0, phd = hd >= 0 ? S.p[hd] : 0.0;
        const double flux = row.c[k] * (pt - phd);
        op.add(is_head ? -flux : flux);
      }
      const double flux = S.face_values[6 * f] * S.corrected_u[f];
      if (is_head) {
        ph.add(-flux);
        ph.add(-S.wall_face[f]);
      } else {
        ph.add(flux);
        ph.add(S.wall_face[f]);
      }
    }
    const double r = rhs - op.flux.total();
    const double dd = ph.flux.total() / v[0];
    const double ident = v[0] * dd + r;
    const double absterms = rhs_abs + op.absolute.total() + ph.absolute.total();
    if (fabs(ident) > 64.0 * DBL_EPSILON * absterms) status = fmax(status, (double)FL_INTERNAL);
    S.residual[t] = r;
    S.defect[t] = dd;
    l2 = r * r;
    maxr = fabs(r) / v[0];
    maxd = fabs(dd);
  }
  double ends[5] = {l2, rhs * rhs, maxr, maxd, status};
  mp_reduce<5, 2>(ends, slots_c, rank);
  if (t == 0) {
    const double norm = sqrt(ends[0]);
    int st = (int)ends[4];  // the gravest of the cells' and faces' codes
    if (st == FL_OK && norm > limit * 1.000001 + 1e-300) st = FL_ABORTED;
    S.out->status = st;
    S.out->iterations = it;
    S.out->true_residual_l2 = norm;
    S.out->max_volume_scaled_residual = ends[2];
    S.out->max_defect = ends[3];
    S.out->rhs_l2 = sqrt(ends[1]);
  }
}

bool cell_less(const int32_t* a, const int32_t* b) {
  if (a[2] != b[2]) return a[2] < b[2];
  if (a[1] != b[1]) return a[1] < b[1];
  return a[0] < b[0];
}

int find_cell(const int32_t* cells, int nc, int32_t x, int32_t y, int32_t z) {
  const int32_t key[3] = {x, y, z};
  int lo = 0, hi = nc;
  while (lo < hi) {
    const int mid = (lo + hi) / 2;
    if (cell_less(cells + 3 * mid, key))
      lo = mid + 1;
    else
      hi = mid;
  }
  if (lo < nc && !cell_less(key, cells + 3 * lo)) return lo;
  return -1;
}

// Owned-slot order of a face in the reference's sparse grid of 4^3 blocks
// (SparseMacGrid3D::FaceSlot, sparse_mac_grid_3d.cc:388-409): blocks in
// (z,y,x) order, then the normal axis, then the local (z,y,x) position; the
// face at lattice index (i,j,k) is owned by the block of cell (i,j,k).
using FaceKey = OwnedFaceKey;

FaceKey face_key(int axis, int64_t x, int64_t y, int64_t z) {
  auto fdiv = [](int64_t a) { return (int32_t)(a >= 0 ? a / 4 : -((-a + 3) / 4)); };
  auto fmod = [](int64_t a) { return (int32_t)(((a % 4) + 4) % 4); };
  return FaceKey{{fdiv(z), fdiv(y), fdiv(x), axis, fmod(z), fmod(y), fmod(x)}};
}

// Largest cell bounding box (in lattice positions) given a dense ordinal lookup.
constexpr size_t kMpLutCap = 1 << 20;

// The owned-slot order of faces as two words: (block z, block y) and
// (block x, axis, local z, y, x); int32 order kept by flipping sign bits.
struct PackedFaceKey {
  uint64_t hi, lo;
  bool operator<(const PackedFaceKey& o) const { return hi != o.hi ? hi < o.hi : lo < o.lo; }
};

PackedFaceKey packed_face_key(int axis, int64_t x, int64_t y, int64_t z) {
  const FaceKey k = face_key(axis, x, y, z);  // block z, y, x, axis, local z, y, x
  auto u = [](int32_t v) { return (uint64_t)((uint32_t)v ^ 0x80000000u); };
  const uint64_t local = (uint64_t)((k.v[3] << 6) | (k.v[4] << 4) | (k.v[5] << 2) | k.v[6]);
  return PackedFaceKey{(u(k.v[0]) << 32) | u(k.v[1]), (u(k.v[2]) << 8) | local};
}

int find_root(std::vector<int>& parent, int c) {
  while (parent[c] != c) c = parent[c];
  return c;
}

}  // namespace

static_assert(sizeof(MpStatus) % sizeof(double) == 0, "the status follows the results in one copy");

// Bytes of the arena's inputs for nc cells, nf faces, ent cell-face entries,
// ncomp unanchored components, comp_faces component face entries.
size_t mp_input_bytes(size_t nc, size_t nf, size_t ent, size_t ncomp, size_t comp_faces) {
  const size_t ni = 3 * nf + ent + nc + (ncomp + 1) + nc + (ncomp + 1) + comp_faces;
  return sizeof(double) * (5 * nc + 6 * nf) + sizeof(int) * ni + nc;
}
// The whole arena.
size_t mp_arena_bytes(size_t nc, size_t nf, size_t ent, size_t ncomp, size_t comp_faces) {
  return (mp_input_bytes(nc, nf, ent, ncomp, comp_faces) + 15) / 16 * 16 + sizeof(double) * (4 * nf + 4 * nc) +
         sizeof(MpStatus);
}

bool MpScratch::reserve_caps() {
  const size_t nc = kMpMaxCells, nf = kMpMaxFaces;
  try {
    lut.reserve(kMpLutCap);
    tail.reserve(nf);
    head.reserve(nf);
    cell_off.reserve(nc + 1);
    cell_ent.reserve(2 * nf);
    fill.reserve(nc);
    parent.reserve(nc);
    root.reserve(nc);
    comp_of.reserve(nc);
    gauges.reserve(nc);
    comp_cell_off.reserve(nc + 1);
    comp_cells.reserve(nc);
    comp_face_off.reserve(nc + 1);
    comp_faces.reserve(2 * nf);
    host_in.reserve(mp_input_bytes(nc, nf, 2 * nf, nc, 2 * nf));
    anchored.reserve(nc);
    pinned.reserve(nc);
    host_out.reserve(4 * nc + nf + sizeof(MpStatus) / sizeof(double));
  } catch (...) {
    return false;
  }
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  arena_bytes = mp_arena_bytes(nc, nf, 2 * nf, nc, 2 * nf);
  if (cudaMalloc(&arena, arena_bytes) != cudaSuccess) {
    cudaGetLastError();
    arena = nullptr;
    arena_bytes = 0;
    return false;
  }
  return true;
}

void MpScratch::release() {
  if (arena) cudaFree(arena);
  arena = nullptr;
  arena_bytes = 0;
}

void MpScratch::destroy() {
  release();
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  e0 = e1 = nullptr;
}

}  // namespace fl

using namespace fl;

extern "C" int fl_project_mac_pressure_3d(double h, double dt, const int32_t* cell_index, const double* cell_values,
                                          uint64_t cell_count, const int32_t* face_index, const int32_t* face_kind,
                                          const double* face_values, uint64_t face_count, int max_iterations,
                                          double rel_tol, double* pressure, double* corrected_u, double* rhs,
                                          double* residual, double* defect, uint64_t* gauge_ordinals,
                                          fl_mac_pressure_diagnostics* diagnostics, fl_measurement* measurement) {
  MpScratch scratch;  // grows for this call and is released after it
  const int st = fl::mp_project(scratch, nullptr, h, dt, cell_index, cell_values, cell_count, face_index, face_kind,
                                face_values, face_count, max_iterations, rel_tol, pressure, corrected_u, rhs,
                                residual, defect, gauge_ordinals, diagnostics, measurement);
  scratch.destroy();
  return st;
}

namespace fl {

int mp_project(MpScratch& X, cudaStream_t stream, double h, double dt, const int32_t* cell_index,
               const double* cell_values, uint64_t cell_count, const int32_t* face_index, const int32_t* face_kind,
               const double* face_values, uint64_t face_count, int max_iterations, double rel_tol, double* pressure,
               double* corrected_u, double* rhs, double* residual, double* defect, uint64_t* gauge_ordinals,
               fl_mac_pressure_diagnostics* diagnostics, fl_measurement* measurement) {
  if (!(h > 0.0) || !std::isfinite(h) || !(dt > 0.0) || !std::isfinite(dt) || !(rel_tol >= 0.0) ||
      !std::isfinite(rel_tol))
    return FL_INVALID_ARGUMENT;
  if (cell_count == 0 || !cell_index || !cell_values || (face_count && (!face_index || !face_kind || !face_values)))
    return FL_INVALID_ARGUMENT;
  if (!pressure || !rhs || !residual || !defect || (face_count && !corrected_u)) return FL_INVALID_ARGUMENT;
  if (max_iterations < 1 || max_iterations > kMpMaxIterations) return FL_INVALID_ARGUMENT;
  if (cell_count > kMpMaxCells || face_count > kMpMaxFaces) return FL_RESOURCE_EXHAUSTED;
  const int nc = (int)cell_count, nf = (int)face_count;
  for (int i = 0; i < nc; ++i) {
    if (i > 0 && !cell_less(cell_index + 3 * (i - 1), cell_index + 3 * i)) return FL_INVALID_ARGUMENT;
    for (int k = 0; k < 5; ++k)
      if (!std::isfinite(cell_values[5 * i + k])) return FL_INVALID_ARGUMENT;
    if (!(cell_values[5 * i] > 0.0) || cell_values[5 * i + 2] < 0.0) return FL_INVALID_ARGUMENT;
  }
  // The faces must be exactly the cells' incident faces (six per cell, shared
  // faces once), unique and in the reference's owned-slot order, as
  // PrepareMacPressureSystem3D requires (mac_pressure_3d_system.cc:223-239).
  // Checked in the face loop below without building the incident set: the
  // owned-slot keys strictly increase, every face touches a listed cell, and
  // the faces' cell incidences number six per cell.
  for (int i = 0; i < nc; ++i)
    for (int a = 0; a < 3; ++a)
      if (cell_index[3 * i + a] == INT32_MAX) return FL_OUT_OF_RANGE;  // its high face is off the lattice
  // Cell lookups: a dense table over the cells' bounding box when it is small
  // enough, else a binary search of the sorted cells.
  int64_t lo[3], ext[3];
  for (int a = 0; a < 3; ++a) {
    int64_t mn = cell_index[a], mx = cell_index[a];
    for (int i = 1; i < nc; ++i) {
      mn = std::min<int64_t>(mn, cell_index[3 * i + a]);
      mx = std::max<int64_t>(mx, cell_index[3 * i + a]);
    }
    lo[a] = mn;
    ext[a] = mx - mn + 1;
  }
  const int64_t cap = (int64_t)kMpLutCap;
  const bool dense = ext[0] <= cap && ext[1] <= cap && ext[2] <= cap && ext[0] * ext[1] <= cap &&
                     ext[0] * ext[1] * ext[2] <= cap;
  auto& lut = X.lut;
  if (dense) {
    lut.assign((size_t)(ext[0] * ext[1] * ext[2]), -1);
    for (int i = 0; i < nc; ++i) {
      const int32_t* c = cell_index + 3 * i;
      lut[(size_t)(((c[2] - lo[2]) * ext[1] + (c[1] - lo[1])) * ext[0] + (c[0] - lo[0]))] = i;
    }
  }
  auto lookup = [&](int64_t x, int64_t y, int64_t z) {
    if (!dense) return find_cell(cell_index, nc, (int32_t)x, (int32_t)y, (int32_t)z);
    x -= lo[0];
    y -= lo[1];
    z -= lo[2];
    if (x < 0 || y < 0 || z < 0 || x >= ext[0] || y >= ext[1] || z >= ext[2]) return -1;
    return lut[(size_t)((z * ext[1] + y) * ext[0] + x)];
  };
  // Face endpoints and the link rules (internal: two cells; Dirichlet: one
  // cell and an open aperture; sealed: closed; the aperture within the full
  // face, mac_pressure_3d_arithmetic.h:182).
  auto& tail = X.tail;
  auto& head = X.head;
  tail.assign(nf, -1);
  head.assign(nf, -1);
  PackedFaceKey prev{0, 0};
  long long incidences = 0;
  for (int f = 0; f < nf; ++f) {
    const int32_t* fi = face_index + 4 * f;
    const double* v = face_values + 6 * f;
    if (fi[0] < 0 || fi[0] > 2 || face_kind[f] < kLinkSealed || face_kind[f] > kLinkDirichlet) return FL_INVALID_ARGUMENT;
    const PackedFaceKey key = packed_face_key(fi[0], fi[1], fi[2], fi[3]);
    if (f > 0 && !(prev < key)) return FL_INVALID_ARGUMENT;
    prev = key;
    for (int k = 0; k < 6; ++k)
      if (!std::isfinite(v[k])) return FL_INVALID_ARGUMENT;
    if (v[0] < 0.0 || v[0] > h * h) return FL_INVALID_ARGUMENT;
    int64_t tc[3] = {fi[1], fi[2], fi[3]};
    tc[fi[0]] -= 1;
    tail[f] = tc[fi[0]] < INT32_MIN ? -1 : lookup(tc[0], tc[1], tc[2]);
    head[f] = lookup(fi[1], fi[2], fi[3]);
    if (tail[f] < 0 && head[f] < 0) return FL_INVALID_ARGUMENT;
    incidences += (tail[f] >= 0) + (head[f] >= 0);
    const bool both = tail[f] >= 0 && head[f] >= 0, one = (tail[f] >= 0) != (head[f] >= 0);
    const int kind = face_kind[f];
    if (kind == kLinkInternal && !both) return FL_INVALID_ARGUMENT;
    if (kind == kLinkDirichlet && (!one || v[0] == 0.0)) return FL_INVALID_ARGUMENT;
    if (kind == kLinkSealed && v[0] != 0.0) return FL_INVALID_ARGUMENT;
    if (v[0] > 0.0 && !(v[2] > 0.0)) return FL_INVALID_ARGUMENT;
  }
  if (incidences != 6LL * nc) return FL_INVALID_ARGUMENT;
  int st = check_device();
  if (st != FL_OK) return st;
  // Per-cell face lists in increasing face order.
  auto& cell_off = X.cell_off;
  auto& cell_ent = X.cell_ent;
  cell_off.assign(nc + 1, 0);
  for (int f = 0; f < nf; ++f) {
    if (tail[f] >= 0) ++cell_off[tail[f] + 1];
    if (head[f] >= 0) ++cell_off[head[f] + 1];
  }
  for (int i = 0; i < nc; ++i) cell_off[i + 1] += cell_off[i];
  cell_ent.assign(std::max(cell_off[nc], 1), 0);
  {
    auto& fill = X.fill;
    fill.assign(cell_off.begin(), cell_off.end() - 1);
    for (int f = 0; f < nf; ++f) {
      if (tail[f] >= 0) cell_ent[fill[tail[f]]++] = f << 1;
      if (head[f] >= 0) cell_ent[fill[head[f]]++] = (f << 1) | 1;
    }
  }
  // Components over conducting two-cell faces (union towards the smaller
  // ordinal, so a component's root is its first cell); anchors are compliant
  // cells and Dirichlet faces; every unanchored component pins its root.
  auto& parent = X.parent;
  parent.resize(nc);
  for (int i = 0; i < nc; ++i) parent[i] = i;
  for (int f = 0; f < nf; ++f) {
    const double* v = face_values + 6 * f;
    const double cond = v[0] > 0.0 ? v[0] * ((dt * v[1]) / v[2]) : 0.0;
    if (cond > 0.0 && tail[f] >= 0 && head[f] >= 0) {
      const int a = find_root(parent, tail[f]), b = find_root(parent, head[f]);
      parent[std::max(a, b)] = std::min(a, b);
    }
  }
  auto& root = X.root;
  auto& anchored = X.anchored;
  auto& pinned = X.pinned;
  root.resize(nc);
  anchored.assign(nc, 0);
  pinned.assign(nc, 0);
  for (int i = 0; i < nc; ++i) {
    root[i] = find_root(parent, i);
    const double* v = cell_values + 5 * i;
    if (v[2] != 0.0 && v[0] / (v[2] * dt) > 0.0) anchored[root[i]] = 1;
  }
  for (int f = 0; f < nf; ++f)
    if (face_kind[f] == kLinkDirichlet) anchored[root[tail[f] >= 0 ? tail[f] : head[f]]] = 1;
  auto& comp_of = X.comp_of;
  auto& gauges = X.gauges;
  comp_of.assign(nc, -1);
  gauges.clear();
  for (int i = 0; i < nc; ++i)
    if (root[i] == i && !anchored[i]) {
      pinned[i] = 1;
      comp_of[i] = (int)gauges.size();
      gauges.push_back(i);
    }
  const int ncomp = (int)gauges.size();
  // Each unanchored component's cells (ascending) and its faces that do not
  // join two cells of the component (ascending), by counting then filling.
  auto& comp_cell_off = X.comp_cell_off;
  auto& comp_cells = X.comp_cells;
  auto& comp_face_off = X.comp_face_off;
  auto& comp_faces = X.comp_faces;
  comp_cell_off.assign(ncomp + 1, 0);
  comp_face_off.assign(ncomp + 1, 0);
  for (int i = 0; i < nc; ++i)
    if (comp_of[root[i]] >= 0) ++comp_cell_off[comp_of[root[i]] + 1];
  for (int f = 0; f < nf; ++f) {
    const int tl = tail[f], hd = head[f];
    if (tl >= 0 && hd >= 0 && root[tl] == root[hd]) continue;
    if (tl >= 0 && comp_of[root[tl]] >= 0) ++comp_face_off[comp_of[root[tl]] + 1];
    if (hd >= 0 && comp_of[root[hd]] >= 0) ++comp_face_off[comp_of[root[hd]] + 1];
  }
  for (int k = 0; k < ncomp; ++k) {
    comp_cell_off[k + 1] += comp_cell_off[k];
    comp_face_off[k + 1] += comp_face_off[k];
  }
  comp_cells.assign(comp_cell_off[ncomp], 0);
  comp_faces.assign(comp_face_off[ncomp], 0);
  {
    auto& fill = X.fill;
    fill.assign(comp_cell_off.begin(), comp_cell_off.end() - 1);
    for (int i = 0; i < nc; ++i)
      if (comp_of[root[i]] >= 0) comp_cells[fill[comp_of[root[i]]]++] = i;
    fill.assign(comp_face_off.begin(), comp_face_off.end() - 1);
    for (int f = 0; f < nf; ++f) {
      const int tl = tail[f], hd = head[f];
      if (tl >= 0 && hd >= 0 && root[tl] == root[hd]) continue;
      if (tl >= 0 && comp_of[root[tl]] >= 0) comp_faces[fill[comp_of[root[tl]]]++] = f << 1;
      if (hd >= 0 && comp_of[root[hd]] >= 0) comp_faces[fill[comp_of[root[hd]]]++] = (f << 1) | 1;
    }
  }
  // One device arena: inputs, index lists, work arrays and the status.
  const size_t bytes = mp_arena_bytes(nc, nf, cell_ent.size(), ncomp, comp_faces.size());
  if (X.arena_bytes < bytes) {
    X.release();
    if (cudaMalloc(&X.arena, bytes) != cudaSuccess) {
      cudaGetLastError();
      X.arena = nullptr;
      return FL_RESOURCE_EXHAUSTED;
    }
    X.arena_bytes = bytes;
  }
  if (!X.e0 && (cudaEventCreate(&X.e0) != cudaSuccess || cudaEventCreate(&X.e1) != cudaSuccess)) {
    cudaGetLastError();
    return FL_INTERNAL;
  }
  MpSystem S{};
  S.nc = nc;
  S.nf = nf;
  S.ncomp = ncomp;
  S.h = h;
  S.dt = dt;
  S.rel_tol = rel_tol;
  S.max_iterations = max_iterations;
  // The arena: the inputs (values, index lists, pins), sent as one copy, then the
  // work arrays, then the results and the status, fetched as one copy.
  auto& host_in = X.host_in;
  host_in.clear();
  auto put = [&](const void* src, size_t n) {
    const size_t at = host_in.size();
    const unsigned char* b = static_cast<const unsigned char*>(src);
    host_in.insert(host_in.end(), b, b + n);
    return X.arena + at;
  };
  auto put_d = [&](const double* src, size_t n) { return reinterpret_cast<const double*>(put(src, sizeof(double) * n)); };
  auto put_i = [&](const int* src, size_t n) { return reinterpret_cast<const int*>(put(src, sizeof(int) * n)); };
  S.cell_values = put_d(cell_values, (size_t)5 * nc);
  S.face_values = put_d(face_values, (size_t)6 * nf);
  S.face_kind = put_i(face_kind, nf);
  S.tail = put_i(tail.data(), nf);
  S.head = put_i(head.data(), nf);
  S.cell_ent = put_i(cell_ent.data(), cell_ent.size());
  S.root = put_i(root.data(), nc);
  S.comp_cell_off = put_i(comp_cell_off.data(), ncomp + 1);
  S.comp_cells = put_i(comp_cells.data(), comp_cells.size());
  S.comp_face_off = put_i(comp_face_off.data(), ncomp + 1);
  S.comp_faces = put_i(comp_faces.data(), comp_faces.size());
  S.pinned = reinterpret_cast<const unsigned char*>(put(pinned.data(), nc));
  double* dp = reinterpret_cast<double*>(X.arena + (host_in.size() + 15) / 16 * 16);
  auto take_d = [&](size_t n) {
    double* r = dp;
    dp += n;
    return r;
  };
  S.scale = take_d(nf);
  S.cond = take_d(nf);
  S.wall_face = take_d(nf);
  S.rhs = take_d(nc);
  S.p = take_d(nc);
  S.residual = take_d(nc);
  S.defect = take_d(nc);
  S.corrected_u = take_d(nf);
  S.out = reinterpret_cast<MpStatus*>(dp);
  auto& host_out = X.host_out;  // rhs, p, residual, defect, corrected_u, status
  const size_t results = (size_t)4 * nc + nf;
  host_out.resize(results + sizeof(MpStatus) / sizeof(double));
  cudaStream_t s = stream;
  float ms = 0.0f;
  bool ok = cudaMemcpyAsync(X.arena, host_in.data(), host_in.size(), cudaMemcpyHostToDevice, s) == cudaSuccess &&
            cudaEventRecord(X.e0, s) == cudaSuccess;
  if (ok) {
    ++g_kernel_launches;
    k_mac_pressure<<<kMpCtas, kMpThreads, 0, s>>>(S);
    ok = cudaGetLastError() == cudaSuccess && cudaEventRecord(X.e1, s) == cudaSuccess &&
         cudaMemcpyAsync(host_out.data(), S.rhs, sizeof(double) * results + sizeof(MpStatus), cudaMemcpyDeviceToHost,
                         s) == cudaSuccess &&
         cudaStreamSynchronize(s) == cudaSuccess && cudaEventElapsedTime(&ms, X.e0, X.e1) == cudaSuccess;
  }
  if (!ok) {
    cudaGetLastError();
    return FL_INTERNAL;
  }
  MpStatus res;
  std::memcpy(&res, host_out.data() + results, sizeof(MpStatus));
  if (diagnostics) {
    diagnostics->iterations = (uint64_t)res.iterations;
    diagnostics->true_residual_l2 = res.true_residual_l2;
    diagnostics->max_volume_scaled_residual = res.max_volume_scaled_residual;
    diagnostics->max_cell_constraint_defect = res.max_defect;
    diagnostics->rhs_l2 = res.rhs_l2;
    diagnostics->gauge_count = (uint64_t)ncomp;
  }
  if (measurement) {
    measurement->compiled_architecture = res.arch;
    measurement->kernel_ms = ms;
  }
  if (res.status != FL_OK) return res.status;  // no projection is published
  const double* r = host_out.data();
  std::memcpy(rhs, r, sizeof(double) * nc);
  std::memcpy(pressure, r + nc, sizeof(double) * nc);
  std::memcpy(residual, r + 2 * nc, sizeof(double) * nc);
  std::memcpy(defect, r + 3 * nc, sizeof(double) * nc);
  if (nf) std::memcpy(corrected_u, r + 4 * nc, sizeof(double) * nf);
  if (gauge_ordinals)
    for (int k = 0; k < ncomp; ++k) gauge_ordinals[k] = (uint64_t)gauges[k];
  return FL_OK;
}

}  // namespace fl
