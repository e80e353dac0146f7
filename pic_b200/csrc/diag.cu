// diag.cu -- device diagnostics of the reference's output routines, computed
// where the data already is (HBM); only the result crosses to the host.
//
//   pic_average_x        Average_x profiles (In-Output/Output_To_Tecplot_IJK_2D.f90:
//                        166-226): the mean of each node field over the nodes of
//                        one mesh column x = x_i, in the file's output scaling.
//   pic_energy_spectrum  Output_Energy.f90:41-71: per-species counts of the
//                        particle energy (eV) in (E_max (b-1)/N, E_max b/N] and
//                        of vx in (V_max (b-1-N/2)/N, V_max (b-N/2)/N].
//   pic_velocity_moments OUTPUT_velocity.f90:48-103: per x-column (floor(X))
//                        particle counts, drift velocity (mean) and thermal
//                        velocity (standard deviation), two passes.
//
// Counts are integers and bit-exact.  The column means sum each column in the
// reference's node order (j ascending) one thread per column, so they are
// bit-exact too.  The velocity sums are FP64 atomics (the reference sums in
// FP32, sequentially): their order, and so their last bits, vary run to run.
// Compiled with --fmad=false like the rest of the library: the absolute
// position rebuilt from a mixed-precision particle equals the one the
// download path writes.
#include <algorithm>
#include <cmath>
#include <vector>

#include "pic_ctx.h"

namespace pic {

namespace {

constexpr int kMaxProfileCols = 3 + 3 * PIC_MAX_SPECIES;

struct ProfK {
  const double *f[kMaxProfileCols];  // null: the column's x coordinate
  double scale[kMaxProfileCols];
  int ncols, nnx, nny;
  const double *xs;
  double *out;  // [ncols][nnx]
};

// Output_To_Tecplot_IJK_2D.f90:184-215: a column's nodes in node order,
// summed, divided by their count, then scaled for the file (:220-223).  The
// sum of a column is one chain (the reference's order), so a thread takes a
// column; its nodes are contiguous, so the block loads tiles of 32 columns x
// 32 nodes with whole lines and the chains read them from shared memory, the
// next tile's loads in flight behind them (a thread a column straight from
// memory touched 32 lines a load: 25 -> 8 us at 257 x 257, nine quantities).
constexpr int kAvgCols = 32, kAvgRows = 32, kAvgThreads = 256;

__global__ void __launch_bounds__(kAvgThreads) k_average_x(ProfK k) {
  __shared__ double tile[2][kAvgCols][kAvgRows + 1];
  const int c = blockIdx.y, i0 = blockIdx.x * kAvgCols;
  const int j = threadIdx.x % kAvgRows, w = threadIdx.x / kAvgRows;  // w: 8 columns apart by kAvgThreads / 32
  constexpr int NL = kAvgCols * kAvgRows / kAvgThreads;
  double s = 0.0;
  if (k.f[c]) {
    double v[NL];
    auto load = [&](int j0) {
#pragma unroll
      for (int q = 0; q < NL; ++q) {
        const int i = i0 + w + q * (kAvgThreads / kAvgRows);
        v[q] = i < k.nnx && j0 + j < k.nny ? k.f[c][(size_t)i * k.nny + j0 + j] : 0.0;
      }
    };
    load(0);
    int buf = 0;
    for (int j0 = 0; j0 < k.nny; j0 += kAvgRows, buf ^= 1) {
#pragma unroll
      for (int q = 0; q < NL; ++q) tile[buf][w + q * (kAvgThreads / kAvgRows)][j] = v[q];
      __syncthreads();
      if (j0 + kAvgRows < k.nny) load(j0 + kAvgRows);
      if (threadIdx.x < kAvgCols) {
        const int m = min(kAvgRows, k.nny - j0);
        for (int q = 0; q < m; ++q) s = s + tile[buf][threadIdx.x][q];
      }
    }
  }
  const int i = i0 + threadIdx.x;
  if (threadIdx.x >= kAvgCols || i >= k.nnx) return;
  k.out[(size_t)c * k.nnx + i] = k.f[c] ? (s / (double)k.nny) * k.scale[c] : k.xs[i] * k.scale[c];
}

// One species' particle arrays; FP32 data in the first half of the double
// storage for F32 kernels (x, y then hold the offsets inside the element loc).
struct PartK {
  const double *x, *vx, *vy, *vz;
  const int32_t *loc;
  int64_t n;
  int ney;
  double xmin, hx;
};

template <bool F32>
__device__ __forceinline__ double vget(const double *a, int64_t p) {
  if constexpr (F32) return (double)reinterpret_cast<const float *>(a)[p];
  else return a[p];
}

// absolute x of a live particle, as the download path writes it
template <bool F32>
__device__ __forceinline__ double xget(const PartK &s, int64_t p, int e) {
  const double x = vget<F32>(s.x, p);
  if constexpr (!F32) return x;
  return s.xmin + ((double)(e / s.ney) + x) * s.hx;
}

// reference bin edges, evaluated in the reference's order
__device__ __forceinline__ double e_edge(double e_max, int i, int n) { return (e_max * (double)i) / (double)n; }
__device__ __forceinline__ double v_edge(double v_max, int i, int n) {
  return (v_max * (double)((float)i - 0.5f * (float)n)) / (double)n;
}

// the bin b (0-based) of (edge[b], edge[b+1]] that holds v, or -1.  t is
// v's position in bin widths from edge[0] (a product with a reciprocal, good
// to a few ulps); the candidate and its two neighbours are checked against
// the exact edges.
__device__ __forceinline__ int find_bin(double v, double t, const double *edge, int n) {
  if (!(t > -2.0) || !(t < n + 2.0)) return -1;
  const int b0 = (int)floor(t);
  for (int b = max(b0 - 1, 0); b <= min(b0 + 1, n - 1); ++b)
    if (v <= edge[b + 1] && v > edge[b]) return b;
  return -1;
}

// The bin of a value at t bin widths from edge[0] where t decides it: off
// every edge by far more than the few ulps t and the edges are good to (edges
// within 4096 bins: 1e-12 widths).  -1: outside; -2: too near an edge.
__device__ __forceinline__ int clear_bin(double t, int n) {
  if (!(t > -2.0) || !(t < n + 2.0)) return t == t ? -1 : -2;
  const double f = floor(t);
  if (t - f < 1e-6 || t - f > 1.0 - 1e-6) return -2;
  return f >= 0.0 && f < (double)n ? (int)f : -1;
}

// add 1 to sh[bin] for every lane with bin >= 0; all 32 lanes call it.  The
// lanes that share lane 0's bin (most of them in a narrow distribution, ions
// in electron bins) count as one; the others add their own.
__device__ __forceinline__ void warp_count(unsigned int *sh, int bin) {
  const int b0 = __shfl_sync(0xffffffffu, bin, 0);
  const unsigned same = __ballot_sync(0xffffffffu, bin == b0);
  if (bin < 0) return;
  if (bin != b0) atomicAdd(&sh[bin], 1u);
  else if ((threadIdx.x & 31) == 0) atomicAdd(&sh[bin], (unsigned)__popc(same));
}

struct SpecK {
  PartK s;
  int nbins;
  double mass, vref, e_max, v_max;
  double e_inv, v_inv;  // nbins / e_max, nbins / v_max
  double ej_inv;        // nbins / (e_max J_to_eV); NaN (no bin is clear) where that could underflow
  unsigned long long *ce, *cv;
};

// Output_Energy.f90:55-71 for one species.  The grid-stride loop runs the
// same number of iterations on every lane of a warp (the base index is
// uniform), so the whole-warp votes are legal.  HBM-bound in aim (28 B a
// particle FP64); 80 -> 42 us for 5.7M FP64 particles against a division, two
// edge searches and two whole-warp matches a particle.
constexpr int kSpecBatch = 4;  // particles a lane has in flight

template <bool F32>
__global__ void __launch_bounds__(256) k_spectrum(SpecK k) {
  extern __shared__ double edges[];  // [nbins+1] energy, [nbins+1] vx edges, then [2][nbins] counts
  double *ee = edges, *ve = edges + k.nbins + 1;
  unsigned int *sh = reinterpret_cast<unsigned int *>(edges + 2 * (k.nbins + 1));
  for (int b = threadIdx.x; b <= k.nbins; b += blockDim.x) {
    ee[b] = e_edge(k.e_max, b, k.nbins);
    ve[b] = v_edge(k.v_max, b, k.nbins);
  }
  for (int b = threadIdx.x; b < 2 * k.nbins; b += blockDim.x) sh[b] = 0u;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < k.s.n; base += kSpecBatch * stride) {
    double v[kSpecBatch][3];
    int e[kSpecBatch];
#pragma unroll
    for (int u = 0; u < kSpecBatch; ++u) {
      const int64_t p = base + u * stride + threadIdx.x;
      e[u] = -1;
      v[u][0] = v[u][1] = v[u][2] = 0.0;
      if (p < k.s.n) {
        e[u] = k.s.loc[p];
        v[u][0] = vget<F32>(k.s.vx, p);
        v[u][1] = vget<F32>(k.s.vy, p);
        v[u][2] = vget<F32>(k.s.vz, p);
      }
    }
#pragma unroll
    for (int u = 0; u < kSpecBatch; ++u) {
      int be = -1, bv = -1;
      if (e[u] >= 0) {
        const double vx = v[u][0], vy = v[u][1], vz = v[u][2];
        // ParticleOne.f90:235-244 EnergyParticleOne with VFactor, then / JtoeV;
        // the division and the edges only where they can decide the bin
        const double ej = (((0.5 * k.mass) * ((vx * vx + vy * vy) + vz * vz)) * k.vref) * k.vref;
        const double tv = vx * k.v_inv + 0.5 * k.nbins;
        be = clear_bin(ej * k.ej_inv, k.nbins);
        if (be == -2) {
          const double ev = ej / PIC_JTOEV;
          be = find_bin(ev, ev * k.e_inv, ee, k.nbins);
        }
        bv = clear_bin(tv, k.nbins);
        if (bv == -2) bv = find_bin(vx, tv, ve, k.nbins);
      }
      warp_count(sh, be);
      warp_count(sh + k.nbins, bv);
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < k.nbins; b += blockDim.x) {
    if (sh[b]) atomicAdd(k.ce + b, (unsigned long long)sh[b]);
    if (sh[k.nbins + b]) atomicAdd(k.cv + b, (unsigned long long)sh[k.nbins + b]);
  }
}

struct MomK {
  PartK s;
  int nbins;
  unsigned long long *count;  // [nbins]
  double *sum;                // [3][nbins] velocity sums, then variance sums
  const double *drift;        // [3][nbins] (second pass)
};

__device__ __forceinline__ int x_bin(double X, int nbins) {
  // OUTPUT_velocity.f90:57 num = MIN(MAX(1, FLOOR(X)+1), N), 0-based here
  const double f = floor(X);
  if (!(f >= 0.0)) return 0;
  if (f >= (double)(nbins - 1)) return nbins - 1;
  return (int)f;
}

// pass 1 (OUTPUT_velocity.f90:55-63): count and velocity sums per column;
// pass 2 (:80-87, kSecond): sums of (v - drift)^2.
//
// Every warp takes one contiguous run of particles.  They are sorted by cell,
// so a run stays within one x column, or two neighbours where a column's edge
// (one Debye length, about one cell) crosses the cells, for a long time: the
// lanes sum those two columns (base, base + 1) in registers and the warp adds
// them to the CTA's shared sums only when a batch has left them.  HBM-bound in
// aim (36 B a particle FP64).  Both passes of a call, 5.2 to 5.7M FP64
// particles (us: warp sums of every 32 particles; two columns that moved at
// every lane outside, which added its own; now):
//   sorted, cells of half a column, 500 columns           262   185   184
//   ten steps after the sort                              553   568   247
//   random order, 500 columns / 64 columns            258/713 327/838 237/505
//   sorted, cells of 1.9 columns, 500 / 8 columns     524/280 480/388 241/214
// (the last: colliding adds, in the few warps that have them as long as all)
constexpr int kMomBatch = 2;  // particles a lane has in flight
constexpr int kMomShare = 4;  // lanes outside in one column whose values the warp sums

template <bool kSecond, bool F32>
__global__ void __launch_bounds__(256, 4) k_vmoments(MomK k) {
  extern __shared__ double shd[];  // [3][nbins] sums, then [3][nbins] drift (pass 2) or [nbins] counts
  double *acc = shd;
  double *dr = shd + 3 * k.nbins;
  unsigned int *cnt = reinterpret_cast<unsigned int *>(shd + 3 * k.nbins);
  for (int b = threadIdx.x; b < 3 * k.nbins; b += blockDim.x) {
    acc[b] = 0.0;
    if (kSecond) dr[b] = k.drift[b];
  }
  if (!kSecond)
    for (int b = threadIdx.x; b < k.nbins; b += blockDim.x) cnt[b] = 0u;
  __syncthreads();
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  const int64_t w = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int64_t run = ((k.s.n + warps - 1) / warps + 32 * kMomBatch - 1) / (32 * kMomBatch) * (32 * kMomBatch);
  const int64_t p1 = min(k.s.n, (w + 1) * run);
  int base = -2;
  double s0[3] = {0.0, 0.0, 0.0}, s1[3] = {0.0, 0.0, 0.0}, d0[3], d1[3];
  unsigned c0 = 0, c1 = 0;
  auto rebase = [&](int b) {  // every lane of the warp, the same b
    if (base >= 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        for (int o = 16; o > 0; o >>= 1) {
          s0[c] += __shfl_xor_sync(full, s0[c], o);
          s1[c] += __shfl_xor_sync(full, s1[c], o);
        }
        if (lane == 0) {
          atomicAdd(&acc[c * k.nbins + base], s0[c]);
          if (base + 1 < k.nbins) atomicAdd(&acc[c * k.nbins + base + 1], s1[c]);
        }
        s0[c] = s1[c] = 0.0;
      }
      if (!kSecond) {
        c0 = __reduce_add_sync(full, c0);
        c1 = __reduce_add_sync(full, c1);
        if (lane == 0) {
          atomicAdd(&cnt[base], c0);
          if (base + 1 < k.nbins) atomicAdd(&cnt[base + 1], c1);
        }
        c0 = c1 = 0;
      }
    }
    base = b;
    if (kSecond && b >= 0)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        d0[c] = dr[c * k.nbins + b];
        d1[c] = b + 1 < k.nbins ? dr[c * k.nbins + b + 1] : 0.0;
      }
  };
  for (int64_t q = w * run; q < p1; q += 32 * kMomBatch) {
    int b[kMomBatch];
    double v[kMomBatch][3];
#pragma unroll
    for (int u = 0; u < kMomBatch; ++u) {
      const int64_t p = q + 32 * u + lane;
      b[u] = -1;
      v[u][0] = v[u][1] = v[u][2] = 0.0;
      if (p < p1) {
        const int e = k.s.loc[p];
        const double X = xget<F32>(k.s, p, max(e, 0));
        v[u][0] = vget<F32>(k.s.vx, p);
        v[u][1] = vget<F32>(k.s.vy, p);
        v[u][2] = vget<F32>(k.s.vz, p);
        if (e >= 0) b[u] = x_bin(X, k.nbins);
      }
    }
#pragma unroll
    for (int u = 0; u < kMomBatch; ++u) {
      // the two columns move on to the lowest of the batch where the new two
      // hold every live lane, or most of them with most of them gone from the
      // old: a run of sorted particles that crosses into its next column.
      // Particles in no order have no such pair.
      const unsigned left = __ballot_sync(full, b[u] >= 0 && b[u] != base && b[u] != base + 1);
      if (left) {
        const int live = __popc(__ballot_sync(full, b[u] >= 0));
        const int lo = (int)__reduce_min_sync(full, b[u] >= 0 ? (unsigned)b[u] : 0xffffffffu);
        const int held = __popc(__ballot_sync(full, b[u] >= 0 && b[u] <= lo + 1));
        if (held == live || (2 * held > live && 2 * __popc(left) > live)) rebase(lo);
      }
      const bool in0 = b[u] >= 0 && b[u] == base, in1 = b[u] >= 0 && b[u] == base + 1;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double t0 = v[u][c], t1 = v[u][c];
        if (kSecond) {
          t0 = v[u][c] - d0[c];
          t1 = v[u][c] - d1[c];
          t0 = t0 * t0;
          t1 = t1 * t1;
        }
        s0[c] += in0 ? t0 : 0.0;
        s1[c] += in1 ? t1 : 0.0;
      }
      c0 += in0 ? 1u : 0u;
      c1 += in1 ? 1u : 0u;
      // the lanes outside: columns that several of them share (cells wider than
      // a column or two) as one sum of the warp, the others on their own
      unsigned out = __ballot_sync(full, b[u] >= 0 && !in0 && !in1);
      if (out) {
        const bool mine = out >> lane & 1;
        double t[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double d = kSecond && mine ? v[u][c] - dr[c * k.nbins + b[u]] : 0.0;
          t[c] = kSecond ? d * d : v[u][c];
        }
        while (out) {
          const int first = __ffs(out) - 1, col = __shfl_sync(full, b[u], first);
          const unsigned share = __ballot_sync(full, b[u] == col);
          if (__popc(share) < kMomShare) break;
          double a[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            a[c] = share >> lane & 1 ? t[c] : 0.0;
            for (int o = 16; o > 0; o >>= 1) a[c] += __shfl_xor_sync(full, a[c], o);
          }
          if (lane == first) {
#pragma unroll
            for (int c = 0; c < 3; ++c) atomicAdd(&acc[c * k.nbins + col], a[c]);
            if (!kSecond) atomicAdd(&cnt[col], (unsigned)__popc(share));
          }
          out &= ~share;
        }
        if (out >> lane & 1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) atomicAdd(&acc[c * k.nbins + b[u]], t[c]);
          if (!kSecond) atomicAdd(&cnt[b[u]], 1u);
        }
      }
    }
  }
  rebase(-2);
  __syncthreads();
  for (int b = threadIdx.x; b < 3 * k.nbins; b += blockDim.x)
    if (acc[b] != 0.0) atomicAdd(&k.sum[b], acc[b]);
  if (!kSecond)
    for (int b = threadIdx.x; b < k.nbins; b += blockDim.x)
      if (cnt[b]) atomicAdd(&k.count[b], (unsigned long long)cnt[b]);
}

// OUTPUT_velocity.f90:64-76 (drift = sum / count, 0 for an empty column) and
// :88-103 (thermal = sqrt(variance sum / count))
__global__ void k_vmoments_div(const unsigned long long *count, const double *sum, double *out, int nbins, int root) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3 * nbins) return;
  const unsigned long long c = count[t % nbins];
  double v = 0.0;
  if (c != 0ull) {
    v = sum[t] / (double)c;
    if (root) v = sqrt(v);
  }
  out[t] = v;
}

PartK part_k(const Species &s) {
  PartK p;
  p.x = s.x;
  p.vx = s.vx;
  p.vy = s.vy;
  p.vz = s.vz;
  p.loc = s.loc;
  p.n = s.n_slots;
  p.ney = g.m.ney;
  p.xmin = g.m.xmin;
  p.hx = g.m.hx;
  return p;
}

// CTAs of one wave (all resident at once), fewer for few particles
template <class K>
int grid_for(K kernel, size_t smem, int64_t n, unsigned *grid) {
  int dev = 0, nsm = 0, per_sm = 1;
  PIC_CUDA(cudaGetDevice(&dev));
  PIC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  PIC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t all = blocks_for(n, 256);
  if (all > nsm) PIC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, smem));
  *grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(all, (int64_t)nsm * std::max(per_sm, 1)));
  return PIC_OK;
}

// device scratch for the diagnostics, grown on demand and freed at finalize
struct DiagScratch {
  void *p = nullptr;
  size_t bytes = 0;
} g_diag;

int scratch(size_t bytes, void **out) {
  if (bytes > g_diag.bytes) {
    if (g_diag.p) cudaFree(g_diag.p);
    g_diag.p = nullptr;
    g_diag.bytes = 0;
    PIC_CUDA(cudaMalloc(&g_diag.p, bytes));
    g_diag.bytes = bytes;
  }
  *out = g_diag.p;
  return PIC_OK;
}

}  // namespace

void diag_free() {
  if (g_diag.p) cudaFree(g_diag.p);
  g_diag.p = nullptr;
  g_diag.bytes = 0;
}

}  // namespace pic

using namespace pic;

extern "C" {

int pic_average_x(double *out) {
  if (!g.inited) {
    set_error("pic_average_x: library not initialised (pic_init)");
    return PIC_ERR_STATE;
  }
  if (int rc = fields_fence(0x3u)) return rc;  // reads rho and phi: after a queued upload
  if (!out) {
    set_error("pic_average_x: null output");
    return PIC_ERR_ARG;
  }
  ProfK k;
  std::memset(&k, 0, sizeof k);
  // the file's columns (Output_To_Tecplot_IJK_2D.f90:219-223): x, Phi, Rho,
  // Rho_s per species, Ek_s per species, Ek_tot per species
  int c = 0;
  auto col = [&](const double *f, double scale) {
    k.f[c] = f;
    k.scale[c] = scale;
    ++c;
  };
  col(nullptr, g.L_ref);
  col(g.d_phi, g.phi_ref);
  col(g.d_rho, g.P.n_ref);
  for (int s = 0; s < g.ns; ++s) col(g.sp[s].rho_s, g.P.n_ref);
  for (int s = 0; s < g.ns; ++s) col(g.sp[s].ek_s, 1.0);
  for (int s = 0; s < g.ns; ++s) col(g.sp[s].ek_tot, 1.0);
  k.ncols = c;
  k.nnx = g.m.nnx;
  k.nny = g.m.nny;
  k.xs = g.d_xs;
  int rc;
  void *d = nullptr;
  const size_t bytes = (size_t)c * g.m.nnx * sizeof(double);
  if ((rc = scratch(bytes, &d))) return rc;
  k.out = static_cast<double *>(d);
  k_average_x<<<dim3((g.m.nnx + kAvgCols - 1) / kAvgCols, c), kAvgThreads, 0, g.st>>>(k);
  PIC_LAUNCHED();
  PIC_CUDA(cudaMemcpyAsync(out, d, bytes, cudaMemcpyDeviceToHost, g.st));
  PIC_CUDA(cudaStreamSynchronize(g.st));
  return PIC_OK;
}

int pic_energy_spectrum(int32_t species, int32_t nbins, double e_max_ev, double v_max, int64_t *count_e,
                        int64_t *count_vx) {
  if (!g.inited) {
    set_error("pic_energy_spectrum: library not initialised (pic_init)");
    return PIC_ERR_STATE;
  }
  if (species < 0 || species >= g.ns || nbins < 1 || nbins > 4096 || !(e_max_ev > 0) || !(v_max > 0) ||
      !count_e || !count_vx) {
    set_error("pic_energy_spectrum: bad arguments");
    return PIC_ERR_ARG;
  }
  const Species &s = g.sp[species];
  int rc;
  void *d = nullptr;
  const size_t bytes = 2 * (size_t)nbins * sizeof(unsigned long long);
  if ((rc = scratch(bytes, &d))) return rc;
  unsigned long long *cnt = static_cast<unsigned long long *>(d);
  PIC_CUDA(cudaMemsetAsync(cnt, 0, bytes, g.st));
  if (s.n_slots > 0) {
    SpecK k{part_k(s), nbins, s.mass, g.v_ref, e_max_ev, v_max, nbins / e_max_ev, nbins / v_max,
            e_max_ev > 1e-200 ? nbins / (e_max_ev * PIC_JTOEV) : std::nan(""), cnt, cnt + nbins};
    const size_t shb = 2 * (nbins + 1) * sizeof(double) + 2 * nbins * sizeof(unsigned int);
    const auto fn = s.f32 ? k_spectrum<true> : k_spectrum<false>;
    unsigned grid = 0;
    if ((rc = grid_for(fn, shb, s.n_slots, &grid))) return rc;
    fn<<<grid, 256, shb, g.st>>>(k);
    PIC_LAUNCHED();
  }
  std::vector<unsigned long long> h(2 * (size_t)nbins);
  PIC_CUDA(cudaMemcpyAsync(h.data(), cnt, bytes, cudaMemcpyDeviceToHost, g.st));
  PIC_CUDA(cudaStreamSynchronize(g.st));
  for (int b = 0; b < nbins; ++b) {
    count_e[b] = (int64_t)h[b];
    count_vx[b] = (int64_t)h[nbins + b];
  }
  return PIC_OK;
}

int pic_velocity_moments(int32_t species, int32_t nbins, int64_t *count, double *drift, double *thermal) {
  if (!g.inited) {
    set_error("pic_velocity_moments: library not initialised (pic_init)");
    return PIC_ERR_STATE;
  }
  if (species < 0 || species >= g.ns || nbins < 1 || nbins > 2048 || !count || !drift || !thermal) {
    set_error("pic_velocity_moments: bad arguments");
    return PIC_ERR_ARG;
  }
  const Species &s = g.sp[species];
  const size_t nb = (size_t)nbins;
  // count [nb] u64, sums [3nb], drift [3nb], thermal [3nb]
  int rc;
  void *d = nullptr;
  if ((rc = scratch(nb * 8 * 10, &d))) return rc;
  unsigned long long *cnt = static_cast<unsigned long long *>(d);
  double *sum = reinterpret_cast<double *>(cnt + nb), *dr = sum + 3 * nb, *th = dr + 3 * nb;
  PIC_CUDA(cudaMemsetAsync(d, 0, nb * 8 * 4, g.st));
  const size_t sh1 = 3 * nb * sizeof(double) + nb * sizeof(unsigned int), sh2 = 6 * nb * sizeof(double);
  const auto fn1 = s.f32 ? k_vmoments<false, true> : k_vmoments<false, false>;
  const auto fn2 = s.f32 ? k_vmoments<true, true> : k_vmoments<true, false>;
  unsigned grid1 = 0, grid2 = 0;
  if ((rc = grid_for(fn1, sh1, s.n_slots, &grid1)) || (rc = grid_for(fn2, sh2, s.n_slots, &grid2))) return rc;
  MomK k{part_k(s), nbins, cnt, sum, dr};
  const unsigned gdiv = (unsigned)((3 * nb + 255) / 256);
  if (s.n_slots > 0) {
    fn1<<<grid1, 256, sh1, g.st>>>(k);
    PIC_LAUNCHED();
  }
  k_vmoments_div<<<gdiv, 256, 0, g.st>>>(cnt, sum, dr, nbins, 0);
  PIC_LAUNCHED();
  PIC_CUDA(cudaMemsetAsync(sum, 0, 3 * nb * sizeof(double), g.st));
  if (s.n_slots > 0) {
    fn2<<<grid2, 256, sh2, g.st>>>(k);
    PIC_LAUNCHED();
  }
  k_vmoments_div<<<gdiv, 256, 0, g.st>>>(cnt, sum, th, nbins, 1);
  PIC_LAUNCHED();
  std::vector<unsigned long long> hc(nb);
  PIC_CUDA(cudaMemcpyAsync(hc.data(), cnt, nb * 8, cudaMemcpyDeviceToHost, g.st));
  PIC_CUDA(cudaMemcpyAsync(drift, dr, 3 * nb * 8, cudaMemcpyDeviceToHost, g.st));
  PIC_CUDA(cudaMemcpyAsync(thermal, th, 3 * nb * 8, cudaMemcpyDeviceToHost, g.st));
  PIC_CUDA(cudaStreamSynchronize(g.st));
  for (size_t b = 0; b < nb; ++b) count[b] = (int64_t)hc[b];
  return PIC_OK;
}

}  // extern "C"
