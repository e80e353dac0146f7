// noalloc.cu -- charge deposit of one species that allocates no memory.
//
// Some callers cannot allocate device memory: a host program whose memory
// pool is owned by another framework (for example a Fortran code whose
// device memory all comes from one pre-sized arena), a real-time loop that
// must not pay for the implicit device synchronisation of cudaMalloc, or a
// process that has already reserved the whole device.  pic_deposit_noalloc
// serves them: the caller passes its own input and output device buffers and
// the int64 fixed-point accumulator lives in a file-scope __device__ array
// of fixed size, so no call allocates or frees anything.
//
// The arithmetic is the one of the GetParChg_2D path of libpicgpu (locate,
// bilinear weights, 2^-40 fixed point with each particle depositing exactly
// 2^40, normalisation by the dual volume), so
// on a Cartesian mesh with FP64 positions the result equals pic_get_par_chg's
// per-species density bit for bit.  It has no r-z (delta 1) weighting and
// takes no FP32 element offsets (the mixed-precision particle layout).
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <string>

#include "../../include/picgpu.h"
#include "div_dev.h"
#include "pic_common.h"

namespace pic {
void set_error(const std::string &msg);
}

// Scratch: one int64 accumulator per mesh node, at most PIC_NOALLOC_MAX_NODES
// nodes (4 MiB).  Every device that loads the library holds it until exit.
static __device__ __align__(256) unsigned long long g_noalloc_acc[PIC_NOALLOC_MAX_NODES];

namespace {

constexpr int kMaxDevices = 64;
// Device address of g_noalloc_acc per device ordinal, looked up on the first
// call with that device current.  Atomic: host threads driving different
// devices may make their first calls at the same time.
std::atomic<unsigned long long *> g_acc_ptr[kMaxDevices];

__global__ void k_na_clear(unsigned long long *acc, int64_t nn) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nn) acc[i] = 0ull;
}

// Sums over lanes [lane, seg_end] of one segment, toward its head.
__device__ __forceinline__ void seg_sums4(long long (&v)[4], int lane, int seg_end, int maxlen) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    if (off >= maxlen) break;
    const bool take = lane + off <= seg_end;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const long long o = __shfl_down_sync(0xffffffffu, v[c], off);
      if (take) v[c] += o;
    }
  }
}

__device__ __forceinline__ void na_add(unsigned long long *acc, int n1, int nny, const long long (&q)[4]) {
  atomicAdd(acc + n1, (unsigned long long)q[0]);
  atomicAdd(acc + n1 + nny, (unsigned long long)q[1]);
  atomicAdd(acc + n1 + nny + 1, (unsigned long long)q[2]);
  atomicAdd(acc + n1 + 1, (unsigned long long)q[3]);
}

// Four consecutive particles a thread.  Bound by the atomics where each
// particle adds its own (3M cell-sorted particles on 257 x 200 nodes: 12M adds
// on 51,400 addresses, 158 us); callers mostly keep particles in cell order,
// so a thread sums its particles in registers while they stay in one element,
// and the warp sums the threads' last runs by segments of equal elements,
// unless nearly every lane holds another one (unsorted particles: then each
// adds its own, as many atomics as before).  The four quotients a particle
// needs are products (div_dev.h, the same bits as the divisions).
// A call with those particles: 158 -> 38 us.
constexpr int kNaRun = 4;
// One particle a thread while a wave of them holds all: the latency of one counts
// (30,001 on 257 x 200 nodes: four each 22.6 us a call, one 20.3, sorted ones too);
// and while there are less than two particles a node, so hardly a run (600,000
// on 700 x 700: 32.6, one each 30.6).
constexpr int64_t kNaFew = 148 * 2048;

template <int RUN>
__global__ void __launch_bounds__(256) k_na_deposit(int nnx, int nny, double xmin, double ymin, double hx, double hy,
                                                    int64_t n, const double *__restrict__ x,
                                                    const double *__restrict__ y, const int32_t *__restrict__ loc,
                                                    int vec, unsigned long long *acc) {
  const int64_t p0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * RUN;
  const int nex = nnx - 1, ney = nny - 1, lane = threadIdx.x & 31;
  const double rhx = RUN > 1 ? pic::recip_const(hx) : 0.0, rhy = RUN > 1 ? pic::recip_const(hy) : 0.0;
  double px[RUN], py[RUN];
  int lc[RUN];
  if (RUN > 1 && vec && p0 + RUN <= n) {  // 16-byte aligned arrays
    if constexpr (RUN > 1) {
#pragma unroll
      for (int k = 0; k < RUN; k += 2) {
        const double2 a = *reinterpret_cast<const double2 *>(x + p0 + k), b = *reinterpret_cast<const double2 *>(y + p0 + k);
        px[k] = a.x;
        px[k + 1] = a.y;
        py[k] = b.x;
        py[k + 1] = b.y;
      }
      const int4 l = loc ? *reinterpret_cast<const int4 *>(loc + p0) : make_int4(0, 0, 0, 0);
      lc[0] = l.x;
      lc[1] = l.y;
      lc[2] = l.z;
      lc[3] = l.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < RUN; ++k) {
      const bool in = p0 + k < n;
      px[k] = in ? x[p0 + k] : 0.0;
      py[k] = in ? y[p0 + k] : 0.0;
      lc[k] = !in ? -1 : loc ? loc[p0 + k] : 0;
    }
  }
  int key = -1;  // the run's first node
  long long q[4] = {0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < RUN; ++k) {
    if (lc[k] < 0) continue;  // absorbed slot
    bool exact = RUN > 1;  // one particle a thread: the divisions are the shorter chain
    double rxp = 0.0, ryp = 0.0;
    if (RUN > 1) {
      rxp = pic::div_const(px[k] - xmin, hx, rhx, exact);
      ryp = pic::div_const(py[k] - ymin, hy, rhy, exact);
    }
    if (!exact) {
      rxp = (px[k] - xmin) / hx;
      ryp = (py[k] - ymin) / hy;
    }
    int i = (int)rxp + 1, j = (int)ryp + 1;
    if (i == nnx) i = nnx - 1;
    if (j == nny) j = nny - 1;
    if (!(rxp >= 0.0) || !(ryp >= 0.0) || i < 1 || j < 1 || i > nex || j > ney) continue;
    const int ie = i - 1, je = j - 1;
    const double x1 = xmin + hx * ie, x2 = xmin + hx * (ie + 1);
    const double y1 = ymin + hy * je, y2 = ymin + hy * (je + 1);
    exact = RUN > 1;
    double dx = 0.0, dy = 0.0;
    if (RUN > 1) {
      dx = pic::div_const(px[k] - x1, x2 - x1, pic::recip_near(x2 - x1, rhx), exact);
      dy = pic::div_const(py[k] - y1, y2 - y1, pic::recip_near(y2 - y1, rhy), exact);
    }
    if (!exact || fabs((x2 - x1) - hx) > 1e-9 * hx || fabs((y2 - y1) - hy) > 1e-9 * hy) {
      dx = (px[k] - x1) / (x2 - x1);
      dy = (py[k] - y1) / (y2 - y1);
    }
    const double xc = 1.0 - dx, yc = 1.0 - dy;
    const int n1 = ie * nny + je;
    if (n1 != key) {
      if (key >= 0) na_add(acc, key, nny, q);
      key = n1;
      q[0] = q[1] = q[2] = q[3] = 0;
    }
    // corner 2 takes the rest of the particle's 2^40, as pic_get_par_chg does
    const long long q0 = __double2ll_rn((xc * yc) * PIC_Q_SCALE), q1 = __double2ll_rn((dx * yc) * PIC_Q_SCALE);
    const long long q3 = __double2ll_rn((xc * dy) * PIC_Q_SCALE);
    q[0] += q0;
    q[1] += q1;
    q[3] += q3;
    q[2] += (1ll << 40) - ((q0 + q1) + q3);
  }
  const int prev = __shfl_up_sync(0xffffffffu, key, 1);
  const bool head = lane == 0 || key != prev;
  const unsigned heads = __ballot_sync(0xffffffffu, head);
  if (__popc(heads) <= 20) {
    const unsigned above = lane == 31 ? 0u : (heads & ~((2u << lane) - 1u));
    const int seg_end = above ? __ffs(above) - 2 : 31;
    const int maxlen = (int)__reduce_max_sync(0xffffffffu, head ? (unsigned)(seg_end - lane + 1) : 0u);
    seg_sums4(q, lane, seg_end, maxlen);
    if (head && key >= 0) na_add(acc, key, nny, q);
  } else if (key >= 0) {
    na_add(acc, key, nny, q);
  }
}

__global__ void k_na_normalize(const unsigned long long *acc, const double *__restrict__ vol, double wq,
                               double L_ref, double n_ref, double *__restrict__ rho, int64_t nn) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nn) return;
  double cnt = (double)(long long)acc[k] * (1.0 / PIC_Q_SCALE);
  rho[k] = ((((wq * cnt) / L_ref) / L_ref) / n_ref) / vol[k];
}

int na_fail(cudaError_t e, const char *where) {
  pic::set_error(std::string("pic_deposit_noalloc: ") + where + ": " + cudaGetErrorString(e));
  return PIC_ERR_CUDA;
}

}  // namespace

extern "C" int pic_deposit_noalloc(int32_t nnx, int32_t nny, double xmin, double xmax, double ymin,
                                   double ymax, int64_t n, const double *x, const double *y,
                                   const int32_t *loc, const double *cell_volume, double weight_charge,
                                   double L_ref, double n_ref, double *rho_out, void *stream) {
  if (nnx < 3 || nny < 3 || !(xmax > xmin) || !(ymax > ymin) || n < 0 || !cell_volume || !rho_out ||
      (n > 0 && (!x || !y)) || !(L_ref > 0) || !(n_ref > 0)) {
    pic::set_error("pic_deposit_noalloc: bad arguments");
    return PIC_ERR_ARG;
  }
  const int64_t nn = (int64_t)nnx * nny;
  if (nn > PIC_NOALLOC_MAX_NODES) {
    char buf[200];
    snprintf(buf, sizeof buf,
             "pic_deposit_noalloc: mesh has %lld nodes, the static scratch holds at most %d",
             (long long)nn, PIC_NOALLOC_MAX_NODES);
    pic::set_error(buf);
    return PIC_ERR_ARG;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return na_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices) {
    pic::set_error("pic_deposit_noalloc: device ordinal beyond the supported range");
    return PIC_ERR_ARG;
  }
  // Set-up, once per device with that device current: the device address of
  // the scratch array (its host-side name is only a stand-in).
  unsigned long long *acc = g_acc_ptr[dev].load(std::memory_order_acquire);
  if (!acc) {
    void *ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_noalloc_acc);
    if (e != cudaSuccess) return na_fail(e, "cudaGetSymbolAddress");
    acc = (unsigned long long *)ptr;
    g_acc_ptr[dev].store(acc, std::memory_order_release);
  }
  cudaStream_t st = (cudaStream_t)stream;
  const double hx = (xmax - xmin) / (nnx - 1), hy = (ymax - ymin) / (nny - 1);
  k_na_clear<<<(unsigned)((nn + 255) / 256), 256, 0, st>>>(acc, nn);
  if (n > 0) {
    const int run = n <= kNaFew || n < 2 * nn ? 1 : kNaRun;
    (run == 1 ? k_na_deposit<1> : k_na_deposit<kNaRun>)<<<(unsigned)((n + 256 * run - 1) / (256 * run)), 256, 0, st>>>(
        nnx, nny, xmin, ymin, hx, hy, n, x, y, loc, (((uintptr_t)x | (uintptr_t)y | (uintptr_t)loc) & 15) == 0, acc);
  }
  k_na_normalize<<<(unsigned)((nn + 255) / 256), 256, 0, st>>>(acc, cell_volume, weight_charge, L_ref, n_ref,
                                                                rho_out, nn);
  e = cudaGetLastError();
  if (e != cudaSuccess) return na_fail(e, "launch");
  return PIC_OK;
}
