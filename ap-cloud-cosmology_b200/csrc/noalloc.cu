// Interpolation + kick for callers that cannot allocate device memory.
//
// Some embedders own every byte of device memory themselves: a host framework with its
// own pooled allocator that forbids outside cudaMalloc, or a real-time loop where the
// implicit device synchronisation of cudaMalloc/cudaFree is not acceptable.  For them
// this entry point runs the same interpolation + kick as apc_move_velocity, on buffers
// the caller passes in, and takes its scratch (a bit per particle and the
// max-change accumulator) from a fixed array compiled into the library instead of
// allocating it.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <mutex>

#include "apc_internal.cuh"

namespace {

// Scratch shared by every call on a device (its size is part of the interface's contract; the
// kernel needs less).  Every GPU that loads the library holds it until the process exits.
constexpr size_t kNoallocScratchBytes = sizeof(int) * (size_t)APC_NOALLOC_MAX_PARTICLES + 256;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
void *g_scratch_ptr[kMaxDevices] = {nullptr};
std::mutex g_call_mutex[kMaxDevices];  // held for a whole call: the scratch is one per device

// The scratch array: one bit per particle, the cells of many particles, and the accumulators,
// which every call clears before its launch and copies to its own stack after it: nothing is
// handed from one call to the next, and a device takes one call at a time.  (Accumulators left
// clear by the kernel and results in pinned words saved the two stream operations, 8 us of
// a call; but a call that broke off spoilt the next, threads read each other's results, and the
// pinned words had to be allocated.)
constexpr int kNoThreads = 512;
constexpr int kNoBig = 2048;  // particles from which a cell is spread over the whole grid
constexpr int kNoWords = APC_NOALLOC_MAX_PARTICLES / 32;
constexpr int kNoBigMax = APC_NOALLOC_MAX_PARTICLES / kNoBig;
struct NoallocAcc {
  unsigned long long maxbits;  // IEEE bits of max |a|^2 c_vel^2 dt^2
  unsigned long long total;    // particles in all ranges
  int bad;                     // ranges outside [0, n), or overlapping
  int err;                     // a grid barrier gave up
  int outcome;                 // of the second barrier, the same for every block: kKick or kLeave
  int nbig;
  GridBar bar;
};
enum { kKick = 1, kLeave = 2 };
struct NoallocScratch {
  unsigned bits[kNoWords];
  int big[kNoBigMax];
  NoallocAcc acc;
};
static_assert(sizeof(NoallocScratch) <= kNoallocScratchBytes, "fits the scratch array");

// The whole call in one cooperative launch, its phases a grid barrier apart: clear the bits,
// mark every range's particles (a bit already set is an overlap; ranges without overlaps
// that hold n particles in all cover every particle), and - when all is well - interpolate and
// kick, LANES lanes per cell, so that no particle -> cell map is written, checked and read
// back.  The last phase is bound by memory: 96 B per particle beside its cell's row.
// 1,000,003 particles in 111,111 cells: two memsets and three kernels took 52 us on the device,
// this kernel 33 us (25 us of it the kick); a call from Python 99 -> 86 us.
template <int LANES>
__global__ void __launch_bounds__(kNoThreads) noalloc_kick(int n, int m, const int *__restrict__ first,
                                                           const int *__restrict__ count,
                                                           const double *__restrict__ deriv,
                                                           const double *__restrict__ cx,
                                                           const double *__restrict__ cy,
                                                           const double *__restrict__ cz,
                                                           const double *__restrict__ x,
                                                           const double *__restrict__ y,
                                                           const double *__restrict__ z, double *__restrict__ vx,
                                                           double *__restrict__ vy, double *__restrict__ vz,
                                                           double *__restrict__ ax, double *__restrict__ ay,
                                                           double *__restrict__ az, double cv, double dt,
                                                           NoallocScratch *S, long long limit0) {
  __shared__ double sm[kNoThreads / 32];
  __shared__ int s_outcome;
  NoallocAcc *acc = &S->acc;
  const int t = threadIdx.x, lane = t & 31;
  const int threads = gridDim.x * kNoThreads, g0 = blockIdx.x * kNoThreads + t;
  unsigned epoch = 0;
  for (int w = g0; w < (n + 31) / 32; w += threads) S->bits[w] = 0u;
  if (!grid_sync(&acc->bar, gridDim.x, epoch, &acc->err)) return;
  // ---- the ranges: a thread per cell; a cell of many words by its whole warp ----
  {
    unsigned long long mine = 0;
    const unsigned rounds = ((unsigned)m + (unsigned)threads - 1u) / (unsigned)threads;
    for (unsigned r = 0; r < rounds; ++r) {  // the same count for every lane (ballots)
      const unsigned i = r * (unsigned)threads + (unsigned)g0;  // past m, a multiple of the grid: no int
      long long f = 0, c = 0;
      if (i < (unsigned)m) {
        f = first[i];
        c = count[i];
        if (c < 0 || (c > 0 && (f < 0 || f + c > n))) {
          atomicOr(&acc->bad, 1);
          c = 0;
        }
        if (c >= kNoBig) {  // more than kNoBigMax of them overlap
          const int q = atomicAdd(&acc->nbig, 1);
          if (q < kNoBigMax) S->big[q] = (int)i;
        }
      }
      mine += (unsigned long long)c;
      auto mark = [&](long long lo, long long hi, int w) {  // bits [lo, hi) of word w
        const int a = (int)max(lo - 32ll * w, 0ll), b = (int)min(hi - 32ll * w, 32ll);
        const unsigned mask = (b == 32 ? ~0u : (1u << b) - 1u) & ~((1u << a) - 1u);
        if (atomicOr(&S->bits[w], mask) & mask) atomicOr(&acc->bad, 1);
      };
      const bool wide = c > 256;
      if (c > 0 && !wide)
        for (int w = (int)(f >> 5); w <= (int)((f + c - 1) >> 5); ++w) mark(f, f + c, w);
      for (unsigned todo = __ballot_sync(0xffffffffu, wide); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const long long bf = __shfl_sync(0xffffffffu, f, src), bc = __shfl_sync(0xffffffffu, c, src);
        for (int w = (int)(bf >> 5) + lane; w <= (int)((bf + bc - 1) >> 5); w += 32) mark(bf, bf + bc, w);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (lane == 0 && mine) atomicAdd(&acc->total, mine);
  }
  // A block whose wait runs out here leaves, and another may still find every block arrived.  All
  // take the first claim, so that a call that gives up has written nothing.
  const bool met = grid_sync(&acc->bar, gridDim.x, epoch, &acc->err, blockIdx.x == 0 ? limit0 : kSpinLimit);
  if (t == 0) {
    const int mine = met ? kKick : kLeave, first_claim = atomicCAS(&acc->outcome, 0, mine);
    s_outcome = first_claim != 0 ? first_claim : mine;
  }
  __syncthreads();
  if (s_outcome != kKick) return;
  // malformed cell ranges leave every output untouched
  const bool ok =
      *(volatile int *)&acc->bad == 0 && *(volatile unsigned long long *)&acc->total == (unsigned long long)n;
  // ---- same arithmetic, operand order and rounding as the kick of apc_move_velocity ----
  double mx = 0.0;
  auto kick_cell = [&](int i, int s0, int s1, int step) {  // particles s0, s0 + step, ... < s1 of cell i
    if (s0 >= s1) return;
    double d[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) d[k] = deriv[(size_t)i * 9 + k];
    const double ccx = cx[i], ccy = cy[i], ccz = cz[i];
    for (int s = s0; s < s1; s += step) {
      const double dx = __dsub_rn(x[s], ccx), dy = __dsub_rn(y[s], ccy), dz = __dsub_rn(z[s], ccz);
      const double a1 = __dadd_rn(__dadd_rn(__dadd_rn(d[0], __dmul_rn(dx, d[3])), __dmul_rn(dy, d[6])), __dmul_rn(dz, d[7]));
      const double a2 = __dadd_rn(__dadd_rn(__dadd_rn(d[1], __dmul_rn(dx, d[6])), __dmul_rn(dy, d[4])), __dmul_rn(dz, d[8]));
      const double a3 = __dadd_rn(__dadd_rn(__dadd_rn(d[2], __dmul_rn(dx, d[7])), __dmul_rn(dy, d[8])), __dmul_rn(dz, d[5]));
      ax[s] = a1;
      ay[s] = a2;
      az[s] = a3;
      vx[s] = __dadd_rn(vx[s], __dmul_rn(__dmul_rn(a1, cv), dt));
      vy[s] = __dadd_rn(vy[s], __dmul_rn(__dmul_rn(a2, cv), dt));
      vz[s] = __dadd_rn(vz[s], __dmul_rn(__dmul_rn(a3, cv), dt));
      const double sq = __dadd_rn(__dadd_rn(__dmul_rn(a1, a1), __dmul_rn(a2, a2)), __dmul_rn(a3, a3));
      mx = fmax(mx, __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(sq, cv), cv), dt), dt));
    }
  };
  for (unsigned i = (unsigned)(g0 / LANES); i < (unsigned)m && ok; i += (unsigned)(threads / LANES)) {
    const int f = first[i], c = count[i];
    // nothing is formed from an empty cell's first: it may be any value
    if (c > 0 && c < kNoBig) kick_cell((int)i, f + g0 % LANES, f + c, LANES);
  }
  const int nbig = ok ? min(*(volatile int *)&acc->nbig, kNoBigMax) : 0;
  for (int q = 0; q < nbig; ++q) {
    const int i = S->big[q], f = first[i];
    kick_cell(i, f + g0, f + count[i], threads);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) sm[t >> 5] = mx;
  __syncthreads();
  if (t == 0) {
    double b = 0.0;
    for (int w = 0; w < kNoThreads / 32; ++w) b = fmax(b, sm[w]);
    atomicMax(&acc->maxbits, (unsigned long long)__double_as_longlong(b));
  }
}

// Device address of the scratch array for `dev`, looked up once per device with that
// device current.  In host code the array's name is only a host-side stand-in, so the
// kernels are always given this address.
int scratch_for(int dev, void **out) {
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (g_scratch_ptr[dev]) {
    *out = g_scratch_ptr[dev];
    return APC_OK;
  }
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess || !p) {
    cudaGetLastError();
    return APC_ERR_CUDA;
  }
  g_scratch_ptr[dev] = p;
  *out = p;
  return APC_OK;
}

}  // namespace

// limit0: polls of the first block at the second barrier
static int noalloc_call(int n_particles, int n_cells, const int *first, const int *count, const double *cx,
                        const double *cy, const double *cz, const double *deriv9, const double *x, const double *y,
                        const double *z, double *vx, double *vy, double *vz, double *ax, double *ay, double *az,
                        double dt, double c_vel, double *max_dv, void *stream, long long limit0) {
  if (n_particles < 1 || n_cells < 1) return APC_ERR_INVALID_ARG;
  if (n_particles > APC_NOALLOC_MAX_PARTICLES) return APC_ERR_INVALID_ARG;  // beyond the scratch array
  if (!first || !count || !cx || !cy || !cz || !deriv9 || !x || !y || !z || !vx || !vy || !vz || !ax || !ay ||
      !az)
    return APC_ERR_INVALID_ARG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return APC_ERR_CUDA;
  }
  void *base = nullptr;
  int rc = scratch_for(dev, &base);
  if (rc != APC_OK) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  NoallocScratch *S = (NoallocScratch *)base;
  // lanes per cell: half the mean count or more, so that most cells take one or two rounds
  const double mean = (double)n_particles / n_cells;
  const void *kern = mean <= 8 ? (const void *)noalloc_kick<4>
                               : (mean <= 16 ? (const void *)noalloc_kick<8>
                                             : (mean <= 32 ? (const void *)noalloc_kick<16>
                                                           : (const void *)noalloc_kick<32>));
  const int lanes = mean <= 8 ? 4 : (mean <= 16 ? 8 : (mean <= 32 ? 16 : 32));
  // as many blocks as are resident together (the phases are grid barriers), no more than the
  // cells' lane groups or the particles need
  int sms = 1, occ = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kNoThreads, 0) != cudaSuccess || occ < 1) {
    cudaGetLastError();
    return APC_ERR_CUDA;
  }
  const long long want = (std::max((long long)n_particles, (long long)n_cells * lanes) + kNoThreads - 1) / kNoThreads;
  const int blocks = (int)std::max(1ll, std::min(want, (long long)sms * occ));
  void *args[] = {&n_particles, &n_cells, &first, &count, &deriv9, &cx, &cy, &cz, &x, &y, &z, &vx, &vy, &vz,
                  &ax, &ay, &az, &c_vel, &dt, &S, &limit0};
  NoallocAcc got;
  std::lock_guard<std::mutex> lock(g_call_mutex[dev]);
  if (cudaMemsetAsync(&S->acc, 0, sizeof(NoallocAcc), s) != cudaSuccess ||
      cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(kNoThreads), args, 0, s) != cudaSuccess ||
      cudaMemcpyAsync(&got, &S->acc, sizeof(got), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess) {
    cudaGetLastError();
    return APC_ERR_CUDA;
  }
  if (got.outcome != kKick) return APC_ERR_TIMEOUT;  // a grid barrier gave up: nothing was written
  // cell ranges outside [0, n), overlapping, or leaving a particle uncovered: caller input,
  // so an invalid argument (the context path builds its ranges itself); nothing was written
  if (got.bad || got.total != (unsigned long long)n_particles) return APC_ERR_INVALID_ARG;
  if (max_dv) {
    double v;
    std::memcpy(&v, &got.maxbits, sizeof(v));
    *max_dv = std::sqrt(v);
  }
  return APC_OK;
}

extern "C" int apc_move_velocity_noalloc(int n_particles, int n_cells, const int *first, const int *count,
                                         const double *cx, const double *cy, const double *cz,
                                         const double *deriv9, const double *x, const double *y,
                                         const double *z, double *vx, double *vy, double *vz, double *ax,
                                         double *ay, double *az, double dt, double c_vel, double *max_dv,
                                         void *stream) {
  return noalloc_call(n_particles, n_cells, first, count, cx, cy, cz, deriv9, x, y, z, vx, vy, vz, ax, ay, az, dt,
                      c_vel, max_dv, stream, kSpinLimit);
}

// For the tests: the same call, with a wait of the first block that gives up after spin_limit polls.
extern "C" int apc_test_move_velocity_noalloc(int spin_limit, int n_particles, int n_cells, const int *first,
                                              const int *count, const double *cx, const double *cy, const double *cz,
                                              const double *deriv9, const double *x, const double *y, const double *z,
                                              double *vx, double *vy, double *vz, double *ax, double *ay, double *az,
                                              double dt, double c_vel, double *max_dv, void *stream) {
  if (spin_limit < 1 || spin_limit > kSpinLimit) return APC_ERR_INVALID_ARG;
  return noalloc_call(n_particles, n_cells, first, count, cx, cy, cz, deriv9, x, y, z, vx, vy, vz, ax, ay, az, dt,
                      c_vel, max_dv, stream, spin_limit);
}
