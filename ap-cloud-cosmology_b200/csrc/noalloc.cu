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
#include <cstddef>
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
constexpr int kNoBig = 256;   // particles from which a cell is spread over the whole grid
constexpr int kNoUnit = 128;  // in pieces of this many, a warp each
constexpr int kNoWords = APC_NOALLOC_MAX_PARTICLES / 32;
constexpr int kNoBigMax = APC_NOALLOC_MAX_PARTICLES / kNoBig;
struct NoallocAcc {
  unsigned long long maxbits;  // IEEE bits of max |a|^2 c_vel^2 dt^2
  unsigned long long total;    // particles in all ranges
  int covered;                 // bits set
  int bad;                     // ranges outside [0, n)
  int err;                     // a grid barrier gave up
  int outcome;                 // of the second barrier, the same for every block: kKick or kLeave
  int nbig;
  GridBar bar;
};
enum { kKick = 1, kLeave = 2 };
struct NoallocScratch {
  NoallocAcc acc;           // cleared before each launch, with the words of the bits that it uses
  unsigned bits[kNoWords];
  int4 big[kNoBigMax];      // a cell of many particles: its index, first and count
};
static_assert(sizeof(NoallocScratch) <= kNoallocScratchBytes, "fits the scratch array");

// The whole call in one cooperative launch, its phases a grid barrier apart: mark every range's
// particles in the bits and add up the ranges; count the bits (ranges that hold n particles in
// all and cover n of them cover each once); and - when all is well - interpolate and kick, LANES
// lanes per cell and a warp per piece of a cell of many, so that no particle -> cell map is
// written, checked and read back.  The marks return nothing, so nobody waits for them.  The last
// phase is bound by memory: 96 B per particle beside its cell's row.  A call for 1,000,000
// particles from the host, in us, by the particles of a cell, as two memsets and three kernels
// and now: 9: 60, 57; 20: 51, 57; 50: 51, 52; 200: 51, 57; 2,500: 78, 57; 50,000: 607, 57.
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
  __shared__ int s_outcome, s_scan[kNoThreads / 32], s_piece[kNoBigMax];
  NoallocAcc *acc = &S->acc;
  const int t = threadIdx.x, lane = t & 31;
  const int threads = gridDim.x * kNoThreads, g0 = blockIdx.x * kNoThreads + t;
  unsigned epoch = 0;
  // ---- the ranges: a lane for about every word of a cell; a cell of many by its whole warp ----
  {
    constexpr int kMark = LANES > 8 ? LANES / 8 : 1;
    const int sub = g0 % kMark;
    const unsigned cells = (unsigned)threads / kMark, rounds = ((unsigned)m + cells - 1u) / cells;
    unsigned long long mine = 0;
    for (unsigned r = 0; r < rounds; ++r) {  // the same count for every lane (ballots)
      const unsigned i = r * cells + (unsigned)(g0 / kMark);  // past m, a multiple of the grid: no int
      long long f = 0, c = 0;
      if (i < (unsigned)m) {
        f = first[i];
        c = count[i];
        if (c < 0 || (c > 0 && (f < 0 || f + c > n))) {
          atomicOr(&acc->bad, 1);
          c = 0;
        }
        if (c >= kNoBig && sub == 0) {  // more than kNoBigMax of them overlap
          const int q = atomicAdd(&acc->nbig, 1);
          if (q < kNoBigMax) S->big[q] = make_int4((int)i, (int)f, (int)c, 0);
        }
      }
      if (sub == 0) mine += (unsigned long long)c;
      auto mark = [&](long long lo, long long hi, int w) {  // bits [lo, hi) of word w
        const int a = (int)max(lo - 32ll * w, 0ll), b = (int)min(hi - 32ll * w, 32ll);
        const unsigned mask = (b == 32 ? ~0u : (1u << b) - 1u) & ~((1u << a) - 1u);
        atomicOr(&S->bits[w], mask);
      };
      const bool wide = c >= kNoBig;
      if (c > 0 && !wide)
        for (int w = (int)(f >> 5) + sub; w <= (int)((f + c - 1) >> 5); w += kMark) mark(f, f + c, w);
      for (unsigned todo = __ballot_sync(0xffffffffu, wide && sub == 0); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const long long bf = __shfl_sync(0xffffffffu, f, src), bc = __shfl_sync(0xffffffffu, c, src);
        for (int w = (int)(bf >> 5) + lane; w <= (int)((bf + bc - 1) >> 5); w += 32) mark(bf, bf + bc, w);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (lane == 0 && mine) atomicAdd(&acc->total, mine);
  }
  if (!grid_sync(&acc->bar, gridDim.x, epoch, &acc->err)) return;
  {
    int mine = 0;
    for (int w = g0; w < (n + 31) / 32; w += threads) mine += __popc(__ldcg(&S->bits[w]));
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0 && mine) atomicAdd(&acc->covered, mine);
  }
  // A block whose wait runs out here leaves, and another may still find every block arrived.  All
  // take the first claim, so that a call that gives up has written nothing.
  const bool met = grid_sync(&acc->bar, gridDim.x, epoch, &acc->err, blockIdx.x == 0 ? limit0 : kSpinLimit);
  if (t == 0) {
    const int mine = met ? kKick : kLeave, first_claim = atomicCAS(&acc->outcome, 0, mine);
    s_outcome = first_claim != 0 ? first_claim : mine;
    if (!met) __threadfence();  // the claim of a block that did see all arrive: its view, in place of the barrier's
  }
  __syncthreads();
  if (s_outcome != kKick) return;
  // malformed cell ranges leave every output untouched
  const bool ok = *(volatile int *)&acc->bad == 0 && *(volatile int *)&acc->covered == n &&
                  *(volatile unsigned long long *)&acc->total == (unsigned long long)n;
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
  // the cells of many particles, piece by piece: every block numbers the pieces of all of them,
  // and a warp finds the cell of its piece.  (Cell after cell, each over the whole grid, took
  // 606 us for 1,000,000 particles in 400 cells, 57 now.)
  const int nbig = ok ? min(*(volatile int *)&acc->nbig, kNoBigMax) : 0;
  if (nbig > 0) {
    constexpr int kEach = kNoBigMax / kNoThreads;
    int mine[kEach], sum = 0, total;
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
      const int q = t * kEach + k;
      mine[k] = sum;
      if (q < nbig) sum += (__ldcg(&S->big[q]).z + kNoUnit - 1) / kNoUnit;
    }
    const int before = block_scan_int<kNoThreads>(sum, s_scan, &total);
#pragma unroll
    for (int k = 0; k < kEach; ++k) s_piece[t * kEach + k] = before + mine[k];
    __syncthreads();
    for (int u = g0 >> 5; u < total; u += threads >> 5) {
      int q = 0;  // the last cell whose pieces begin at or before u
#pragma unroll
      for (int step = kNoBigMax / 2; step > 0; step >>= 1)
        if (q + step < nbig && s_piece[q + step] <= u) q += step;
      const int4 cell = __ldcg(&S->big[q]);
      const int at = cell.y + (u - s_piece[q]) * kNoUnit;
      kick_cell(cell.x, at + lane, min(at + kNoUnit, cell.y + cell.z), 32);
    }
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
  // lanes per cell: half the mean count or more, so that most cells take one or two rounds and
  // a last wave of blocks that is nearly empty stays short
  const double mean = (double)n_particles / n_cells;
  const struct {
    double mean;
    int lanes;
    const void *kern;
  } forms[] = {{8, 4, (const void *)noalloc_kick<4>},     {16, 8, (const void *)noalloc_kick<8>},
               {32, 16, (const void *)noalloc_kick<16>},  {64, 32, (const void *)noalloc_kick<32>},
               {1e300, 64, (const void *)noalloc_kick<64>}};
  int form = 0;
  while (mean > forms[form].mean) ++form;
  const int lanes = forms[form].lanes;
  const void *kern = forms[form].kern;
  std::lock_guard<std::mutex> lock(g_call_mutex[dev]);
  // as many blocks as are resident together (the phases are grid barriers; asked once per device
  // and form), no more than the cells' lane groups or the particles need
  static int resident[kMaxDevices][sizeof(forms) / sizeof(forms[0])] = {};
  if (resident[dev][form] == 0) {
    int sms = 0, occ = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kNoThreads, 0) != cudaSuccess || occ < 1) {
      cudaGetLastError();
      return APC_ERR_CUDA;
    }
    resident[dev][form] = sms * occ;
  }
  const long long want = (std::max((long long)n_particles, (long long)n_cells * lanes) + kNoThreads - 1) / kNoThreads;
  const int blocks = (int)std::max(1ll, std::min(want, (long long)resident[dev][form]));
  void *args[] = {&n_particles, &n_cells, &first, &count, &deriv9, &cx, &cy, &cz, &x, &y, &z, &vx, &vy, &vz,
                  &ax, &ay, &az, &c_vel, &dt, &S, &limit0};
  NoallocAcc got;
  const size_t clear = offsetof(NoallocScratch, bits) + sizeof(unsigned) * (size_t)((n_particles + 31) / 32);
  if (cudaMemsetAsync(S, 0, clear, s) != cudaSuccess ||
      cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(kNoThreads), args, 0, s) != cudaSuccess ||
      cudaMemcpyAsync(&got, &S->acc, sizeof(got), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess) {
    cudaGetLastError();
    return APC_ERR_CUDA;
  }
  if (got.outcome != kKick) return APC_ERR_TIMEOUT;  // a grid barrier gave up: nothing was written
  // cell ranges outside [0, n), overlapping, or leaving a particle uncovered: caller input,
  // so an invalid argument (the context path builds its ranges itself); nothing was written
  if (got.bad || got.covered != n_particles || got.total != (unsigned long long)n_particles) return APC_ERR_INVALID_ARG;
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
