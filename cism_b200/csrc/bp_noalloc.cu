// bp_noalloc.cu -- residual and norms without any device allocation.
//
// bp_residual_noalloc computes resid = A x - b on the locally owned active
// rows of a system held by the caller in device memory, in the reference's
// own layout (matrix blocks (27,nz,nx-1,ny-1), vectors (nz,nx-1,ny-1), halo
// included and already halo-consistent), plus |A x - b|, |b| and their
// ratio.  It is the allocation-free variant of the residual kernel of the
// solver (k_resid<MV_INIT>): its only scratch -- one partial sum pair per
// block and the ticket that elects the block doing the final sum -- lives in
// the file-scope array below instead of in memory from cudaMalloc.
//
// Who needs it: a host model that owns all device memory itself (a fixed
// pool or budget set up once) or that must not trigger the implicit
// device-wide synchronisation of cudaMalloc/cudaFree in the middle of a
// time step can call this with its own buffers and nothing else.
//
// Limits and sharing: at most kNaMaxRows = 16,777,216 rows (nz*(nx-1)*(ny-1));
// larger systems are rejected with BP_ERR_ARGS (a limit of the call that its
// users know, not of the scratch: the blocks loop over the rows).  The array is global to the
// process and to each device, and every call reuses it: two calls whose
// work overlaps on the GPU (different streams, or different host threads on
// one device) race on the partial sums and give wrong norms, or leave theirs
// unwritten.  Serialise them.  Calls after an overlap are right again: the
// ticket is where it was once all of them are done (ticket_share), in graph
// replays too and without a launch to reset it; a count of blocks that wraps
// at each launch's own number does not come back.  The first call on a device
// (and the first after the device's context was torn down and made again, e.g.
// by cudaDeviceReset) looks up the array's device address
// (cudaGetSymbolAddress); make that call before any stream capture.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <mutex>

#include "bp_b200.h"
#include "bp_common.h"

namespace {

constexpr int kNaRows = 32;           // rows of a chunk; a block is one warp
constexpr int kNaBlocks = 8 * 148;    // resident blocks of the GPU (27 KB of shared memory each)
constexpr long kNaMaxRows = 1L << 24;
constexpr int kNaMaxDevices = 64;

struct NaScratch {
  double partial[2 * kNaBlocks];     // per block: sum (Ax-b)^2, sum b^2
  unsigned ticket;                   // shares of the blocks that have finished; 0 between launches
  unsigned pad[63];
};

// 19 KB on every device that loads the library, held until exit.
static __device__ __align__(256) NaScratch g_na_scratch;

std::mutex g_na_mutex;
NaScratch* g_na_ptr[kNaMaxDevices] = {nullptr};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Bounded wait on a shared-memory barrier (phase `parity`).
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity) {
  for (int i = 0; i < (1 << 24); ++i) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// The matrix is the whole traffic (4 x 216 B of a row against 48 B of
// vectors) and a row's 27 entries are contiguous, so a thread that walks
// its own row in global memory makes every load of a warp touch 32 sectors.
// Here one warp takes a chunk of 32 consecutive rows at a time: one bulk
// copy per matrix block brings the chunk's rows (from its first to its last
// active one) into shared memory -- 27 KB, eight one-warp blocks per SM, so
// that copies are always in flight and no block waits on another -- while
// the threads load their rows' 54 source values (consecutive rows:
// consecutive addresses) into registers; then each thread sums its row from
// shared memory (27 doubles apart: no bank conflict).  BULK = false copies
// with plain loads, for matrix pointers that are not 16-byte aligned (a
// bulk copy must start on 16 bytes).  A pair of rows is 27 x 16 B, so
// copies start and end on even rows; the pair of the last active row never
// passes the end of the arrays, whose last column is no owned one (i <= nx - 2
// and j <= ny - 2, while the arrays end with column (nx - 1, ny - 1)).  Bound: DRAM.  A round ice sheet on 160 x 160 x 11 (16 thousand
// active columns, 165 MB): 35 us, 4.7 TB/s, against 82 us for the thread-per-
// row loads with the ticket's memset before each launch; 31 x 31 x 10: the
// call is bound by the host's one launch (10.2 us a call against 13.0).
template <bool BULK>
__global__ void __launch_bounds__(kNaRows)
k_resid_ref_layout(int nx, int ny, int nz, int periodic, const int* __restrict__ active_vertex,
                   const double* __restrict__ Auu, const double* __restrict__ Auv,
                   const double* __restrict__ Avu, const double* __restrict__ Avv,
                   const double* __restrict__ xu, const double* __restrict__ xv,
                   const double* __restrict__ bu, const double* __restrict__ bv,
                   double* __restrict__ ru, double* __restrict__ rv, double* __restrict__ norms,
                   NaScratch* S) {
  extern __shared__ __align__(16) double na_sm[];  // [4][kNaRows][27]
  __shared__ __align__(8) unsigned long long bar;
  const int tid = threadIdx.x;
  const int V = nx - 1, W = ny - 1;
  const long rows = (long)nz * V * W;
  const long chunks = (rows + kNaRows - 1) / kNaRows;
  if (BULK && tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  double s_r = 0.0, s_b = 0.0;
  unsigned phase = 0;
  bool ok = true;
  for (long ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
    const long t0 = ch * kNaRows, t = t0 + tid;
    int k = 0;
    bool mine = false;
    if (t < rows) {
      const long c = t / nz;
      k = (int)(t - c * nz);
      const int j0 = (int)(c / V), i0 = (int)(c - (long)j0 * V);  // 0-based vertex indices
      const int lo = periodic ? 2 : 1;
      mine = i0 >= lo && i0 <= nx - 3 && j0 >= lo && j0 <= ny - 3 && active_vertex[c] != 0;
    }
    const unsigned act = __ballot_sync(0xffffffffu, mine);
    if (act) {
      const int r0 = (__ffs((int)act) - 1) & ~1;
      const int r1 = (33 - __clz((int)act)) & ~1;  // [r0, r1) holds the active rows, both even
      if (BULK) {
        if (tid == 0) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          const unsigned bytes = (unsigned)(r1 - r0) * 216u;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %0;" ::"r"(4u * bytes),
                       "r"(smem_addr(&bar))
                       : "memory");
          const double* src[4] = {Auu, Auv, Avu, Avv};
#pragma unroll
          for (int q = 0; q < 4; ++q)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    smem_addr(na_sm + (q * kNaRows + r0) * 27)),
                "l"(src[q] + (t0 + r0) * 27), "r"(bytes), "r"(smem_addr(&bar))
                : "memory");
        }
      } else {
        for (int e = r0 * 27 + tid; e < r1 * 27; e += kNaRows) {
          na_sm[e] = Auu[t0 * 27 + e];
          na_sm[kNaRows * 27 + e] = Auv[t0 * 27 + e];
          na_sm[2 * kNaRows * 27 + e] = Avu[t0 * 27 + e];
          na_sm[3 * kNaRows * 27 + e] = Avv[t0 * 27 + e];
        }
      }
      // the source values while the copies are in flight: neighbours are
      // read directly at (halo) indices, as the reference does, at one
      // offset from the row's own for all rows
      double su[27], sv[27], b0 = 0.0, b1 = 0.0;
      if (mine) {
#pragma unroll
        for (int q = 0; q < 27; ++q) {
          const int kA = q / 9 - 1, jA = (q / 3) % 3 - 1, iA = q % 3 - 1;
          const bool in = k + kA >= 0 && k + kA < nz;
          const long x = in ? t + ((long)jA * V + iA) * nz + kA : t;
          su[q] = xu[x];
          sv[q] = xv[x];
        }
        b0 = bu[t];
        b1 = bv[t];
      }
      if (BULK) {
        ok = bar_wait(smem_addr(&bar), phase);
        if (!__all_sync(0xffffffffu, ok)) {  // give the copies in flight one more bounded wait, then give up
          bar_wait(smem_addr(&bar), phase);
          ok = false;
          break;
        }
        phase ^= 1u;
      }
      __syncwarp();
      double yu = 0.0, yv = 0.0;
      if (mine) {
        // matvec_multiply_structured_3d order: kA, jA, iA
#pragma unroll
        for (int q = 0; q < 27; ++q) {
          const int kA = q / 9 - 1;
          if (k + kA < 0 || k + kA >= nz) continue;
          const double* A = na_sm + tid * 27 + q;
          yu = yu + A[0] * su[q] + A[kNaRows * 27] * sv[q];
          yv = yv + A[2 * kNaRows * 27] * su[q] + A[3 * kNaRows * 27] * sv[q];
        }
        yu -= b0;
        yv -= b1;
        s_r += yu * yu + yv * yv;
        s_b += b0 * b0 + b1 * b1;
      }
      if (t < rows) {
        ru[t] = yu;
        rv[t] = yv;
      }
    } else if (t < rows) {
      ru[t] = 0.0;
      rv[t] = 0.0;
    }
    __syncwarp();  // the rows are free for the next chunk
  }
  if (!ok) s_r = __longlong_as_double(0x7ff8000000000000LL);  // a copy that never arrived: the norms say so
  // warp sums (fixed tree), one partial pair per block
  for (int o = 16; o > 0; o >>= 1) {
    s_r += __shfl_xor_sync(0xffffffffu, s_r, o);
    s_b += __shfl_xor_sync(0xffffffffu, s_b, o);
  }
  int last = 0;
  if (tid == 0) {
    __stcg(reinterpret_cast<double2*>(S->partial) + blockIdx.x, make_double2(s_r, s_b));
    __threadfence();
    const unsigned share = bp::ticket_share(blockIdx.x, gridDim.x);
    last = atomicAdd(&S->ticket, share) + share == 0u ? 1 : 0;
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return;
  // the last block sums every partial, each thread in block order
  __threadfence();
  double a = 0.0, b = 0.0;
#pragma unroll 8
  for (unsigned q = tid; q < gridDim.x; q += kNaRows) {
    const double2 pq = __ldcg(reinterpret_cast<const double2*>(S->partial) + q);
    a += pq.x;
    b += pq.y;
  }
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (tid == 0) {
    const double nr = sqrt(a), nb = sqrt(b);
    norms[0] = nr;
    norms[1] = nb;
    norms[2] = nb > 0.0 ? nr / nb : 0.0;
  }
}

// The CUDA context current on the calling thread (the driver's
// cuCtxGetCurrent, reached through the runtime so that no driver library
// is linked), or null when it cannot be asked.
using CtxGetCurrent = int (*)(void**);
void* current_context() {
  static CtxGetCurrent fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<CtxGetCurrent>(f);
  }();
  void* c = nullptr;
  if (!fn || fn(&c) != 0) return nullptr;
  return c;
}

void* g_na_ctx[kNaMaxDevices] = {nullptr};

// Device address of the scratch array on the current device, looked up
// once per device and context: after cudaDeviceReset (or any teardown of
// the device's context) the module is loaded again into the new context,
// where the array may sit at another address, so a change of the current
// context triggers a new lookup.
NaScratch* scratch_for_current_device(int* status) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNaMaxDevices) {
    *status = BP_ERR_NO_DEVICE;
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(g_na_mutex);
  void* ctx = current_context();
  if (!g_na_ptr[dev] || !ctx || ctx != g_na_ctx[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_na_scratch);
    if (e != cudaSuccess || !p) {
      std::fprintf(stderr, "bp_residual_noalloc: cudaGetSymbolAddress failed: %s\n",
                   cudaGetErrorString(e));
      *status = BP_ERR_CUDA;
      return nullptr;
    }
    g_na_ptr[dev] = static_cast<NaScratch*>(p);
    g_na_ctx[dev] = current_context();  // current now that the lookup made the runtime initialise it
  }
  *status = BP_OK;
  return g_na_ptr[dev];
}

}  // namespace

extern "C" int bp_residual_noalloc(int nx, int ny, int nz, int periodic,
                                   const int* active_vertex, const double* Auu,
                                   const double* Auv, const double* Avu, const double* Avv,
                                   const double* xu, const double* xv, const double* bu,
                                   const double* bv, double* resid_u, double* resid_v,
                                   double* norms, void* stream) {
  if (nx < 6 || ny < 6 || nz < 1) return BP_ERR_ARGS;
  if (!active_vertex || !Auu || !Auv || !Avu || !Avv || !xu || !xv || !bu || !bv || !resid_u ||
      !resid_v || !norms)
    return BP_ERR_ARGS;
  const long rows = (long)nz * (nx - 1) * (ny - 1);
  if (rows > kNaMaxRows) {
    std::fprintf(stderr,
                 "bp_residual_noalloc: %ld rows exceed the fixed scratch limit of %ld "
                 "(nz*(nx-1)*(ny-1)); use bp_matvec for larger systems\n",
                 rows, kNaMaxRows);
    return BP_ERR_ARGS;
  }
  int st = BP_OK;
  NaScratch* S = scratch_for_current_device(&st);
  if (!S) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long chunks = (rows + kNaRows - 1) / kNaRows;
  const unsigned blocks = (unsigned)(chunks < kNaBlocks ? chunks : kNaBlocks);
  const size_t smem = sizeof(double) * 4 * kNaRows * 27;
  const bool aligned = !((reinterpret_cast<uintptr_t>(Auu) | reinterpret_cast<uintptr_t>(Auv) |
                          reinterpret_cast<uintptr_t>(Avu) | reinterpret_cast<uintptr_t>(Avv)) & 15u);
  auto kernel = aligned ? k_resid_ref_layout<true> : k_resid_ref_layout<false>;
  kernel<<<blocks, kNaRows, smem, s>>>(nx, ny, nz, periodic, active_vertex, Auu, Auv, Avu, Avv, xu, xv, bu, bv,
                                       resid_u, resid_v, norms, S);
  return cudaGetLastError() == cudaSuccess ? BP_OK : BP_ERR_CUDA;
}
