// hostengine.cpp -- TEST ONLY.  The host engine (cism_b200/csrc/bp_engine.cpp)
// on a fake CUDA runtime: "device" memory is host memory, copies happen at
// once, kernels do next to nothing (a linear solve or a Picard loop "converges"
// at its first update), and a launch can be refused on demand, so that what
// the engine does around its launches can be tested without a GPU.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>

#include "bp_guess.h"
#include "bp_kernels.h"

using namespace bp;

namespace {
struct Fake {
  cudaError_t last = cudaSuccess;
  int capturing = 0;       // a capture is open on the stream
  int refuse = 0;          // 1: Krylov matvecs inside a capture, 2: all Krylov matvecs
  int graph_launches = 0, resident_halo = 0;
  bool copies_open = false;  // host-to-device copies since the last synchronisation
  DevView v;               // of the last launch
} F;

cudaError_t fail(cudaError_t e) { return F.last = e; }
void seen(const DevView& v) { F.v = v; }
void pcg_done(const DevView& v) {
  for (int b = 0; b < v.ninst; ++b) {
    v.st[b].pcg_active = 0;
    v.st[b].pcg_converged = 1;
  }
  v.cnt->pcg_active = 0;
}
void picard_done(const DevView& v) {
  for (int b = 0; b < v.ninst; ++b) {
    v.st[b].picard_active = 0;
    v.st[b].picard_converged = v.st[b].pcg_converged = 1;
    v.st[b].picard_iter = 1;
  }
  v.cnt->picard_active = 0;
}
}  // namespace

extern "C" {
// -- the test's controls -----------------------------------------------------
void fake_refuse(int what) { F.refuse = what; }
int fake_capturing() { return F.capturing; }
int fake_graph_launches() { return F.graph_launches; }
// most halo columns of a tile in the last question for resident CTAs
int fake_resident_halo() { return F.resident_halo; }
int fake_copies_open() { return F.copies_open ? 1 : 0; }
// Slots of the zeroed node vectors that belong to no column (the end of each
// instance's last tile) and do not hold zero; -1 where there are none.
long fake_nonzero_holes() {
  const DevView& v = F.v;
  long holes = 0, bad = 0;
  for (int t = 0; t < v.ntiles; ++t)
    for (int k = 0; k < v.nz; ++k)
      for (int c = v.tile_ncols[t]; c < v.W; ++c, ++holes)
        for (const double2* vec : {v.x, v.b, v.r, v.d0, v.z, v.q, v.Az, v.Dinv, v.usav}) {
          const double2 a = vec[v.tile_start[t] + (size_t)k * v.W + c];
          bad += a.x != 0.0 || a.y != 0.0;
        }
  return holes ? bad : -1;
}

// -- runtime -----------------------------------------------------------------
cudaError_t cudaGetLastError() {
  const cudaError_t e = F.last;
  F.last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetLimit(size_t* v, cudaLimit) { *v = 0; return cudaSuccess; }
cudaError_t cudaDeviceSetLimit(cudaLimit, size_t) { return cudaSuccess; }
cudaError_t cudaCtxResetPersistingL2Cache() { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 30; return cudaSuccess; }
// every byte 0x5a: what the engine does not write does not pass for zero
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = std::malloc(n);
  if (*p) std::memset(*p, 0x5a, n);
  return *p ? cudaSuccess : fail(cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  std::memcpy(d, s, n);
  F.copies_open = F.copies_open || k == cudaMemcpyHostToDevice;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)8; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  if (F.capturing) return fail(cudaErrorStreamCaptureUnsupported);
  F.copies_open = false;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)8; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)8; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  if (F.capturing) return fail(cudaErrorIllegalState);
  F.capturing = 1;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t s, cudaGraph_t, const cudaGraphNode_t*,
                                          const cudaGraphEdgeData*, size_t, cudaStreamCaptureMode m) {
  return cudaStreamBeginCapture(s, m);
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  if (!F.capturing) return fail(cudaErrorIllegalState);
  F.capturing = 0;
  *g = (cudaGraph_t)8;
  return cudaSuccess;
}
cudaError_t cudaStreamGetCaptureInfo_v2(cudaStream_t, cudaStreamCaptureStatus* st, unsigned long long*, cudaGraph_t*,
                                        const cudaGraphNode_t** deps, size_t* n) {
  static const cudaGraphNode_t node = (cudaGraphNode_t)8;
  *st = cudaStreamCaptureStatusActive;
  *deps = &node;
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) { *g = (cudaGraph_t)8; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t, unsigned, unsigned) {
  *h = 8;
  return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t* n, size_t* k) {
  if (n) *n = (cudaGraphNode_t)8;
  *k = 1;
  return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t* n, cudaGraph_t, const cudaGraphNode_t*, size_t, cudaGraphNodeParams* p) {
  static cudaGraph_t body = (cudaGraph_t)8;
  *n = (cudaGraphNode_t)8;
  p->conditional.phGraph_out = &body;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t)8;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
  ++F.graph_launches;
  pcg_done(F.v);
  picard_done(F.v);
  return cudaSuccess;
}
}  // extern "C"

// -- kernels -----------------------------------------------------------------
namespace bp {
cudaError_t upload_ref_tables() { return cudaSuccess; }
void set_pdl(bool) {}
int resident_ctas(const DevView& v, int, int num_sms) {
  F.resident_halo = v.halo_max;
  return v.W * v.nz <= 256 ? num_sms : 0;
}
int staged_per_sm(const DevView&) { return 1; }
int krylov_resident_ctas(const DevView&, int, int) { return 1; }
void launch_staged_desc(const DevView& v, unsigned char*, cudaStream_t) { seen(v); }
cudaError_t launch_pcg_resident(const DevView& v, int, cudaStream_t) { seen(v); pcg_done(v); return cudaSuccess; }
void launch_mv(int mode, const DevView& v, cudaStream_t) {
  seen(v);
  const bool krylov = mode == MV_STD_A || mode == MV_CG_FIRST || mode == MV_CG1;
  if (krylov && (F.refuse == 2 || (F.refuse == 1 && F.capturing))) fail(cudaErrorInvalidValue);
}
void launch_std_update(bool, const DevView& v, cudaStream_t) { seen(v); pcg_done(v); }
void launch_cg_update(bool, const DevView& v, cudaStream_t) { seen(v); pcg_done(v); }
void launch_cg_first_update(const DevView& v, cudaStream_t) { seen(v); }
void launch_picard_check(const DevView& v, cudaStream_t) { seen(v); picard_done(v); }
void launch_std_dir(const DevView& v, cudaStream_t) { seen(v); }
void launch_picard_begin(const DevView& v, cudaStream_t) { seen(v); }
void launch_save_usav(const DevView& v, cudaStream_t) { seen(v); }
void launch_slide_beta(const DevView&, cudaStream_t) {}
void launch_asm_qp(const DevView&, cudaStream_t) {}
void launch_asm_rows(const DevView&, cudaStream_t) {}
void launch_rhs(const DevView&, cudaStream_t) {}
void launch_l1l2_velocity(const DevView&, cudaStream_t) {}
void launch_diva_beta(const DevView&, cudaStream_t) {}
void launch_diva_velocity(const DevView&, cudaStream_t) {}
void launch_loop_cond(cudaGraphConditionalHandle, const DevView&, bool, int*, int, bool, cudaStream_t) {}
void launch_make_a32(const DevView&, cudaStream_t) {}
void launch_sia_factor(const DevView&, cudaStream_t) {}
void launch_matvec_plain(const DevView&, const double2*, double2*, cudaStream_t) {}
void launch_gather_matrix(const DevView&, const double*, const int*, long, long, cudaStream_t) {}
void launch_dinv(const DevView&, int, cudaStream_t) {}
void launch_bb(const DevView&, cudaStream_t) {}
void launch_diagnostics(const DevView&, int, double*, double*, cudaStream_t) {}
void launch_levels_from_2d(const DevView&, double2*, int, cudaStream_t) {}
void launch_corner_beta(const DevView&, cudaStream_t) {}
int launch_tune_mv(int, int, int, const DevView&, cudaStream_t) { return -1; }
void launch_pack(const DevView& v, const double2* x, double* u, double* w, cudaStream_t) {
  seen(v);
  for (long t = 0; t < (long)v.ncols * v.nz; ++t) {
    const double2 a = x[node_of(v, (int)(t / v.nz), (int)(t % v.nz))];
    u[t] = a.x;
    w[t] = a.y;
  }
}
void launch_unpack(const DevView& v, int c0, int c1, const double* u, const double* w, double2* x, cudaStream_t) {
  seen(v);
  for (long t = (long)c0 * v.nz; t < (long)c1 * v.nz; ++t)
    x[node_of(v, (int)(t / v.nz), (int)(t % v.nz))] = double2{u[t], w[t]};
}

GuessNet* guess_net_load(const char*, std::string* err) { *err = "no network here"; return nullptr; }
void guess_net_free(GuessNet*) {}
int guess_net_run(GuessNet*, const HostPlan&, const DevView&, const std::vector<int>&, double2*, cudaStream_t, int*) {
  return 6;
}
}  // namespace bp
