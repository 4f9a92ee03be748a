// bp_kernels.cu -- sm_100a kernels of the Blatter-Pattyn solve.
//
// All node kernels walk tiles of at most kTile consecutive nodes (one tile per CTA
// iteration, grid-stride, so the same code runs as a one-shot grid or as a
// persistent grid).  A tile never spans two instances, so per-instance
// reductions are: block reduce -> per-tile partial -> the last CTA of the
// instance (atomic ticket) sums the partials in tile order and runs the
// scalar update (alpha, beta, convergence) on the device.  The result is
// bitwise reproducible run to run and needs no host round trip.
#include <cstdio>
#include <type_traits>

#include "bp_body.h"
#include "bp_b200.h"
#include "bp_kernels.h"

#include <cstdlib>

namespace bp {

__constant__ RefTables c_T;

// ---------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------
template <int NV, bool MAX0>
__device__ __forceinline__ void block_reduce(double (&val)[NV], double* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double x = val[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double y = __shfl_xor_sync(0xffffffffu, x, o);
      x = (MAX0 && i == 0) ? fmax(x, y) : x + y;
    }
    if (lane == 0) sm[i * 32 + warp] = x;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      double x = lane < nw ? sm[i * 32 + lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, x, o);
        x = (MAX0 && i == 0) ? fmax(x, y) : x + y;
      }
      val[i] = x;
    }
  }
  __syncthreads();
}

// Reduce NV values of this tile; the last tile of the instance sums all
// tile partials of the instance in tile order and calls fin(inst, sums).
// U: tiles whose partials a thread has in flight there, where the kernel has
// registers to spare (k_std_update: 15.3 -> 14.1 us at 1,600 tiles; k_resid
// loses more to its occupancy than the tail gains, 53 -> 66 us).
template <int NV, bool MAX0, int U = 1, typename Fin>
__device__ __forceinline__ void tile_finish(const DevView& v, int t, int inst,
                                            double (&val)[NV], Fin fin) {
  __shared__ double sm[NV * 32];
  __shared__ int last;
  block_reduce<NV, MAX0>(val, sm);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) v.partials[(size_t)i * v.ntiles + t] = val[i];
    __threadfence();
    const InstParams& ip = v.inst[inst];
    const unsigned ntl = (unsigned)(ip.tile_end - ip.tile_begin);
    const unsigned prev = atomicAdd(&v.tile_counter[inst], 1u);
    last = (prev == ntl - 1) ? 1 : 0;
  }
  __syncthreads();
  if (last) {
    __threadfence();
    const InstParams& ip = v.inst[inst];
    double s[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) s[i] = 0.0;
    for (int t0 = ip.tile_begin + threadIdx.x; t0 < ip.tile_end; t0 += U * blockDim.x) {
      double p[U][NV];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int tt = t0 + u * blockDim.x;
          p[u][i] = U == 1 || tt < ip.tile_end ? __ldcg(v.partials + (size_t)i * v.ntiles + tt) : 0.0;
        }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (U == 1 || t0 + u * (int)blockDim.x < ip.tile_end)
#pragma unroll
          for (int i = 0; i < NV; ++i) s[i] = (MAX0 && i == 0) ? fmax(s[i], p[u][i]) : s[i] + p[u][i];
    }
    block_reduce<NV, MAX0>(s, sm);
    if (threadIdx.x == 0) {
      v.tile_counter[inst] = 0;
      fin(inst, s);
      __threadfence();
    }
  }
  __syncthreads();
}

// How a scalar update ends an instance's linear solve or its run.  The
// launched kernels (Shared = true: one thread per instance, on the state in
// device memory) count it off in the problem's counters at once; the CTAs
// of a resident PCG each update their own copy of the state, and one of
// them settles the counters when it writes the state back.
template <bool Shared>
__device__ __forceinline__ void pcg_stop(const DevView& v, InstState& S, bool converged) {
  S.pcg_active = 0;
  S.pcg_converged = converged ? 1 : 0;
  S.pcg_iters_last = S.pcg_iter;
  S.pcg_iters_total += S.pcg_iter;
  if (Shared) atomicSub(&v.cnt->pcg_active, 1);
}

template <bool Shared>
__device__ __forceinline__ void fail(const DevView& v, InstState& S, int code) {
  if (S.status == BP_OK || S.status == BP_WARN_PCG_NOT_CONVERGED) S.status = code;
  if (S.pcg_active) pcg_stop<Shared>(v, S, false);
  if (S.refine_active) {
    S.refine_active = 0;
    if (Shared) atomicSub(&v.cnt->refine_active, 1);
  }
  if (S.picard_active) {
    S.picard_active = 0;
    if (Shared) atomicSub(&v.cnt->picard_active, 1);
  }
}

__device__ __forceinline__ bool is_nan(double x) { return x != x; }

struct TileRange {
  int inst, n0, nend, ncols, col0;
};

// Programmatic dependent launch: the PCG kernels are launched so that the
// next one may be scheduled while its predecessor drains; each calls
// pdl_wait() (which returns once the predecessor grid has completed and its
// writes are visible) before it reads anything, in every CTA, so a grid
// also completes only after its predecessor.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_next() { asm volatile("griddepcontrol.launch_dependents;"); }

__device__ __forceinline__ TileRange tile_range(const DevView& v, int t) {
  TileRange r;
  r.inst = v.tile_inst[t];
  r.n0 = v.tile_start[t];
  r.nend = v.tile_end[t];
  r.ncols = v.tile_ncols[t];
  r.col0 = v.tile_col0[t];
  return r;
}

// Thread i of a tile's CTA owns node n0 + i: level i >> lsh, column col0 +
// (i & (W-1)); the slots past the block's columns are holes.
__device__ __forceinline__ bool tile_mine(const DevView& v, const TileRange& R, int i) {
  return R.n0 + i < R.nend && (i & (v.W - 1)) < R.ncols;
}
__device__ __forceinline__ int tile_col(const DevView& v, const TileRange& R, int i) {
  return R.col0 + (i & (v.W - 1));
}
__device__ __forceinline__ int tile_k(const DevView& v, int i) { return i >> v.lsh; }

// ---------------------------------------------------------------------
// Picard iteration start (one CTA): counter, reset of the PCG state.
// ---------------------------------------------------------------------
__global__ void k_picard_begin(DevView v) {
  __shared__ int cnt;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  int mine = 0;
  for (int i = threadIdx.x; i < v.ninst; i += blockDim.x) {
    InstState& S = v.st[i];
    if (!S.picard_active) continue;
    S.picard_iter += 1;
    S.nonzero = 0;
    S.pcg_active = 1;
    S.pcg_iter = 1;
    S.pcg_converged = 0;
    S.rz = 1.0;
    S.rz_old = 1.0;
    S.alpha = 0.0;
    S.beta = 0.0;
    S.err = -1.0;
    S.refine_steps = 0;
    S.refine_active = 1;
    S.inner_iter = 0;
    S.pcg_iters_last = 0;
    S.krylov_fp64 = 0;
    S.need_true = 0;
    S.restart = 0;
    S.last_true_iter = 0;
    S.r_true = 0.0;
    ++mine;
  }
  atomicAdd(&cnt, mine);
  __syncthreads();
  if (threadIdx.x == 0) {
    v.cnt->pcg_active = cnt;
    v.cnt->refine_active = cnt;
  }
}

// calcbeta with a velocity-dependent law at the start of a Picard iteration
// (glissade_velo_higher.F90:2502-2517): beta of every column of an active
// instance from its basal velocity x(nz-1).  An invalid beta (negative or
// NaN, glissade_basal_traction.F90:570-582) marks the instance; k_rhs ends
// it with BP_ERR_BAD_BETA before its linear solve.
__global__ void __launch_bounds__(kTile) k_slide_beta(DevView v) {
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < v.ncols; col += gridDim.x * blockDim.x) {
    const int inst = v.col_inst[col];
    const InstParams& ip = v.inst[inst];
    InstState& S = v.st[inst];
    if (!S.picard_active || ip.slide.law == 0) continue;
    const size_t nc = (size_t)v.ncols;
    // the basal velocity: DIVA's 3-D one (:2240-2243), else the bed node
    const double2 ub = v.diva ? v.x3[(size_t)col * (v.nl + 1) + v.nl] : v.x[node_of(v, col, v.nz - 1)];
    const double beta = slide_beta(ip.slide, v.col_slide[col], v.col_slide[nc + col],
                                   v.col_slide[2 * nc + col], ub.x, ub.y);
    if (!(beta >= 0.0) && (S.status == BP_OK || S.status == BP_WARN_PCG_NOT_CONVERGED))
      S.status = BP_ERR_BAD_BETA;
    v.col_beta[col] = beta;
  }
}

// Corner betas of the bed faces for the standard basal assembly
// (basal_sliding_bc :8234-8363) after k_slide_beta: the corner's column,
// or 0 where the corner has no column (a vertex outside an outflow domain,
// zeroed by the staggered halo update).
__global__ void __launch_bounds__(kTile) k_cell_beta(DevView v) {
  for (int cell = blockIdx.x * blockDim.x + threadIdx.x; cell < v.ncells; cell += gridDim.x * blockDim.x) {
    const int inst = v.cell_inst[cell];
    if (!v.st[inst].picard_active || v.inst[inst].slide.law == 0) continue;
    for (int q = 0; q < 4; ++q) {
      const int col = v.cell_cols[(size_t)q * v.ncells + cell];
      v.cell_beta[(size_t)q * v.ncells + cell] = col >= 0 ? v.col_beta[col] : 0.0;
    }
  }
}

__global__ void __launch_bounds__(kTile) k_save_usav(DevView v) {
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    if (!v.st[R.inst].picard_active) continue;
    const int n = R.n0 + threadIdx.x;
    if (tile_mine(v, R, threadIdx.x)) v.usav[n] = v.x[n];
  }
}

// ---------------------------------------------------------------------
// Assembly pass 1: thread = (element, quadrature point).
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_asm_qp(DevView v) {
  const long gtid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int e = (int)(gtid >> 3), p = (int)(gtid & 7);
  bool valid = e < v.nelem;
  int inst = 0;
  if (valid) {
    inst = v.cell_inst[e / (v.nz - 1)];
    valid = v.st[inst].picard_active != 0;
  }
  const unsigned mask = __ballot_sync(0xffffffffu, valid);
  if (!valid) return;
  double out[10], eq = 0.0;
  const bool ok = qp_element_point(v, c_T, e, p, out, &eq);
  if (!ok) {
    atomicExch(&v.st[inst].status, BP_ERR_SINGULAR_JAC);
    eq = 0.0;
#pragma unroll
    for (int i = 0; i < 10; ++i) out[i] = 0.0;
  }
  double2* dst = reinterpret_cast<double2*>(v.qp + ((size_t)e * 8 + p) * 10);
#pragma unroll
  for (int i = 0; i < 5; ++i) dst[i] = make_double2(out[2 * i], out[2 * i + 1]);
  // element average of the quadrature-point viscosity, in point order
  const int lane0 = (threadIdx.x & 31) & ~7;
  double s = 0.0;
#pragma unroll
  for (int q = 0; q < 8; ++q) s += __shfl_sync(mask, eq, lane0 + q);
  if (p == 0) v.efvs[e] = s / 8.0;
}

// Pass 1 of the shallow-shelf assembly: one thread per (active cell, 2-D
// point), the cell's viscosity the mean of its 4 points (:5539-5545).
// LAYERS: the L1L2 and DIVA solves, with a viscosity per layer (kept in
// a per-thread array the shallow-shelf instance does without).
template <bool LAYERS>
__global__ void __launch_bounds__(256) k_asm2_qp(DevView v) {
  const long gtid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int c = (int)(gtid >> 2), p = (int)(gtid & 3);
  bool valid = c < v.ncells;
  int inst = 0;
  if (valid) {
    inst = v.cell_inst[c];
    valid = v.st[inst].picard_active != 0;
  }
  const unsigned mask = __ballot_sync(0xffffffffu, valid);
  if (!valid) return;
  double out[5], eq = 0.0, ek[LAYERS ? kNzMax - 1 : 1];
  const bool ok = qp2_element_point(v, c_T, c, p, out, &eq, LAYERS ? ek : nullptr);
  if (!ok) {
    atomicExch(&v.st[inst].status, BP_ERR_SINGULAR_JAC);
    eq = 0.0;
    for (int i = 0; i < 5; ++i) out[i] = 0.0;
  }
  double* dst = v.qp + ((size_t)c * 8 + p) * 10;
  for (int i = 0; i < 5; ++i) dst[i] = out[i];
  const int lane0 = (threadIdx.x & 31) & ~3;
  if (LAYERS) {  // efvs(k) = the mean of the layer's point values (:5565-5572)
    for (int k = 0; k < v.nl; ++k) {
      const double e = ok ? ek[k] : 0.0;
      double sum = 0.0;
#pragma unroll
      for (int q = 0; q < 4; ++q) sum += __shfl_sync(mask, e, lane0 + q);
      if (p == 0) v.efvs[(size_t)c * v.nl + k] = sum / 4.0;
    }
    return;
  }
  double sum = 0.0;
#pragma unroll
  for (int q = 0; q < 4; ++q) sum += __shfl_sync(mask, eq, lane0 + q);
  if (p == 0) v.efvs[c] = sum / 4.0;
}

// L1L2 3-D velocity after the Picard loop (compute_3d_velocity_L1L2,
// glissade_velo_higher.F90:5834-6356): the cell pass (l1l2_cell), then
// one thread per column integrates from the bed up (l1l2_column).  Run
// once per solve; bounded by the nl * 4 cell values each column reads.
__global__ void __launch_bounds__(256) k_l1l2_cells(DevView v) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < v.ncells) l1l2_cell(v, c);
}

__global__ void __launch_bounds__(256) k_l1l2_columns(DevView v) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col < v.ncols) l1l2_column(v, col);
}

// DIVA, every Picard iteration of an active instance: after assembly pass
// 1 the cells' omega integrals (k_diva_cells), beta_eff at the columns
// (k_diva_beta) and at the bed-face corners for the standard basal
// assembly (k_diva_cell_beta); after the linear solve the traction and
// the 3-D velocity (k_diva_velocity).
__global__ void __launch_bounds__(256) k_diva_cells(DevView v) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < v.ncells && v.st[v.cell_inst[c]].picard_active) diva_cell_integrals(v, c);
}

__global__ void __launch_bounds__(256) k_diva_beta(DevView v) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col < v.ncols && v.st[v.col_inst[col]].picard_active) diva_column_beta(v, col);
}

__global__ void __launch_bounds__(256) k_diva_cell_beta(DevView v) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= v.ncells || !v.st[v.cell_inst[cell]].picard_active) return;
  for (int q = 0; q < 4; ++q) {
    const int col = v.cell_cols[(size_t)q * v.ncells + cell];
    v.cell_beta[(size_t)q * v.ncells + cell] = col >= 0 ? v.col_beff[col] : 0.0;
  }
}

__global__ void __launch_bounds__(256) k_diva_velocity(DevView v) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col < v.ncols && v.st[v.col_inst[col]].picard_active) diva_column_velocity(v, col);
}

// ---------------------------------------------------------------------
// Assembly pass 2 + basal BC + Dirichlet BC: thread = (block B, node).
// ---------------------------------------------------------------------
enum { ASM_ROWS = 0, ASM_GATHER = 1, ASM_2D = 2 };

// Element-centric pass 2a: thread = (element, corner nr); the corner's rows
// of the element's four blocks (element_row_blocks) into Ke, the eight
// threads of an element writing 64 consecutive doubles per block.
__global__ void __launch_bounds__(256, 2) k_asm_elem(DevView v) {
  const long gtid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int e = (int)(gtid >> 3), nr = (int)(gtid & 7);
  if (e >= v.nelem) return;
  if (!v.st[v.cell_inst[e / (v.nz - 1)]].picard_active) return;
  double K[32];
  element_row_blocks(c_T, v.qp + (size_t)e * 80, nr, K);
  double2* out = reinterpret_cast<double2*>(v.Ke + (size_t)e * 256 + nr * 8);
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int i = 0; i < 4; ++i) out[b * 32 + i] = make_double2(K[b * 8 + 2 * i], K[b * 8 + 2 * i + 1]);
}
template <int B, int MODE>
__device__ __forceinline__ bool asm_row(const DevView& v, int n, int col, int k) {
  double acc[27];
  if (MODE == ASM_2D) row_assemble2<B>(v, c_T, col, acc);
  else if (MODE == ASM_GATHER) row_gather<B>(v, v.Ke, col, k, acc);
  else row_assemble<B>(v, c_T, col, k, acc);
  row_basal<B>(v, c_T, col, k, acc);
  const double adj = row_dirichlet<B>(v, col, k, acc);
  bool nz = false;
  double* Ad = reinterpret_cast<double*>(v.A);
  const size_t np = (size_t)v.npad;
  const int h = B >> 1, comp = B & 1;
#pragma unroll
  for (int m = 0; m < 27; ++m) {
    nz |= (acc[m] != 0.0);
    if (v.sym) {
      if (m >= 13) Ad[(((size_t)(h * 14 + m - 13)) * np + n) * 2 + comp] = acc[m];
    } else {
      Ad[(((size_t)(h * 27 + m)) * np + n) * 2 + comp] = acc[m];
    }
  }
  v.badj[(size_t)B * np + n] = adj;
  return nz;
}

// MODE: ASM_ROWS (3-D, each row integrates its incident elements),
// ASM_GATHER (3-D, each row sums the element rows k_asm_elem stored) or
// ASM_2D (the rows of the 2-D solves: shallow-shelf, L1L2; nz = 1).
template <int MODE>
__global__ void __launch_bounds__(kTile) k_asm_rows(DevView v) {
  const int B = blockIdx.y;
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    if (!v.st[R.inst].picard_active) continue;
    const int n = R.n0 + threadIdx.x;
    int nzl = 0;
    if (tile_mine(v, R, threadIdx.x)) {
      const int col = tile_col(v, R, threadIdx.x), k = tile_k(v, threadIdx.x);
      switch (B) {
        case 0: nzl = asm_row<0, MODE>(v, n, col, k); break;
        case 1: nzl = asm_row<1, MODE>(v, n, col, k); break;
        case 2: nzl = asm_row<2, MODE>(v, n, col, k); break;
        default: nzl = asm_row<3, MODE>(v, n, col, k); break;
      }
    }
    if (__syncthreads_or(nzl) && threadIdx.x == 0) atomicOr(&v.st[R.inst].nonzero, 1);
  }
}

// ---------------------------------------------------------------------
// Right-hand side (load + Dirichlet moves), preconditioner, (b,b).
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(kTile) k_rhs(DevView v) {
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    if (!v.st[R.inst].picard_active) continue;
    const InstParams& ip = v.inst[R.inst];
    const int n = R.n0 + threadIdx.x;
    double part[1] = {0.0};
    if (tile_mine(v, R, threadIdx.x)) {
      const size_t np = (size_t)v.npad;
      const uint8_t dm = v.dmask[n];
      const double2 ld = v.load[n];
      const double2 xn = v.x[n];
      double bu = ld.x - v.badj[0 * np + n] - v.badj[1 * np + n];
      double bv = ld.y - v.badj[2 * np + n] - v.badj[3 * np + n];
      if (dm & 1) bu = xn.x;
      if (dm & 2) bv = xn.y;
      v.b[n] = make_double2(bu, bv);
      double2 di = make_double2(1.0, 1.0);
      if (ip.precond == 1) {
        const double du = diag_u(v, n), dv = diag_v(v, n);
        di.x = du != 0.0 ? 1.0 / du : 0.0;
        di.y = dv != 0.0 ? 1.0 / dv : 0.0;
      }
      v.Dinv[n] = di;
      part[0] = bu * bu + bv * bv;
    }
    tile_finish<1, false>(v, t, R.inst, part, [&](int inst, const double* s) {
      InstState& S = v.st[inst];
      S.bb = s[0];
      S.L2_rhs = sqrt(s[0]);
      if (S.status == BP_ERR_SINGULAR_JAC || S.status == BP_ERR_BAD_BETA) {
        fail<true>(v, S, S.status);
      } else if (!S.nonzero) {
        S.status = BP_ZERO_MATRIX;
        S.zero_x = 1;
        fail<true>(v, S, BP_ZERO_MATRIX);
      } else if (v.solve2d && !v.diva && v.inst[inst].which_babc == 6) {
        // 2-D solve on a no-slip bed: the 2-D velocity is zero and nothing is solved
        // (glissade_velo_higher.F90:3227-3240)
        S.frozen = 1;
        S.L2_norm = 0.0;
        S.L2_rel = 0.0;
        S.pcg_iter = 0;
        pcg_stop<true>(v, S, true);
        if (S.refine_active) {
          S.refine_active = 0;
          atomicSub(&v.cnt->refine_active, 1);
        }
      }
    });
  }
}

// ---------------------------------------------------------------------
// SIA column preconditioner on a tile of whole columns: every thread puts
// its node's r and its node's factors (a, beta, gamma for u and v) into
// shared memory, one thread per (column, component) runs the two Thomas
// sweeps from there (sia_sweeps), every thread takes back its z.  The
// sweeps are a chain of dependent steps; with the factors staged by
// coalesced loads beforehand, no step of the chain waits on global memory.
// Called by all threads of the CTA (uniform per tile).
// ---------------------------------------------------------------------
struct SiaTile {
  double s[2 * kTile], a[2 * kTile], b[2 * kTile], g[2 * kTile];
};

__device__ __forceinline__ double2 sia_tile(const DevView& v, const TileRange& R, double2 r) {
  __shared__ SiaTile T;
  const int i = threadIdx.x, nz = v.nz;
  const bool mine = tile_mine(v, R, i);
  // shared memory holds the tile column by column: j = c * nz + k
  const int k = tile_k(v, i), j = (i & (v.W - 1)) * nz + k;
  if (mine) {
    const size_t n = (size_t)R.n0 + i, np = (size_t)v.npad;
    const double2 fa = v.sia_f[n], fb = v.sia_f[np + n], fg = v.sia_f[2 * np + n];
    T.s[2 * j] = r.x;
    T.s[2 * j + 1] = r.y;
    T.a[2 * j] = fa.x;
    T.a[2 * j + 1] = fa.y;
    T.b[2 * j] = fb.x;
    T.b[2 * j + 1] = fb.y;
    T.g[2 * j] = fg.x;
    T.g[2 * j + 1] = fg.y;
  }
  __syncthreads();
  if (i < 2 * R.ncols) {
    const int c = i >> 1, h = i & 1, o = 2 * c * nz + h;
    sia_sweeps(
        nz, [&](int kk) { return SiaFac{T.a[o + 2 * kk], T.b[o + 2 * kk], T.g[o + 2 * kk]}; }, &T.s[o], 2);
  }
  __syncthreads();
  const double2 z = mine ? make_double2(T.s[2 * j], T.s[2 * j + 1]) : make_double2(0.0, 0.0);
  __syncthreads();  // T is reused by the CTA's next tile
  return z;
}

// z = M^-1 r for the instance's preconditioner (diagonal or none: D^-1
// from k_rhs / k_dinv; SIA: column solves).  Called by all threads.
__device__ __forceinline__ double2 precondition(const DevView& v, const TileRange& R, bool mine, size_t n,
                                                double2 r) {
  if (v.inst[R.inst].precond == 2) return sia_tile(v, R, r);
  if (!mine) return make_double2(0.0, 0.0);
  const double2 di = v.Dinv[n];
  return make_double2(r.x * di.x, r.y * di.y);
}

// ---------------------------------------------------------------------
// PCG kernels.  Every Krylov matvec reads one stored source vector (d for
// the standard PCG, z = D^-1 r for Chronopoulos-Gear, x for residuals), so
// each matvec is a plain y = A s with its dot products fused in.  Storage
// variants: full FP64 rows, symmetric FP64, symmetric FP32 (Krylov matvecs
// of the mixed path; residuals always use the FP64 matrix).
// ---------------------------------------------------------------------
enum { ST_FULL = 0, ST_SYM = 1, ST_SYM32 = 2 };

struct SrcX {
  const double2* x;
  __device__ double2 operator()(size_t m) const { return x[m]; }
};

template <int STORE>
__device__ __forceinline__ double2 mv_row(const DevView& v, int col, int k, size_t n,
                                          const double2* s) {
  const SrcX src{s};
  if (STORE == ST_FULL) return matvec_row(v, v.A, col, k, n, src);
  if (STORE == ST_SYM) return matvec_row_sym(v, v.A, col, k, n, src);
  return matvec_row_sym32(v, v.A32, col, k, n, src);
}

// Mixed precision (iterative refinement): the Krylov iteration runs on the
// FP32 matrix with FP64 vectors and reductions; the FP64 residual b - A x
// replaces the recurrence residual only once the latter has fallen by
// inner_tol since the last replacement (or below the final tolerance, or
// after 500 iterations), and each replacement restarts the Krylov process,
// so every cycle is a clean conjugate-gradient solve of A32 e = r.  Called
// after iteration pcg_iter; replacements follow iterations that are
// multiples of ncheck.
__device__ __forceinline__ void refine_request(const InstParams& ip, InstState& S, double rr) {
  if (S.pcg_iter % ip.ncheck != 0) return;
  const double rn = sqrt(rr);
  if (rn < ip.inner_tol * S.r_true || rn < 0.5 * ip.pcg_tol * S.L2_rhs ||
      S.pcg_iter - S.last_true_iter >= 500)
    S.need_true = 1;
}

// After a residual r = b - A x with (r,z), (r,r) = s[0], s[1].
template <int MODE, bool Shared>
__device__ __forceinline__ void resid_fin(const DevView& v, const InstParams& ip, InstState& S, const double* s) {
  const double rt = sqrt(s[1]);
  if (MODE == MV_INIT) {
    S.L2_norm = rt;
    S.L2_rel = S.L2_rhs > 0.0 ? S.L2_norm / S.L2_rhs : 0.0;
    S.r_true = rt;
    S.last_true_iter = S.pcg_iter;
  } else {
    S.err = rt / S.L2_rhs;
    S.refine_steps_total += 1;
    if (MODE == MV_REFINE) {
      S.need_true = 0;
      S.last_true_iter = S.pcg_iter;
    }
    if (S.err < ip.pcg_tol) { pcg_stop<Shared>(v, S, true); return; }
    if (S.pcg_iter >= ip.pcg_maxiters) { pcg_stop<Shared>(v, S, false); return; }
    if (MODE == MV_REFINE) {
      // a cycle that did not halve the residual: the FP32 operator is
      // too coarse for this system, finish with the FP64 matrix
      if (rt > 0.5 * S.r_true) S.krylov_fp64 = 1;
      S.r_true = rt;
    }
  }
  if (ip.variant != 3) {  // standard PCG: eta1 of the next iteration
    if (is_nan(s[0])) { fail<Shared>(v, S, BP_ERR_NAN); return; }
    S.beta = MODE == MV_REFINE ? 0.0 : s[0] / S.rz;  // refinement restarts: d = z
    S.rz = s[0];
    if (MODE == MV_CHECK) S.pcg_iter += 1;
  } else if (MODE == MV_REFINE) {
    S.restart = 1;
  }
}

// r = b - A x with the FP64 matrix; z = D^-1 r stored; (r,z) and (r,r).
// MV_INIT starts a linear solve (also compute_residual_vector_3d's norms);
// MV_CHECK is the every-ncheck true residual (pcg:478-536, 1542-1597);
// MV_REFINE the mixed-precision refinement step, for instances that
// requested it.
template <int MODE, int STORE, int MINB>
__global__ void __launch_bounds__(kTile, MINB) k_resid(DevView v) {
  pdl_wait();
  pdl_launch_next();
  constexpr int ST64 = STORE == ST_SYM32 ? ST_SYM : STORE;
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const InstState& S0 = v.st[R.inst];
    if (!S0.pcg_active || (MODE == MV_REFINE && !S0.need_true)) continue;
    const int n = R.n0 + threadIdx.x;
    const bool mine = tile_mine(v, R, threadIdx.x);
    double part[2] = {0.0, 0.0};
    double2 r = make_double2(0.0, 0.0);
    if (mine) {
      const int col = tile_col(v, R, threadIdx.x), k = tile_k(v, threadIdx.x);
      const double2 y = mv_row<ST64>(v, col, k, n, v.x);
      const double2 b = v.b[n];
      r = make_double2(b.x - y.x, b.y - y.y);
    }
    const double2 z = precondition(v, R, mine, n, r);
    if (mine) {
      v.r[n] = r;
      v.z[n] = z;
      part[0] = r.x * z.x + r.y * z.y;
      part[1] = r.x * r.x + r.y * r.y;
    }
    tile_finish<2, false>(v, t, R.inst, part, [&](int inst, const double* s) {
      resid_fin<MODE, true>(v, v.inst[inst], v.st[inst], s);
    });
  }
}

// Krylov matvec of the mixed path: FP32 matrix unless the instance's
// refinement stalled (krylov_fp64), FP64 then.  In timing runs the nodes
// through each precision are counted, to turn the measured time into bytes.
// The FP64 Krylov matvec of an instance whose FP32 refinement stalled,
// out of line: inlined, its registers would count against every launch of
// the FP32 kernel, which is sized to fit 32 registers per thread.
struct MvGeom {
  int nz, ncols, npad, lsh;
  const int* col_nbn;
};
__device__ __noinline__ double2 mv_row_sym64_call(MvGeom g, const double2* A, int col, int k, size_t n,
                                                  const double2* s) {
  return matvec_row_sym(g, A, col, k, n, SrcX{s});
}

template <int STORE>
__device__ __forceinline__ double2 krylov_row(const DevView& v, const InstState& S, int col, int k,
                                              size_t n, const double2* s) {
  if (STORE == ST_SYM32 && S.krylov_fp64)
    return mv_row_sym64_call(MvGeom{v.nz, v.ncols, v.npad, v.lsh, v.col_nbn}, v.A, col, k, n, s);
  return mv_row<STORE>(v, col, k, n, s);
}

template <int STORE>
__device__ __forceinline__ void count_tile(const DevView& v, const InstState& S, const TileRange& R) {
  if (v.mv_nodes && !v.dry && threadIdx.x == 0) {
    const bool f32 = STORE == ST_SYM32 && !S.krylov_fp64;
    atomicAdd(&v.mv_nodes[f32 ? 1 : 0], (unsigned long long)R.ncols * v.nz);
  }
}

// alpha = eta1 / (d, q) of the standard PCG (pcg:426-463).
template <bool Shared>
__device__ __forceinline__ void std_mv_fin(const DevView& v, InstState& S, const double* s) {
  const double alpha = S.rz / s[0];
  if (is_nan(alpha)) { fail<Shared>(v, S, BP_ERR_NAN); return; }
  S.alpha = alpha;
}

// beta and eta1 of the standard PCG's next iteration from (r,z), (r,r)
// (pcg:347-407).
template <bool Shared>
__device__ __forceinline__ void std_update_fin(const DevView& v, const InstParams& ip, InstState& S,
                                               const double* s) {
  if (S.pcg_iter >= ip.pcg_maxiters) { pcg_stop<Shared>(v, S, false); return; }
  if (is_nan(s[0])) { fail<Shared>(v, S, BP_ERR_NAN); return; }
  S.beta = s[0] / S.rz;
  S.rz = s[0];
  if (v.A32) refine_request(ip, S, s[1]);
  S.pcg_iter += 1;
}

// The Chronopoulos-Gear scalar recurrences from (r,z), (Az,z), (r,r)
// (pcg:1461-1512); FIRST: the first pass (pcg:1304-1405).
template <bool FIRST, bool Shared>
__device__ __forceinline__ void cg_mv_fin(const DevView& v, const InstParams& ip, InstState& S, const double* s) {
  if (FIRST) {
    S.rz_old = s[0];
    S.sigma = s[1];
    const double alpha = s[0] / s[1];
    if (is_nan(alpha)) { fail<Shared>(v, S, BP_ERR_NAN); return; }
    S.alpha = alpha;
    return;
  }
  S.pcg_iter += 1;
  if (S.pcg_iter > ip.pcg_maxiters) {
    S.pcg_iter = ip.pcg_maxiters;
    pcg_stop<Shared>(v, S, false);
    return;
  }
  const double rho = s[0], delta = s[1];
  double beta, sigma;
  if (S.restart) {  // after a refinement: d = z, q = A z (the first pass)
    beta = 0.0;
    sigma = delta;
    S.restart = 0;
  } else {
    beta = rho / S.rz_old;
    sigma = delta - beta * rho / S.alpha;
  }
  const double alpha = rho / sigma;
  S.rz_old = rho;
  S.beta = beta;
  S.sigma = sigma;
  if (is_nan(alpha)) { fail<Shared>(v, S, BP_ERR_NAN); return; }
  S.alpha = alpha;
  if (v.A32) refine_request(ip, S, s[2]);
}

// Standard PCG: q = A d; (d, q); alpha = eta1 / (d, q)   (pcg:426-463).
// In the autotuner's dry pass (v.dry) the Krylov matvecs run on every tile
// and skip the scalar tail, so timing them changes no instance state.
template <int STORE, int MINB>
__global__ void __launch_bounds__(kTile, MINB) k_std_mv(DevView v) {
  pdl_wait();
  pdl_launch_next();
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const InstState& S0 = v.st[R.inst];
    if (!S0.pcg_active && !v.dry) continue;
    count_tile<STORE>(v, S0, R);
    const int n = R.n0 + threadIdx.x;
    double part[1] = {0.0};
    if (tile_mine(v, R, threadIdx.x)) {
      const int col = tile_col(v, R, threadIdx.x), k = tile_k(v, threadIdx.x);
      const double2 y = krylov_row<STORE>(v, S0, col, k, n, v.d0);
      const double2 d = v.d0[n];
      v.q[n] = y;
      part[0] = d.x * y.x + d.y * y.y;
    }
    tile_finish<1, false>(v, t, R.inst, part, [&](int inst, const double* s) {
      if (!v.dry) std_mv_fin<true>(v, v.st[inst], s);
    });
  }
}

// x += alpha d; r -= alpha q; z = D^-1 r; (r, z) -> beta  (pcg:347-407, 468-472).
// On check iterations only x is updated (r is recomputed from b - A x).
template <bool CHECK>
__global__ void __launch_bounds__(kTile) k_std_update(DevView v) {
  pdl_wait();
  pdl_launch_next();
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const InstState& S = v.st[R.inst];
    if (!S.pcg_active) continue;
    const int n = R.n0 + threadIdx.x;
    const double alpha = S.alpha;
    const bool mine = tile_mine(v, R, threadIdx.x);
    double part[2] = {0.0, 0.0};
    double2 r = make_double2(0.0, 0.0);
    if (mine) {
      const double2 d = v.d0[n];
      double2 x = v.x[n];
      x.x = x.x + alpha * d.x;
      x.y = x.y + alpha * d.y;
      v.x[n] = x;
      if (!CHECK) {
        const double2 q = v.q[n];
        r = v.r[n];
        r.x = r.x - alpha * q.x;
        r.y = r.y - alpha * q.y;
        v.r[n] = r;
      }
    }
    if (!CHECK) {
      const double2 z = precondition(v, R, mine, n, r);
      if (mine) {
        v.z[n] = z;
        part[0] = r.x * z.x + r.y * z.y;
        part[1] = r.x * r.x + r.y * r.y;
      }
    }
    if (!CHECK) {
      tile_finish<2, false, 4>(v, t, R.inst, part, [&](int inst, const double* s) {
        std_update_fin<true>(v, v.inst[inst], v.st[inst], s);
      });
    }
  }
}

// d = z + beta d; d = z at the first iteration (pcg:403-407).
__global__ void __launch_bounds__(kTile) k_std_dir(DevView v) {
  pdl_wait();
  pdl_launch_next();
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const InstState& S = v.st[R.inst];
    if (!S.pcg_active) continue;
    const int n = R.n0 + threadIdx.x;
    if (!tile_mine(v, R, threadIdx.x)) continue;
    const double2 z = v.z[n];
    if (S.pcg_iter == 1) {
      v.d0[n] = z;
    } else {
      const double beta = S.beta;
      const double2 d = v.d0[n];
      v.d0[n] = make_double2(z.x + beta * d.x, z.y + beta * d.y);
    }
  }
}

// Chronopoulos-Gear matvec Az = A z with (r,z), (Az,z) and the scalar
// recurrences (pcg:1461-1512).  FIRST: the first pass (pcg:1304-1405),
// which also sets d = z, q = A d.
template <bool FIRST, int STORE, int MINB>
__global__ void __launch_bounds__(kTile, MINB) k_cg_mv(DevView v) {
  pdl_wait();
  pdl_launch_next();
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const InstState& S0 = v.st[R.inst];
    if (!S0.pcg_active && !v.dry) continue;
    count_tile<STORE>(v, S0, R);
    const int n = R.n0 + threadIdx.x;
    double part[3] = {0.0, 0.0, 0.0};
    if (tile_mine(v, R, threadIdx.x)) {
      const int col = tile_col(v, R, threadIdx.x), k = tile_k(v, threadIdx.x);
      const double2 y = krylov_row<STORE>(v, S0, col, k, n, v.z);
      const double2 z = v.z[n], r = v.r[n];
      if (FIRST) {
        v.d0[n] = z;
        v.q[n] = y;
      } else {
        v.Az[n] = y;
      }
      part[0] = r.x * z.x + r.y * z.y;
      part[1] = y.x * z.x + y.y * z.y;
      part[2] = r.x * r.x + r.y * r.y;
    }
    tile_finish<3, false>(v, t, R.inst, part, [&](int inst, const double* s) {
      if (!v.dry) cg_mv_fin<FIRST, true>(v, v.inst[inst], v.st[inst], s);
    });
  }
}

// Chronopoulos-Gear first-pass update: x += alpha d; r -= alpha q; z = D^-1 r.
__global__ void __launch_bounds__(kTile) k_cg_first_update(DevView v) {
  pdl_wait();
  pdl_launch_next();
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const InstState& S = v.st[R.inst];
    if (!S.pcg_active) continue;
    const int n = R.n0 + threadIdx.x;
    const bool mine = tile_mine(v, R, threadIdx.x);
    const double alpha = S.alpha;
    double2 r = make_double2(0.0, 0.0);
    if (mine) {
      const double2 d = v.d0[n], q = v.q[n];
      double2 x = v.x[n];
      r = v.r[n];
      x.x = x.x + alpha * d.x; x.y = x.y + alpha * d.y;
      r.x = r.x - alpha * q.x; r.y = r.y - alpha * q.y;
      v.x[n] = x;
      v.r[n] = r;
    }
    const double2 z = precondition(v, R, mine, n, r);
    if (mine) v.z[n] = z;
  }
}

// Chronopoulos-Gear loop update (pcg:1519-1534): d = z + beta d;
// q = Az + beta q; x += alpha d; r -= alpha q; z = D^-1 r for the next
// iteration (skipped on check iterations, where r and z come from b - A x).
template <bool CHECK>
__global__ void __launch_bounds__(kTile) k_cg_update(DevView v) {
  pdl_wait();
  pdl_launch_next();
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const InstState& S = v.st[R.inst];
    if (!S.pcg_active) continue;
    const int n = R.n0 + threadIdx.x;
    const bool mine = tile_mine(v, R, threadIdx.x);
    const bool keep_r = !CHECK && !S.need_true;  // a refinement recomputes r and z
    const double alpha = S.alpha, beta = S.beta;
    double2 r = make_double2(0.0, 0.0);
    if (mine) {
      const double2 z = v.z[n], az = v.Az[n];
      double2 d = v.d0[n], q = v.q[n], x = v.x[n];
      d.x = z.x + beta * d.x; d.y = z.y + beta * d.y;
      q.x = az.x + beta * q.x; q.y = az.y + beta * q.y;
      x.x = x.x + alpha * d.x; x.y = x.y + alpha * d.y;
      v.d0[n] = d;
      v.q[n] = q;
      v.x[n] = x;
      if (keep_r) {
        r = v.r[n];
        r.x = r.x - alpha * q.x;
        r.y = r.y - alpha * q.y;
        v.r[n] = r;
      }
    }
    if (keep_r) {
      const double2 z = precondition(v, R, mine, n, r);
      if (mine) v.z[n] = z;
    }
  }
}

// ---------------------------------------------------------------------
// Resident PCG: the whole linear solve of a problem whose tiles all fit on
// the GPU at once, in one cooperative launch of one CTA per tile.
//
// At these sizes (a few hundred tiles and fewer) a launched PCG step does
// microseconds of work between launches that cost as much again, so the
// solve is bound by launches and by the drain and refill at each of them.
// Here a CTA keeps its tile for the whole solve: x, r, d, q in registers,
// the matrix rows, the SIA factors and the source vector of the tile and of
// its halo columns in shared memory.  Two things pass between CTAs, both as
// 16-byte (value, epoch) slots, each written by one relaxed 128-bit store
// and read by polling 128-bit loads, so that a value and the news of its
// arrival are one trip through L2 with no fence and no atomic:
//  * the global sums: every tile publishes its block sums, every CTA reads
//    those of its instance, adds them in the order of tile_finish and runs
//    the scalar recurrences on its own copy of the state;
//  * the halo: every tile publishes its nodes of the new z, and for a
//    residual of x; the standard PCG's halo direction z + beta d is formed
//    by each reader as its owner forms it.
// Instances of a batch never wait for one another.  All arithmetic is the
// launched kernels', in their order, so the results are the same bitwise.
//
// Slots are rewritten only after every reader is past them.  Sums are
// double-buffered by the epoch's parity: a tile publishes sum e + 2 after it
// has every tile's e + 1, each published after its CTA has read all of sum
// e.  Nodes: a tile publishes the next z (or x) after a sum that every CTA
// contributed to after its product with the last one.  Every wait is bounded:
// past the limit the CTA leaves, and the instance ends with BP_ERR_BUDGET.
//
// What bounds it: the trips through L2.  One slot takes about 500 cycles to
// another SM of the same die and 900 to the other die, an iteration makes
// two trips in a row (z and the halo's arrive with the second sum, or follow
// the one sum of Chronopoulos-Gear), and each is followed by two shuffle
// trees; the product from shared memory (864 B a node) is 1,900 of the 11,000
// cycles of an iteration of the 34-tile dome.
// Measured, launched kernels -> this one, diagonal preconditioner: 31 x 31 x
// 10 dome, FP64, standard PCG, 34 tiles: 21 -> 5.6 us an iteration (7.8 with
// the column preconditioner); 128 x 128 2-D marine sheet, Chronopoulos-Gear,
// 39 tiles: 18 -> 5.1 us; 48 x 48 x 11 slab, 144 tiles: 23 -> 6.3 us.
// The limit (every tile resident: 148 tiles of FP64 rows, 296 of FP32 ones) is
// where shared memory ends.
// ---------------------------------------------------------------------
constexpr int kXchSpins = 1 << 22;  // a second or more of polling

__device__ __forceinline__ void xch_put(ulonglong2* p, double val, unsigned long long tag) {
  asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(val)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ void xch_ld(const ulonglong2* p, double* val, unsigned long long* tag) {
  unsigned long long lo;
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(lo), "=l"(*tag)
               : "l"(p)
               : "memory");
  *val = __longlong_as_double((long long)lo);
}
// NS slots from p on with epoch e into w, loaded together; false past the limit.
template <int NS>
__device__ __forceinline__ bool xch_poll(const ulonglong2* p, unsigned long long e, double* w) {
  for (int spin = 0; spin < kXchSpins; ++spin) {
    unsigned long long tag[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) xch_ld(p + i, &w[i], &tag[i]);
    bool there = true;
#pragma unroll
    for (int i = 0; i < NS; ++i) there = there && tag[i] == e;
    if (there) return true;
  }
  return false;
}

// a.x b.x + a.y b.y in one fixed fused form, the one the compiler gives the
// launched kernels' sums (left to it, a product that appears twice in this
// kernel would be formed once and rounded).
__device__ __forceinline__ double dot2(double2 a, double2 b) {
  return __fma_rn(a.x, b.x, __dmul_rn(a.y, b.y));
}

__device__ __forceinline__ int xch_copies(const DevView& v) { return v.ntiles > 64 ? kXchSumCopies : 1; }

// The sum of NV values of every thread of the instance's CTAs, in
// tile_finish's order, in two steps so that other waiting can go between
// them.  xch_put_sum publishes the tile's block sums; a tile has at most
// eight warps, so the second stage of block_reduce's tree over 32 lanes is
// its three last steps.  Past 64 tiles each sum goes to kXchSumCopies copies,
// each read by every kXchSumCopies-th CTA only: all CTAs polling one line queue
// up at its L2 slice (an all-to-all round of bare slots takes 1,430 cycles
// among 34 CTAs and 1,890 with eight copies, but 3,030 and 2,460 among 144).
// xch_get_sum waits for all tiles' sums and returns
// their total in val on every thread.  red: two arrays of 8 x 4 doubles.
template <int NV>
__device__ __forceinline__ void xch_put_sum(const DevView& v, int t, unsigned long long e, const double* val,
                                            double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double x = val[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp * 4 + i] = x;
  }
  __syncthreads();
  if (warp == 0) {  // the lanes w * 4 + i sum value i over the warps w
    const int w = lane >> 2, i = lane & 3;
    double x = (w < nw && i < NV) ? red[w * 4 + i] : 0.0;
    x += __shfl_xor_sync(0xffffffffu, x, 16);
    x += __shfl_xor_sync(0xffffffffu, x, 8);
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    x = __shfl_sync(0xffffffffu, x, lane % NV);
    const int copy = lane / NV;
    if (copy < xch_copies(v))
      xch_put(v.xch + ((size_t)((e & 1) * kXchSumCopies + copy) * v.ntiles + t) * 4 + lane % NV, x, e);
  }
}
template <int NV>
__device__ __forceinline__ bool xch_get_sum(const DevView& v, const InstParams& ip, int t, unsigned long long e,
                                            double* val, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const ulonglong2* slots =
      v.xch + ((size_t)((e & 1) * kXchSumCopies + t % xch_copies(v)) * v.ntiles + ip.tile_begin) * 4;
  double s[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) s[i] = 0.0;
  bool ok = true;
  const int ntl = ip.tile_end - ip.tile_begin;
  for (int tt = threadIdx.x; tt < ntl && ok; tt += blockDim.x) {
    double w[NV];
    ok = xch_poll<NV>(slots + (size_t)tt * 4, e, w);
#pragma unroll
    for (int i = 0; i < NV; ++i) s[i] += w[i];
  }
  double* red2 = red + 32;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double x = s[i];
    if (warp * 32 < ntl) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    }
    if (lane == 0) red2[warp * 4 + i] = x;
  }
  ok = __syncthreads_and(ok);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = j < nw ? red2[j * 4 + i] : 0.0;
    val[i] = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
  }
  return ok;
}
template <int NV>
__device__ __forceinline__ bool xch_sum(const DevView& v, const InstParams& ip, int t, unsigned long long e,
                                        double* val, double* red) {
  xch_put_sum<NV>(v, t, e, val, red);
  return xch_get_sum<NV>(v, ip, t, e, val, red);
}

// Shared memory of a tile: the matrix rows -- offset m (3 x 9; nz = 1: the 9
// of the level) of node i at [m * slots + i], (uu, uv) and (vu, vv) in FP64,
// or packed FP32 with the FP64 diagonal block after them --; the source
// vector, level k of column slot c at [(k + 1) * ls + c], with a level of
// zeros above and below and a last column of zeros that absent neighbours
// read (twice for the standard PCG: its residuals read x while the
// directions stay); the SIA sweeps' s, a, beta, gamma; and each node's
// nine neighbour columns as slots, [q * slots + i].
struct ResidentShape {
  int slots, offsets, ls;
  size_t matrix, source, sia, bytes;
};
__host__ __device__ inline ResidentShape resident_shape(const DevView& v, bool f32, int variant) {
  ResidentShape h;
  h.slots = v.W * v.nz;
  h.offsets = v.nz == 1 ? 9 : 27;
  h.ls = v.W + v.halo_max + 1;
  h.matrix = (size_t)h.slots * (f32 ? 16 * h.offsets + 32 : 32 * h.offsets);
  h.source = 16 * (size_t)(v.nz + 2) * h.ls;
  h.sia = v.sia_f ? sizeof(double) * 8 * h.slots : 0;
  h.bytes = h.matrix + h.source * (variant == 3 ? 1 : 2) + h.sia + sizeof(uint16_t) * 9 * h.slots;
  return h;
}

// PER_SM: CTAs the kernel is built to run on an SM: 1, or 2 for FP32 tiles of
// at most 192 threads.
template <int STORE, int VARIANT, int PER_SM>
__global__ void __launch_bounds__(PER_SM == 2 ? 192 : kTile, PER_SM) k_pcg_resident(DevView v) {
  extern __shared__ __align__(16) unsigned char rs_sm[];
  __shared__ InstState S;
  __shared__ double red[2 * 32];
  constexpr bool MIXED = STORE == ST_SYM32;
  const int t = blockIdx.x, i = threadIdx.x;
  const TileRange R = tile_range(v, t);
  InstState& G = v.st[R.inst];
  if (!G.pcg_active) return;  // the same for all CTAs of the instance: none writes G before all have begun
  const InstParams& ip = v.inst[R.inst];
  unsigned long long es = v.xch_epoch[R.inst], en = es;  // epochs of the sums and of the nodes
  const ResidentShape H = resident_shape(v, MIXED, VARIANT);
  const int nz = v.nz, W = v.W, slots = H.slots, ls = H.ls;
  const int ncheck = ip.ncheck > 0 ? ip.ncheck : 1;
  const size_t np = (size_t)v.npad;
  const bool mine = tile_mine(v, R, i);
  const size_t n = (size_t)R.n0 + i;
  const int col = mine ? tile_col(v, R, i) : 0, k = mine ? tile_k(v, i) : 0;
  const int lev = (k + 1) * ls, me = lev + (i & (W - 1));  // this node in the source vector
  double2* M0 = reinterpret_cast<double2*>(rs_sm);
  double2* M1 = M0 + (size_t)slots * H.offsets;
  float4* MF = reinterpret_cast<float4*>(rs_sm);
  double2* DG = reinterpret_cast<double2*>(MF + (size_t)slots * H.offsets);
  double2* src = reinterpret_cast<double2*>(rs_sm + H.matrix);
  double2* srcx = VARIANT == 3 ? src : reinterpret_cast<double2*>(rs_sm + H.matrix + H.source);
  double* sia = reinterpret_cast<double*>(rs_sm + H.matrix + H.source * (VARIANT == 3 ? 1 : 2));
  uint16_t* nbr = reinterpret_cast<uint16_t*>(reinterpret_cast<unsigned char*>(sia) + H.sia) + i;
  const int js = 2 * ((i & (W - 1)) * nz + k), so = 2 * slots;
  const bool column_pc = ip.precond == 2;
  const int h0 = v.halo_begin[t], nh = v.halo_begin[t + 1] - h0;
  const double2 zero = make_double2(0.0, 0.0);
  double2 x = zero, r = zero, z = zero, d = zero, q = zero, di = zero;

  if (i == 0) S = G;
  for (int o = i; o < (nz + 2) * ls; o += blockDim.x) {
    src[o] = zero;
    srcx[o] = zero;
  }
  __syncthreads();
  if (mine) {
    for (int c = 0; c < 9; ++c) {
      const int lc = v.col_loc[c * v.ncols + col], cq = v.col_nbn[c * v.ncols + col];
      nbr[c * slots] = (uint16_t)(lc >= 0 ? lc : ls - 1);
      for (int kA = nz == 1 ? 0 : -1; kA <= (nz == 1 ? 0 : 1); ++kA) {
        const int m = (kA + 1) * 9 + c, o = (nz == 1 ? c : m) * slots + i, kn = k + kA;
        const bool there = lc >= 0 && kn >= 0 && kn < nz;
        const size_t p = there ? (size_t)cq + ((size_t)kn << v.lsh) : n;
        if (STORE == ST_SYM32) {
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
          if (there && m > 13) a = v.A32[(size_t)(m - 13) * np + n];
          if (there && m < 13) {
            const float4 b = v.A32[(size_t)(13 - m) * np + p];
            a = make_float4(b.x, b.z, b.y, b.w);
          }
          MF[o] = a;
        } else {
          double2 a0 = zero, a1 = zero;
          if (there && STORE == ST_FULL) {
            a0 = v.A[(size_t)m * np + n];
            a1 = v.A[(size_t)(27 + m) * np + n];
          } else if (there && m >= 13) {
            a0 = v.A[(size_t)(m - 13) * np + n];
            a1 = v.A[(size_t)(m + 1) * np + n];
          } else if (there) {
            const double2 b0 = v.A[(size_t)(13 - m) * np + p], b1 = v.A[(size_t)(27 - m) * np + p];
            a0 = make_double2(b0.x, b1.x);
            a1 = make_double2(b0.y, b1.y);
          }
          M0[o] = a0;
          M1[o] = a1;
        }
      }
    }
    if (STORE == ST_SYM32) {
      DG[i] = v.A32d[n];
      DG[slots + i] = v.A32d[np + n];
    }
    x = v.x[n];
    r = v.r[n];
    z = v.z[n];
    src[me] = z;
    if (column_pc) {
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        const double2 c = v.sia_f[(size_t)f * np + n];
        sia[(f + 1) * so + js] = c.x;
        sia[(f + 1) * so + js + 1] = c.y;
      }
    } else {
      di = v.Dinv[n];
    }
  }
  // halo node h (slot c of level kk): its node, its place in the source vector
  auto halo_at = [&](int h, size_t* node) {
    const int kk = h / nh, c = h - kk * nh;
    *node = (size_t)v.halo_node[h0 + c] + ((size_t)kk << v.lsh);
    return (kk + 1) * ls + W + c;
  };
  for (int h = i; h < nh * nz; h += blockDim.x) {  // MV_INIT's z of the halo
    size_t p;
    const int o = halo_at(h, &p);
    src[o] = v.z[p];
  }
  // a thread's first nodes of the halo, which is two to three times the CTA
  // in the tiles of a filled grid, stay known to it
  constexpr int B = 3;
  const ulonglong2* hp[B];
  int ho[B];
  unsigned hmine = 0;
#pragma unroll
  for (int j = 0; j < B; ++j) {
    const int h = i + j * blockDim.x;
    size_t p = 0;
    ho[j] = h < nh * nz ? halo_at(h, &p) : 0;
    hp[j] = v.xch_node + 2 * p;
    if (h < nh * nz) hmine |= 1u << j;
  }
  __syncthreads();

  // this node's value to the tiles that read it; the halo's new values, each
  // through f(value, source slot), once per halo node
  auto publish = [&](double2 a, unsigned long long e, size_t buf) {
    xch_put(v.xch_node + 2 * n + buf, a.x, e);
    xch_put(v.xch_node + 2 * n + buf + 1, a.y, e);
  };
  constexpr size_t ZBUF = 0;
  const size_t XBUF = 2 * np;
  double2 ha[B];
  auto halo_wait = [&](unsigned long long e, size_t buf) -> bool {  // the thread's first nodes
    unsigned left = hmine;
    for (int spin = 0; spin < kXchSpins && left; ++spin) {  // those still missing, loaded together
      unsigned long long tx[B], ty[B];
#pragma unroll
      for (int j = 0; j < B; ++j)
        if (left >> j & 1) {
          xch_ld(hp[j] + buf, &ha[j].x, &tx[j]);
          xch_ld(hp[j] + buf + 1, &ha[j].y, &ty[j]);
        }
#pragma unroll
      for (int j = 0; j < B; ++j)
        if ((left >> j & 1) && tx[j] == e && ty[j] == e) left &= ~(1u << j);
    }
    return left == 0;
  };
  auto halo_take = [&](unsigned long long e, size_t buf, auto f) -> bool {  // all of them, after halo_wait
    bool ok = true;
#pragma unroll
    for (int j = 0; j < B; ++j)
      if (hmine >> j & 1) f(ha[j], ho[j]);
    for (int h = i + B * blockDim.x; h < nh * nz && ok; h += blockDim.x) {  // the rest of a ragged tile's halo
      size_t p;
      const int o = halo_at(h, &p);
      double w[2];
      ok = xch_poll<2>(v.xch_node + 2 * p + buf, e, w);
      f(make_double2(w[0], w[1]), o);
    }
    return ok;
  };
  auto precondition_r = [&] {  // z = M^-1 r
    if (column_pc) {
      if (mine) {
        sia[js] = r.x;
        sia[js + 1] = r.y;
      }
      __syncthreads();
      if (i < 2 * R.ncols) {
        const int o = 2 * (i >> 1) * nz + (i & 1);
        sia_sweeps(
            nz,
            [&](int kk) { return SiaFac{sia[so + o + 2 * kk], sia[2 * so + o + 2 * kk], sia[3 * so + o + 2 * kk]}; },
            &sia[o], 2);
      }
      __syncthreads();
      if (mine) z = make_double2(sia[js], sia[js + 1]);
    } else if (mine) {
      z = make_double2(r.x * di.x, r.y * di.y);
    }
  };
  // this node's row times the source vector s, from the tile's rows in
  // shared memory, in matvec_row's order (FULL: levels outer) or
  // matvec_row_sym's (neighbour columns outer)
  auto row = [&](const double2* s) -> double2 {
    double yu = 0.0, yv = 0.0;
    if (!mine) return zero;
    auto term = [&](int c, int kA) {
      const int m = ((nz == 1 ? 0 : (kA + 1) * 9) + c) * slots + i;
      const double2 sv = s[lev + kA * ls + nbr[c * slots]];
      if (MIXED && !(kA == 0 && c == 4)) {
        const float4 a = MF[m];
        yu += dot2(make_double2((double)a.x, (double)a.y), sv);
        yv += dot2(make_double2((double)a.z, (double)a.w), sv);
      } else {
        yu += dot2(MIXED ? DG[i] : M0[m], sv);
        yv += dot2(MIXED ? DG[slots + i] : M1[m], sv);
      }
    };
    if (nz == 1) {
#pragma unroll
      for (int c = 0; c < 9; ++c) term(c, 0);
    } else if (STORE == ST_FULL) {
#pragma unroll
      for (int kA = -1; kA <= 1; ++kA)
#pragma unroll
        for (int c = 0; c < 9; ++c) term(c, kA);
    } else {
#pragma unroll
      for (int c = 0; c < 9; ++c)
#pragma unroll
        for (int kA = -1; kA <= 1; ++kA) term(c, kA);
    }
    return make_double2(yu, yv);
  };
  // the same with the FP64 matrix of a mixed solve, from device memory
  auto row64 = [&](const double2* s) -> double2 {
    double yu = 0.0, yv = 0.0;
    if (!mine) return zero;
#pragma unroll 3
    for (int c = 0; c < 9; ++c) {
      const int lc = v.col_loc[c * v.ncols + col], cq = v.col_nbn[c * v.ncols + col];
#pragma unroll
      for (int kA = -1; kA <= 1; ++kA) {
        const int m = (kA + 1) * 9 + c, kn = k + kA;
        const bool there = lc >= 0 && kn >= 0 && kn < nz;
        const size_t p = there ? (size_t)cq + ((size_t)kn << v.lsh) : n;
        const double2 sv = s[lev + kA * ls + (lc >= 0 ? lc : ls - 1)];
        if (m >= 13) {
          yu += dot2(v.A[(size_t)(m - 13) * np + n], sv);
          yv += dot2(v.A[(size_t)(m + 1) * np + n], sv);
        } else {
          const double2 b0 = v.A[(size_t)(13 - m) * np + p], b1 = v.A[(size_t)(27 - m) * np + p];
          yu += dot2(make_double2(b0.x, b1.x), sv);
          yv += dot2(make_double2(b0.y, b1.y), sv);
        }
      }
    }
    return make_double2(yu, yv);
  };
  double val[3];
  bool ok = true;
  // r = b - A x, z and their sums with the scalar update
  auto residual = [&](auto mode) {
    constexpr int MODE = decltype(mode)::value;
    ++en;
    if (mine) {
      publish(x, en, XBUF);
      srcx[me] = x;
    }
    ok = __syncthreads_and(halo_wait(en, XBUF) && halo_take(en, XBUF, [&](double2 a, int o) { srcx[o] = a; }));
    if (!ok) return;
    const double2 y = MIXED ? row64(srcx) : row(srcx);
    if (mine) {
      const double2 b = v.b[n];
      r = make_double2(b.x - y.x, b.y - y.y);
    }
    precondition_r();
    ++en;
    if (mine) publish(z, en, ZBUF);
    val[0] = mine ? dot2(r, z) : 0.0;
    val[1] = mine ? dot2(r, r) : 0.0;
    xch_put_sum<2>(v, t, ++es, val, red);
    const bool zs = halo_wait(en, ZBUF);  // z arrives with the sums
    ok = xch_get_sum<2>(v, ip, t, es, val, red);
    ok = __syncthreads_and(ok && zs);
    if (i == 0 && ok) resid_fin<MODE, false>(v, ip, S, val);
    __syncthreads();
  };
  using Check = std::integral_constant<int, MV_CHECK>;
  using Refine = std::integral_constant<int, MV_REFINE>;

  if (VARIANT == 2) {
    for (int it = 1; ok; ++it) {
      const bool check = it % ncheck == 0;
      // d = z + beta d (k_std_dir) here and in the halo
      const double beta = S.beta;
      if (it > 1) {
        if (mine) {
          d = make_double2(z.x + beta * d.x, z.y + beta * d.y);
          src[me] = d;
        }
        ok = __syncthreads_and(halo_take(en, ZBUF, [&](double2 a, int o) {
          const double2 b = src[o];
          src[o] = make_double2(a.x + beta * b.x, a.y + beta * b.y);
        }));
        if (!ok) break;
      } else {
        d = z;
      }
      const double2 y = MIXED && S.krylov_fp64 ? row64(src) : row(src);
      val[0] = mine ? dot2(d, y) : 0.0;
      ok = xch_sum<1>(v, ip, t, ++es, val, red);
      if (i == 0 && ok) std_mv_fin<false>(v, S, val);
      __syncthreads();
      if (!ok || !S.pcg_active) break;
      const double alpha = S.alpha;
      if (mine) {
        x.x = x.x + alpha * d.x;
        x.y = x.y + alpha * d.y;
      }
      if (check && !MIXED) {
        residual(Check{});
      } else {
        if (mine) {
          r.x = r.x - alpha * y.x;
          r.y = r.y - alpha * y.y;
        }
        precondition_r();
        ++en;
        if (mine) publish(z, en, ZBUF);
        val[0] = mine ? dot2(r, z) : 0.0;
        val[1] = mine ? dot2(r, r) : 0.0;
        xch_put_sum<2>(v, t, ++es, val, red);
        const bool zs = halo_wait(en, ZBUF);  // the next z arrives with the sums
        ok = xch_get_sum<2>(v, ip, t, es, val, red);
        ok = __syncthreads_and(ok && zs);
        if (i == 0 && ok) std_update_fin<false>(v, ip, S, val);
        __syncthreads();
        if (ok && MIXED && check && S.pcg_active && S.need_true) residual(Refine{});
      }
      if (!S.pcg_active) break;
    }
  } else {
    bool z_waited = false;
    for (int it = 1; ok; ++it) {
      const bool check = it > 1 && it % ncheck == 0;
      const bool waited = z_waited;  // a residual has fetched the halo of its z
      if (it > 1) {
        if (mine) src[me] = z;
        ok = __syncthreads_and((waited || halo_wait(en, ZBUF)) &&
                               halo_take(en, ZBUF, [&](double2 a, int o) { src[o] = a; }));
        if (!ok) break;
      }
      const double2 y = MIXED && S.krylov_fp64 ? row64(src) : row(src);
      val[0] = mine ? dot2(r, z) : 0.0;
      val[1] = mine ? dot2(y, z) : 0.0;
      val[2] = mine ? dot2(r, r) : 0.0;
      ok = xch_sum<3>(v, ip, t, ++es, val, red);
      if (i == 0 && ok) {
        if (it == 1) cg_mv_fin<true, false>(v, ip, S, val);
        else cg_mv_fin<false, false>(v, ip, S, val);
      }
      __syncthreads();
      if (!ok || !S.pcg_active) break;
      const double alpha = S.alpha, beta = S.beta;
      const bool keep_r = it == 1 || (!(check && !MIXED) && !S.need_true);
      if (mine) {
        if (it == 1) {
          d = z;
          q = y;
        } else {
          d.x = z.x + beta * d.x; d.y = z.y + beta * d.y;
          q.x = y.x + beta * q.x; q.y = y.y + beta * q.y;
        }
        x.x = x.x + alpha * d.x; x.y = x.y + alpha * d.y;
        if (keep_r) {
          r.x = r.x - alpha * q.x;
          r.y = r.y - alpha * q.y;
        }
      }
      z_waited = !keep_r;
      if (keep_r) {
        precondition_r();
        ++en;
        if (mine) publish(z, en, ZBUF);
      } else if (MIXED) {
        residual(Refine{});
      } else {
        residual(Check{});
      }
      if (!S.pcg_active) break;
    }
  }
  if (mine) v.x[n] = x;
  if (t == ip.tile_begin && i == 0) {
    if (!ok) fail<false>(v, S, BP_ERR_BUDGET);  // a wait ran out
    if (!S.pcg_active) atomicSub(&v.cnt->pcg_active, 1);
    if (G.refine_active && !S.refine_active) atomicSub(&v.cnt->refine_active, 1);
    if (G.picard_active && !S.picard_active) atomicSub(&v.cnt->picard_active, 1);
    G = S;
    v.xch_epoch[R.inst] = (es > en ? es : en) + (ok ? 0 : 4);  // after a failed wait other CTAs may be ahead
  }
}

// ---------------------------------------------------------------------
// Staged Krylov matvec: k_cg_mv and k_std_mv on half storage, for problems
// too large for the resident PCG.
//
// The per-node kernels run at 0.4 of the copy bandwidth with no unit
// saturated: a thread's 55 16-byte loads, two thirds of them gathers, go
// through L1 with the few registers that eight CTAs an SM leave, and each
// tile ends in a fence and a ticket that its warps wait for.  Here a CTA
// walks its tiles as a pipeline.  A producer warp brings each tile's own
// matrix rows (one bulk copy per offset: the DRAM stream) and its source
// vector with the halo columns' (16-byte asynchronous copies, each value
// once instead of up to 27 times) into one of two shared-memory stages
// while the other is computed, so the stream never waits for arithmetic;
// the consumer warps, one thread per node, hold the 13 transposed entries
// of the neighbours' rows in registers and load the next tile's into the
// same registers as they use this one's.  Sums: each warp stores its
// tile's, and the CTA adds them, in block_reduce's order, and takes its
// tickets once, after its last tile.  What follows the last ticket is a chain
// that no other work hides, so it is kept short: one ticket per warp and
// instance, an instance's partials fetched to shared memory in one flight
// instead of a few a thread, the next instance's meanwhile, and the scalar
// updates of all instances side by side (a tail of 41 -> 13 us with four
// instances of 2,460 tiles, 20 -> 10 with one of 5,980, 45 -> 15 with 16 of
// 220).  The arithmetic and its order are the per-node kernels' (bitwise the
// same results).
//
// Barriers, all waits bounded (past the limit a warp leaves as one, the producer
// once its copies have landed or after another limit, and the CTA marks the
// instances' sums as NaN, which ends their solve with BP_ERR_NAN): full[stage]
// -- the stage's copies have landed (32 producer lanes and the bulk bytes);
// empty[stage] -- every consumer warp is done with it; dfull[slot] -- a
// descriptor (ring of four, two tiles ahead of the copies) has landed.
//
// What bounds it: the consumers, six warps a tile (one CTA an SM in FP64,
// whose two stages are 177 KB; two in FP32), wait on shared memory and on
// their own chains; DRAM is at 0.65 of the copy bandwidth in FP64 and L2
// hands the SMs 8 of the 10 TB/s that it can (the matrix twice, as own rows
// and as the neighbours').
// Measured, the fastest per-node shape -> this kernel, a launch of
// k_cg_mv's work: 400 x 400 x 11 marine sheet, FP64 (1.05 M nodes) 156 ->
// 115 us; 160 x 160 x 11 slab, FP64, standard PCG 46.5 -> 36.5 us; four
// 256 x 256 x 11 sheets, FP32 (1.73 M nodes) 172 -> 145 us; 16 uneven domains,
// FP32 (0.62 M nodes) 65 -> 68 us.  The autotuner times both on the problem.
// ---------------------------------------------------------------------
constexpr int kStages = 2, kDescs = 4;


template <int STORE>
__host__ __device__ constexpr int staged_own() { return STORE == ST_SYM32 ? 15 : 28; }  // 16-byte rows per node
struct StagedShape {
  int slots, ls, desc;
  size_t own, stage, bytes;
};
__host__ __device__ inline StagedShape staged_shape(const DevView& v, bool f32) {
  StagedShape h;
  h.slots = v.W * v.nz;
  h.ls = StagedDesc::zero_slot(v.W) + 1;
  h.desc = StagedDesc::bytes(v.W);
  h.own = (size_t)16 * h.slots * (f32 ? staged_own<ST_SYM32>() : staged_own<ST_SYM>());
  h.stage = h.own + (size_t)16 * (v.nz + 2) * h.ls;
  h.bytes = kStages * h.stage + (size_t)kDescs * h.desc + 8 * (2 * kStages + kDescs);
  return h;
}

__device__ __forceinline__ unsigned smem_at(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity) {
  for (int i = 0; i < (1 << 22); ++i) {
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
__device__ __forceinline__ void bar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %0;" ::"r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// One CTA per tile: the tile's halo columns, in order of first appearance
// over (neighbour, column), and its descriptor.
__global__ void __launch_bounds__(256) k_staged_desc(const __grid_constant__ DevView v, unsigned char* desc) {
  extern __shared__ int sd[];  // [9 W] neighbour (-1: none or own), then its halo index
  __shared__ int nh;
  const int t = blockIdx.x, W = v.W, E = 9 * W, cap = StagedDesc::halo_cap(W);
  const int c0 = v.tile_col0[t], ncols = v.tile_ncols[t];
  unsigned char* d = desc + (size_t)t * StagedDesc::bytes(W);
  int* node = reinterpret_cast<int*>(d + StagedDesc::nodes_at(W));
  if (threadIdx.x == 0) nh = 0;
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const int q = e / W, c = e - q * W;
    int nb = c < ncols ? v.col_nbr[(size_t)q * v.ncols + c0 + c] : -1;
    if (nb >= c0 && nb < c0 + ncols) nb = -1;
    sd[e] = nb;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {  // first[e]: where this column appears first
    int first = e;
    if (sd[e] >= 0)
      for (int f = 0; f < e; ++f)
        if (sd[f] == sd[e]) { first = f; break; }
    sd[E + e] = sd[e] >= 0 && first == e ? 1 : 0;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const int q = e / W, c = e - q * W;
    int slot = StagedDesc::zero_slot(W);
    const int nb = c < ncols ? v.col_nbr[(size_t)q * v.ncols + c0 + c] : -1;
    if (nb >= c0 && nb < c0 + ncols) {
      slot = nb - c0;
    } else if (nb >= 0) {
      int first = 0, h = 0;
      while (sd[first] != nb) h += sd[E + first++];
      slot = h < cap ? W + h : slot;
      if (first == e) {
        atomicAdd(&nh, 1);
        if (h < cap) node[W + h] = v.col_node[nb];
      }
    }
    d[16 + 64 * c + q] = (unsigned char)slot;
    reinterpret_cast<int*>(d + 32 + 64 * c)[q] = nb >= 0 ? v.col_node[nb] : v.tile_start[t] + c;
  }
  for (int c = threadIdx.x; c < W; c += blockDim.x) node[c] = v.tile_start[t] + c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int* m = reinterpret_cast<int*>(d);
    m[0] = t;
    m[1] = ncols;
    m[2] = nh <= cap ? nh : -1;
    m[3] = v.tile_inst[t];
  }
}

// The product of one row by the per-node bodies, out of line, for tiles of
// an instance whose FP32 refinement stalled and tiles without a descriptor.
template <int STORE>
__device__ __noinline__ double2 plain_row_call(const DevView& v, bool fp64, int col, int k, size_t n,
                                               const double2* s) {
  const SrcX src{s};
  if (STORE == ST_SYM32 && !fp64) return matvec_row_sym32(v, v.A32, col, k, n, src);
  return matvec_row_sym(v, v.A, col, k, n, src);
}

// LS: slots per level of the source vector, compile-time for the usual 16
// columns (0: from W).  THREADS: the most a CTA has (a tile's and the producer's 32); registers are
// granted in groups of four warps, so 7 warps leave far more than 9.
template <int STORE, int MODE, int THREADS, int LS>
__global__ void __launch_bounds__(THREADS, STORE == ST_SYM32 ? 2 : 1)
    k_mv_staged(const __grid_constant__ DevView v) {
  constexpr bool F32 = STORE == ST_SYM32;
  constexpr int NV = MODE == MV_STD_A ? 1 : 3, NOWN = staged_own<STORE>();
  extern __shared__ __align__(128) unsigned char st_sm[];
  const StagedShape H = staged_shape(v, F32);
  const int slots = H.slots, ls = LS > 0 ? LS : H.ls, nz = v.nz, W = LS > 0 ? 16 : v.W, G = gridDim.x;
  const int i = threadIdx.x, lane = i & 31, warp = i >> 5, nw = (blockDim.x >> 5) - 1;
  const double2* s = MODE == MV_STD_A ? v.d0 : v.z;
  unsigned char* descs = st_sm + kStages * H.stage;
  uint64_t* bars = reinterpret_cast<uint64_t*>(descs + kDescs * H.desc);
  auto full = [&](int b) { return smem_at(bars + b); };
  auto empty = [&](int b) { return smem_at(bars + kStages + b); };
  auto dfull = [&](int b) { return smem_at(bars + 2 * kStages + b); };
  auto stage_own = [&](int b) { return st_sm + b * H.stage; };
  auto stage_src = [&](int b) { return reinterpret_cast<double2*>(st_sm + b * H.stage + H.own); };
  if (i == 0) {
    for (int b = 0; b < kStages; ++b) {
      bar_init(full(b), 33);
      bar_init(empty(b), nw);
    }
    for (int b = 0; b < kDescs; ++b) bar_init(dfull(b), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the zeros that absent neighbours read: the last slot of every level, and
  // a level above and below
  for (int e = i; e < kStages * (nz + 2) * ls; e += blockDim.x) {
    const int b = e / ((nz + 2) * ls), o = e - b * (nz + 2) * ls, lev = o / ls;
    if (lev == 0 || lev == nz + 1 || o - lev * ls == ls - 1) stage_src(b)[o] = make_double2(0.0, 0.0);
  }
  __syncthreads();
  pdl_wait();
  pdl_launch_next();
  bool ok = true;

  if (warp == nw) {  // producer
    // the CTA's tiles: every G-th, of the instances that are solving, looked up
    // 32 at a time (a tile at a time, a batch with few instances left passed
    // the others' tiles at two trips to L2 each)
    unsigned live = 0;  // of the 32 from tile t32 on, those still to come
    long t32 = (long)blockIdx.x - 32L * G;
    auto next_tile = [&]() {
      while (live == 0) {
        t32 += 32L * G;
        if (t32 >= v.ntiles) return -1;
        const long t = t32 + (long)lane * G;
        live = __ballot_sync(0xffffffffu, t < v.ntiles && (v.dry || v.st[v.tile_inst[t]].pcg_active));
      }
      const int q = __ffs(live) - 1;
      live &= live - 1;
      return (int)(t32 + (long)q * G);
    };
    int tn = next_tile();  // the next tile whose descriptor is fetched
    auto fetch = [&](int j) {        // descriptor j of the sequence (after the last: tile -1)
      unsigned char* d = descs + (j % kDescs) * H.desc;
      if (lane == 0) {
        if (tn >= 0) {
          bar_expect(dfull(j % kDescs), H.desc);
          bulk_load(smem_at(d), v.desc + (size_t)tn * H.desc, H.desc, dfull(j % kDescs));
        } else {
          *reinterpret_cast<int*>(d) = -1;
          bar_arrive(dfull(j % kDescs));
        }
      }
      if (tn >= 0) tn = next_tile();
    };
    fetch(0);
    fetch(1);
    int j = 0;
    for (; ok; ++j) {
      const int b = j % kStages;
      if (j >= kStages) ok = bar_wait(empty(b), ((j / kStages) - 1) & 1);
      ok = ok && bar_wait(dfull(j % kDescs), (j / kDescs) & 1);
      const unsigned char* d = descs + (j % kDescs) * H.desc;
      // tile, columns, halo columns, instance
      const int4 m = ok ? *reinterpret_cast<const int4*>(d) : make_int4(-1, 0, 0, 0);
      const int nc = m.z < 0 ? 0 : W + m.z;
      if (lane == 0 && m.x >= 0) bar_expect(full(b), nc ? 16u * slots * NOWN : 0u);
      ok = __all_sync(0xffffffffu, ok);  // the lanes leave together
      if (!ok || m.x < 0) break;
      if (nc) {
        const size_t n0 = (size_t)m.x * slots, np = (size_t)v.npad;
        if (lane < NOWN) {
          const void* g = F32 ? (lane < 13 ? static_cast<const void*>(v.A32 + (size_t)(lane + 1) * np + n0)
                                           : static_cast<const void*>(v.A32d + (size_t)(lane - 13) * np + n0))
                              : static_cast<const void*>(v.A + (size_t)lane * np + n0);
          bulk_load(smem_at(stage_own(b)) + 16u * slots * lane, g, 16u * slots, full(b));
        }
        const int* node = reinterpret_cast<const int*>(d + StagedDesc::nodes_at(W));
        const unsigned dst = smem_at(stage_src(b) + ls);
        for (int c = lane; c < nc; c += 32) {
          const double2* g = s + node[c];
          unsigned a = dst + 16u * c;
          for (int k = 0; k < nz; ++k, a += 16u * ls, g += W)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(g) : "memory");
        }
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full(b)) : "memory");
      fetch(j + 2);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!ok) {  // the bulk copies of j tiles and j + 2 descriptors still land in this CTA's memory
      for (int q = max(j - kStages, 0); q < j; ++q) bar_wait(full(q % kStages), (q / kStages) & 1);
      for (int q = max(j + 2 - kDescs, 0); q < j + 2; ++q) bar_wait(dfull(q % kDescs), (q / kDescs) & 1);
    }
  } else {  // consumers: thread i is node i of every tile
    const bool inside = i < slots;
    const int k = inside ? i >> v.lsh : 0, c = i & (W - 1);
    constexpr int NT = F32 ? 13 : 26;
    typedef typename std::conditional<F32, float4, double2>::type Entry;
    Entry T[NT];  // entries of the neighbours' rows toward this node, offset m at [m] (FP64: [2 m], [2 m + 1])
    const Entry* mat = F32 ? reinterpret_cast<const Entry*>(v.A32) : reinterpret_cast<const Entry*>(v.A);
    const unsigned np = (unsigned)v.npad;
    const int klev = k * W, kup = max(k - 1, 0) * W;
    // nb: the neighbour columns' nodes; loads entry m of their tile into T
    // (an absent neighbour's stand-in, this column's own node, meets a zero)
    struct Nodes { int4 a, b; int c; };
    auto load_t = [&](int m, const Nodes& nb) {
      const int q = m % 9, kA = m / 9 - 1;
      const int n0 = q == 0 ? nb.a.x : q == 1 ? nb.a.y : q == 2 ? nb.a.z : q == 3 ? nb.a.w : q == 4 ? nb.b.x
                   : q == 5 ? nb.b.y : q == 6 ? nb.b.z : q == 7 ? nb.b.w : nb.c;
      const unsigned p = (unsigned)(n0 + (kA < 0 ? kup : klev));
      if (F32) {
        T[m] = __ldg(mat + (size_t)(13 - m) * np + p);
      } else {
        T[2 * m] = __ldg(mat + (size_t)(13 - m) * np + p);
        T[2 * m + 1] = __ldg(mat + (size_t)(27 - m) * np + p);
      }
    };
    auto slot_of = [](const uint4& r, int q) {
      const unsigned w = q < 4 ? r.x : (q < 8 ? r.y : r.z);
      return (int)((w >> (8 * (q & 3))) & 255u);
    };
    auto desc_meta = [&](int j) { return *reinterpret_cast<const int4*>(descs + (j % kDescs) * H.desc); };
    auto desc_rec = [&](int j) { return *reinterpret_cast<const uint4*>(descs + (j % kDescs) * H.desc + 16 + 64 * c); };
    auto desc_nodes = [&](int j) {
      const int4* p = reinterpret_cast<const int4*>(descs + (j % kDescs) * H.desc + 32 + 64 * c);
      return Nodes{p[0], p[1], p[2].x};
    };
    ok = __all_sync(0xffffffffu, bar_wait(dfull(0), 0));
    int4 m = ok ? desc_meta(0) : make_int4(-1, 0, 0, 0);
    uint4 rec = make_uint4(0, 0, 0, 0);
    Nodes nb = {make_int4(0, 0, 0, 0), make_int4(0, 0, 0, 0), 0};
    if (m.x >= 0) {
      rec = desc_rec(0);
      nb = desc_nodes(0);
#pragma unroll
      for (int e = 0; e < 13; ++e) load_t(e, nb);
    }
    for (int j = 0; ok && m.x >= 0; ++j) {
      const int b = j % kStages;
      const bool mine = inside && c < m.y;
      const size_t n = (size_t)m.x * slots + i;
      const InstState& S0 = v.st[m.w];
      const bool fp64 = F32 && S0.krylov_fp64;
      double2 r = make_double2(0.0, 0.0);
      if (MODE != MV_STD_A && mine) r = v.r[n];
      ok = bar_wait(dfull((j + 1) % kDescs), ((j + 1) / kDescs) & 1);
      const int4 mn = ok ? desc_meta(j + 1) : make_int4(-1, 0, 0, 0);
      if (mn.x >= 0) nb = desc_nodes(j + 1);  // after the last tile its own entries once more
      const uint4 recn = mn.x >= 0 ? desc_rec(j + 1) : rec;
      ok = ok && bar_wait(full(b), (j / kStages) & 1);
      double yu = 0.0, yv = 0.0;
      double2 sn = make_double2(0.0, 0.0);
      const double2* src = stage_src(b);
      if (m.z >= 0 && !fp64) {
        const Entry* own = reinterpret_cast<const Entry*>(stage_own(b)) + (inside ? i : 0);
        const double2* dg = reinterpret_cast<const double2*>(stage_own(b)) + (inside ? i : 0) + 13 * slots;
#pragma unroll
        for (int q = 0; q < 9; ++q) {
          const double2* sq = src + (k + 1) * ls + slot_of(rec, q);
#pragma unroll
          for (int kA = -1; kA <= 1; ++kA) {
            const int mm = (kA + 1) * 9 + q;
            const double2 sv = sq[kA * ls];
            if (mm == 13) sn = sv;
            double2 a0, a1;
            if (mm < 13) {
              if constexpr (F32) {
                a0 = make_double2((double)T[mm].x, (double)T[mm].z);
                a1 = make_double2((double)T[mm].y, (double)T[mm].w);
              } else {
                a0 = make_double2(T[2 * mm].x, T[2 * mm + 1].x);
                a1 = make_double2(T[2 * mm].y, T[2 * mm + 1].y);
              }
              load_t(mm, nb);
            } else if constexpr (F32) {
              if (mm == 13) {
                a0 = dg[0];
                a1 = dg[slots];
              } else {
                const Entry a = own[(mm - 14) * slots];
                a0 = make_double2((double)a.x, (double)a.y);
                a1 = make_double2((double)a.z, (double)a.w);
              }
            } else {
              a0 = own[(mm - 13) * slots];
              a1 = own[(mm + 1) * slots];
            }
            yu += dot2(a0, sv);
            yv += dot2(a1, sv);
          }
        }
      }
      ok = __all_sync(0xffffffffu, ok);  // the lanes leave together, with nothing stored
      if (!ok) break;
      if (lane == 0) bar_arrive(empty(b));
      if (m.z < 0 || fp64) {
        if (mine) {
          const double2 y = plain_row_call<STORE>(v, fp64, v.tile_col0[m.x] + c, k, n, s);
          yu = y.x;
          yv = y.y;
          sn = s[n];
        }
#pragma unroll
        for (int e = 0; e < 13; ++e) load_t(e, nb);
      }
      double part[NV];
#pragma unroll
      for (int e = 0; e < NV; ++e) part[e] = 0.0;
      if (mine) {
        const double2 y = make_double2(yu, yv);
        if (MODE == MV_CG_FIRST) v.d0[n] = sn;
        if (MODE == MV_CG1) v.Az[n] = y;
        else v.q[n] = y;
        if (MODE == MV_STD_A) {
          part[0] = dot2(sn, y);
        } else {
          part[0] = dot2(r, sn);
          part[NV > 1 ? 1 : 0] = dot2(y, sn);
          part[NV > 2 ? 2 : 0] = dot2(r, r);
        }
      }
#pragma unroll
      for (int e = 0; e < NV; ++e) {
        double x = part[e];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) v.wsum[((size_t)m.x * 8 + warp) * 3 + e] = x;
      }
      if (i == 0 && v.mv_nodes && !v.dry) atomicAdd(&v.mv_nodes[F32 && !fp64 ? 1 : 0], (unsigned long long)m.y * nz);
      m = mn;
      rec = recn;
    }
  }
  // the tiles' sums, tickets, and where this CTA brought an instance's last
  // tile the instance's sums (tile_finish's order) and scalar update
  const bool all_ok = __syncthreads_and(ok);
  __shared__ double sm[NV * 32];
  constexpr int kFins = 32;
  __shared__ int fins[kFins], nfin;
  __shared__ double fin_sum[kFins][NV];
  const int bd = v.tile_threads;  // the threads tile_finish sums with
  // the stages are free: two halves, each for the partials of every sum of
  // `chunk` tiles (three more for alignment), whole rounds of bd
  double* buf = reinterpret_cast<double*>(st_sm);
  const int chunk = ((int)(H.stage / (8 * NV)) - 3) / bd * bd, pitch = (chunk + 3) & ~1;
  auto stage_partials = [&](int c0, int end, int half) {  // by 16-byte copies
    const int n = end - c0 < chunk ? end - c0 : chunk;
#pragma unroll
    for (int e = 0; e < NV; ++e) {
      const size_t at = (size_t)e * v.ntiles + c0, at0 = at & ~(size_t)1;
      const int n16 = (int)((at + n - at0 + 1) >> 1);
      for (int q = i; q < n16; q += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_at(buf + (half * NV + e) * pitch + 2 * q)),
                     "l"(v.partials + at0 + 2 * q)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int base = blockIdx.x; base < v.ntiles; base += G * blockDim.x) {
    const long tl = (long)base + (long)i * G;
    const int t = tl < v.ntiles ? (int)tl : -1;
    int inst = -1, done = 0;
    if (t >= 0) {
      inst = v.tile_inst[t];
      if (v.dry || v.st[inst].pcg_active) {
#pragma unroll
        for (int e = 0; e < NV; ++e) {
          double w[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) w[q] = q < nw ? v.wsum[((size_t)t * 8 + q) * 3 + e] : 0.0;
          const double x = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
          v.partials[(size_t)e * v.ntiles + t] = all_ok ? x : __longlong_as_double(0x7ff8000000000000LL);
        }
        __threadfence();
      } else {
        inst = -1;
      }
    }
    // one ticket for a warp's tiles of an instance (thousands of atomics on
    // one address, all at the end, are a queue)
    const unsigned same = __match_any_sync(0xffffffffu, inst);
    __syncwarp();
    if (inst >= 0 && lane == __ffs(same) - 1) {
      const InstParams& ip = v.inst[inst];
      const unsigned cnt = __popc(same);
      done = atomicAdd(&v.tile_counter[inst], cnt) + cnt == (unsigned)(ip.tile_end - ip.tile_begin);
    }
    // the instances whose last tickets came to this CTA, a list at a time:
    // their sums one after the other, each thread in tile_finish's order, the
    // next one's partials on their way meanwhile, then the scalar updates
    // side by side
    for (;;) {
      if (i == 0) nfin = 0;
      __syncthreads();
      if (done) {
        const int p = atomicAdd(&nfin, 1);
        if (p < kFins) {
          fins[p] = inst;
          done = 0;
        }
      }
      __syncthreads();
      const int nf = nfin < kFins ? nfin : kFins;
      if (nf == 0) break;
      __threadfence();
      // what the updates read, on its way meanwhile
      constexpr int kLines = (sizeof(InstState) + 63) / 64;
      for (int q = i; q < nf * kLines; q += blockDim.x)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char*>(v.st + fins[q / kLines]) +
                                                      64 * (q % kLines)));
      double x[NV];
#pragma unroll
      for (int e = 0; e < NV; ++e) x[e] = 0.0;
      int f = 0, c0 = v.inst[fins[0]].tile_begin, end = v.inst[fins[0]].tile_end, half = 0;
      stage_partials(c0, end, 0);
      while (f < nf) {
        const int n = end - c0 < chunk ? end - c0 : chunk;
        int f1 = f, c1 = c0 + chunk, end1 = end;
        if (c1 >= end && ++f1 < nf) {
          c1 = v.inst[fins[f1]].tile_begin;
          end1 = v.inst[fins[f1]].tile_end;
        }
        if (f1 < nf) {
          stage_partials(c1, end1, half ^ 1);
          asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
          asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (i < bd)
#pragma unroll
          for (int e = 0; e < NV; ++e) {
            const double* p = buf + (half * NV + e) * pitch + (((size_t)e * v.ntiles + c0) & 1);
#pragma unroll 4
            for (int t = i; t < n; t += bd) x[e] += p[t];
          }
        if (f1 != f) {
          block_reduce<NV, false>(x, sm);
#pragma unroll
          for (int e = 0; e < NV; ++e) {
            if (i == 0) fin_sum[f][e] = all_ok ? x[e] : __longlong_as_double(0x7ff8000000000000LL);
            x[e] = 0.0;
          }
        }
        __syncthreads();
        f = f1;
        c0 = c1;
        end = end1;
        half ^= 1;
      }
      if (i < nf) {
        const int in = fins[i];
        v.tile_counter[in] = 0;
        if (!v.dry) {
          double x[NV];
#pragma unroll
          for (int e = 0; e < NV; ++e) x[e] = fin_sum[i][e];
          if (MODE == MV_STD_A) std_mv_fin<true>(v, v.st[in], x);
          else cg_mv_fin<MODE == MV_CG_FIRST, true>(v, v.inst[in], v.st[in], x);
        }
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------
// Picard convergence: compute_residual_velocity_3d (:9111-9234).
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(kTile) k_picard_check(DevView v) {
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    InstState& S = v.st[R.inst];
    const InstParams& ip = v.inst[R.inst];
    const int n = R.n0 + threadIdx.x;
    const bool mine = tile_mine(v, R, threadIdx.x);
    if (S.zero_x) {
      if (mine) v.x[n] = make_double2(0.0, 0.0);
      continue;
    }
    if (!S.picard_active) continue;
    const bool meanu = ip.which_resid == 2;
    // the 2-D criterion has no bed layer to leave out (:9238-9351)
    const bool nobed = !v.solve2d && (ip.which_resid == 1 || meanu);
    double part[2] = {0.0, 0.0};
    if (mine) {
      if (S.frozen) v.x[n] = make_double2(0.0, 0.0);  // 2-D solve on a no-slip bed
      const int k = tile_k(v, threadIdx.x);
      if (!(nobed && k == v.nz - 1)) {
        const double2 x = v.x[n], o = v.usav[n];
        const double speed = sqrt(x.x * x.x + x.y * x.y);
        if (speed != 0.0) {
          const double old = sqrt(o.x * o.x + o.y * o.y);
          part[0] = fabs((old - speed) / speed);
          part[1] = 1.0;
        }
      }
    }
    auto fin = [&](int inst, const double* s) {
      InstState& S2 = v.st[inst];
      const InstParams& ip2 = v.inst[inst];
      const bool mean2 = ip2.which_resid == 2;
      S2.resid_velo = mean2 ? (s[1] > 0.0 ? s[0] / s[1] : 0.0) : s[0];
      double crit, target;
      if (ip2.which_resid == 3) { crit = S2.L2_norm; target = 1.0e-4; }
      else if (ip2.which_resid == 4) { crit = S2.L2_rel; target = 1.0e-7; }
      else { crit = S2.resid_velo; target = 1.0e-4; }
      const bool done = !(crit >= target) || S2.picard_iter >= ip2.maxiter_nonlinear;
      if (done) {
        S2.picard_converged = S2.picard_iter < ip2.maxiter_nonlinear ? 1 : 0;
        S2.picard_active = 0;
        atomicSub(&v.cnt->picard_active, 1);
      }
    };
    if (meanu) tile_finish<2, false>(v, t, R.inst, part, fin);
    else tile_finish<2, true>(v, t, R.inst, part, fin);
  }
}

// ---------------------------------------------------------------------
// Mixed precision: FP32 copy of the symmetric matrix for the Krylov
// iteration; the every-ncheck true residual r = b - A x stays FP64, so the
// iteration is a reliable-update PCG that converges to the FP64 solution.
// ---------------------------------------------------------------------
// FP32 copy of the symmetric matrix with the row-sum compensated FP64
// diagonal block (make_a32_row).
__global__ void __launch_bounds__(kTile) k_make_a32(DevView v) {
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    if (!v.st[R.inst].pcg_active) continue;
    const int n = R.n0 + threadIdx.x;
    if (!tile_mine(v, R, threadIdx.x)) continue;
    const int col = tile_col(v, R, threadIdx.x), k = tile_k(v, threadIdx.x);
    make_a32_row(v, col, k, (size_t)n);
  }
}

// Factors of the SIA column preconditioner for the linear solve ahead:
// one thread per (column, component) of the instances that use it and are
// solving (sia_factor_column).
__global__ void __launch_bounds__(256) k_sia_factor(DevView v) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 2L * v.ncols) return;
  const int col = (int)(t >> 1), h = (int)(t & 1);
  const int inst = v.col_inst[col];
  if (v.inst[inst].precond != 2 || !v.st[inst].pcg_active) return;
  sia_factor_column(v, col, h);
}

// Post-solve diagnostics (glissade_velo_higher.F90:3847-3872) at the
// current velocity: the element stresses of compute_internal_stress into
// out[6][nelem] (a singular Jacobian marks the instance, as assembly pass 1
// does) and the basal frictional heat flux of
// compute_basal_friction_heatflx into bf (per active cell for the
// finite-element method, per column for the local one).
__global__ void __launch_bounds__(256) k_internal_stress(DevView v, double* out) {
  const size_t ne = (size_t)v.nelem;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < v.nelem; e += gridDim.x * blockDim.x) {
    double tau[6];
    if (!stress_element(v, c_T, e, tau)) {
      atomicExch(&v.st[v.cell_inst[e / (v.nz - 1)]].status, BP_ERR_SINGULAR_JAC);
      for (int q = 0; q < 6; ++q) tau[q] = 0.0;
    }
    for (int q = 0; q < 6; ++q) out[(size_t)q * ne + e] = tau[q];
  }
}

__global__ void __launch_bounds__(256) k_bfric(DevView v, int which, double* bf) {
  const int n = which == 0 ? v.ncells : v.ncols;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    bf[i] = which == 0 ? bfric_cell(v, c_T, i) : bfric_vertex(v, i);
}

// Plain y = A x for bp_matvec.
__global__ void __launch_bounds__(kTile) k_matvec_plain(DevView v, const double2* x, double2* y) {
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const int n = R.n0 + threadIdx.x;
    if (!tile_mine(v, R, threadIdx.x)) continue;
    const int col = tile_col(v, R, threadIdx.x), k = tile_k(v, threadIdx.x);
    y[n] = v.sym ? matvec_row_sym(v, v.A, col, k, n, SrcX{x}) : matvec_row(v, v.A, col, k, n, SrcX{x});
  }
}

// y = A x for the autotuner and the kernel sweep: one storage variant and
// one occupancy target (MINB = minimum resident CTAs per SM, 0 = free).
template <int STORE, int MINB>
__global__ void __launch_bounds__(kTile, MINB) k_tune_mv(DevView v) {
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const int n = R.n0 + threadIdx.x;
    if (!tile_mine(v, R, threadIdx.x)) continue;
    const int col = tile_col(v, R, threadIdx.x), k = tile_k(v, threadIdx.x);
    v.Az[n] = mv_row<STORE>(v, col, k, n, v.x);
  }
}

// Diagonal preconditioner for matrix-level entry points.
__global__ void __launch_bounds__(kTile) k_dinv(DevView v, int precond) {
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const int n = R.n0 + threadIdx.x;
    if (!tile_mine(v, R, threadIdx.x)) continue;
    const size_t np = (size_t)v.npad;
    double2 di = make_double2(1.0, 1.0);
    (void)np;
    if (precond == 1) {
      const double du = diag_u(v, n), dv = diag_v(v, n);
      di.x = du != 0.0 ? 1.0 / du : 0.0;
      di.y = dv != 0.0 ? 1.0 / dv : 0.0;
    }
    v.Dinv[n] = di;
  }
}

// (b,b) for matrix-level entry points.
__global__ void __launch_bounds__(kTile) k_bb(DevView v) {
  for (int t = blockIdx.x; t < v.ntiles; t += gridDim.x) {
    const TileRange R = tile_range(v, t);
    const int n = R.n0 + threadIdx.x;
    double part[1] = {0.0};
    if (tile_mine(v, R, threadIdx.x)) {
      const double2 b = v.b[n];
      part[0] = b.x * b.x + b.y * b.y;
    }
    tile_finish<1, false>(v, t, R.inst, part, [&](int inst, const double* s) {
      v.st[inst].bb = s[0];
      v.st[inst].L2_rhs = sqrt(s[0]);
    });
  }
}

// ---------------------------------------------------------------------
// host-side launchers
// ---------------------------------------------------------------------
static inline int tile_grid(const DevView& v) {
  int g = v.ntiles > 0 ? v.ntiles : 1;
  if (v.grid_cap > 0 && g > v.grid_cap) g = v.grid_cap;
  return g;
}

cudaError_t upload_ref_tables() {
  RefTables t;
  fill_ref_tables(&t);
  return cudaMemcpyToSymbol(c_T, &t, sizeof(t));
}

void launch_picard_begin(const DevView& v, cudaStream_t s) { k_picard_begin<<<1, 256, 0, s>>>(v); }
void launch_save_usav(const DevView& v, cudaStream_t s) { k_save_usav<<<tile_grid(v), v.tile_threads, 0, s>>>(v); }
void launch_slide_beta(const DevView& v, cudaStream_t s) {
  if (v.ncols > 0) k_slide_beta<<<(v.ncols + kTile - 1) / kTile, kTile, 0, s>>>(v);
  if (v.ncells > 0) k_cell_beta<<<(v.ncells + kTile - 1) / kTile, kTile, 0, s>>>(v);
}
void launch_asm_qp(const DevView& v, cudaStream_t s) {
  if (v.solve2d) {
    if (v.ncells > 0) {
      const long threads = (long)v.ncells * 4;
      if (v.l1l2 || v.diva) k_asm2_qp<true><<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(v);
      else k_asm2_qp<false><<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(v);
    }
  } else if (v.nelem > 0) {
    const long threads = (long)v.nelem * 8;
    k_asm_qp<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(v);
  }
}
void launch_asm_rows(const DevView& v, cudaStream_t s) {
  dim3 g(tile_grid(v), 4);
  if (v.solve2d) {
    k_asm_rows<ASM_2D><<<g, v.tile_threads, 0, s>>>(v);
  } else if (v.Ke) {
    if (v.nelem > 0) k_asm_elem<<<(unsigned)(((long)v.nelem * 8 + 255) / 256), 256, 0, s>>>(v);
    k_asm_rows<ASM_GATHER><<<g, v.tile_threads, 0, s>>>(v);
  } else {
    k_asm_rows<ASM_ROWS><<<g, v.tile_threads, 0, s>>>(v);
  }
}
void launch_rhs(const DevView& v, cudaStream_t s) { k_rhs<<<tile_grid(v), v.tile_threads, 0, s>>>(v); }
void launch_diva_beta(const DevView& v, cudaStream_t s) {
  if (v.ncells > 0) k_diva_cells<<<(unsigned)((v.ncells + 255) / 256), 256, 0, s>>>(v);
  if (v.ncols > 0) k_diva_beta<<<(unsigned)((v.ncols + 255) / 256), 256, 0, s>>>(v);
  if (v.ncells > 0) k_diva_cell_beta<<<(unsigned)((v.ncells + 255) / 256), 256, 0, s>>>(v);
}
void launch_diva_velocity(const DevView& v, cudaStream_t s) {
  if (v.ncols > 0) k_diva_velocity<<<(unsigned)((v.ncols + 255) / 256), 256, 0, s>>>(v);
}
void launch_l1l2_velocity(const DevView& v, cudaStream_t s) {
  if (v.ncells > 0) k_l1l2_cells<<<(unsigned)((v.ncells + 255) / 256), 256, 0, s>>>(v);
  if (v.ncols > 0) k_l1l2_columns<<<(unsigned)((v.ncols + 255) / 256), 256, 0, s>>>(v);
}
void launch_assemble(const DevView& v, cudaStream_t s) {
  launch_asm_qp(v, s);
  launch_asm_rows(v, s);
  launch_rhs(v, s);
}
// PCG kernels are launched as programmatic dependents of their stream
// predecessor (BP_PDL=0 turns this off, and so does set_pdl(false), e.g.
// while a graph that cannot hold programmatic edges is captured), and with
// the problem's L2 access-policy window when it has one.
static const bool g_pdl_env = [] {
  const char* e = std::getenv("BP_PDL");
  return !(e && e[0] == '0');
}();
static thread_local bool g_pdl_on = true;
void set_pdl(bool on) { g_pdl_on = on; }

static void launch_pcg(void (*kernel)(DevView), int g, cudaStream_t s, const DevView& v, int block = 0,
                       size_t smem = 0) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g);
  cfg.blockDim = dim3(block > 0 ? block : v.tile_threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  unsigned na = 0;
  if (g_pdl_env && g_pdl_on) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (v.l2_bytes > 0) {
    at[na].id = cudaLaunchAttributeAccessPolicyWindow;
    at[na].val.accessPolicyWindow.base_ptr = const_cast<void*>(v.l2_base);
    at[na].val.accessPolicyWindow.num_bytes = v.l2_bytes;
    at[na].val.accessPolicyWindow.hitRatio = v.l2_hit;
    at[na].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    at[na].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    ++na;
  }
  cfg.attrs = at;
  cfg.numAttrs = na;
  cudaLaunchKernelEx(&cfg, kernel, v);
}

using TileKernel = void (*)(DevView);

template <int STORE, int MINB>
static void launch_resid_store(int mode, const DevView& v, cudaStream_t s, int g) {
  switch (mode) {
    case MV_INIT: launch_pcg(k_resid<MV_INIT, STORE, MINB>, g, s, v); break;
    case MV_CHECK: launch_pcg(k_resid<MV_CHECK, STORE, MINB>, g, s, v); break;
    default: launch_pcg(k_resid<MV_REFINE, STORE, MINB>, g, s, v); break;
  }
}
template <int STORE, int MINB>
static TileKernel krylov_kernel(int mode) {
  switch (mode) {
    case MV_STD_A: return k_std_mv<STORE, MINB>;
    case MV_CG_FIRST: return k_cg_mv<true, STORE, MINB>;
    default: return k_cg_mv<false, STORE, MINB>;
  }
}
template <int STORE>
static TileKernel krylov_kernel_st(int mode, int minb) {
  if (minb == 8) return krylov_kernel<STORE, 8>(mode);
  if (minb == 6) return krylov_kernel<STORE, 6>(mode);
  if (minb == 4) return krylov_kernel<STORE, 4>(mode);
  return krylov_kernel<STORE, 0>(mode);
}
static TileKernel krylov_kernel_for(const DevView& v, int mode, int minb) {
  if (!v.sym) return krylov_kernel_st<ST_FULL>(mode, minb);
  if (v.A32) return krylov_kernel_st<ST_SYM32>(mode, minb);
  return krylov_kernel_st<ST_SYM>(mode, minb);
}
static inline bool is_krylov(int mode) {
  return mode == MV_STD_A || mode == MV_CG_FIRST || mode == MV_CG1;
}
template <int STORE>
static void launch_resid_minb(int mode, const DevView& v, cudaStream_t s, int g) {
  if (v.minb == 4) launch_resid_store<STORE, 4>(mode, v, s, g);
  else launch_resid_store<STORE, 0>(mode, v, s, g);
}
// CTAs of `threads` threads and `smem` bytes of dynamic shared memory that an
// SM holds of kernel k (0: none, or an error).  The kernel is first allowed all
// that a block may have: that limit is one value per kernel and device for the
// whole process, so it is never the size one problem needs -- a problem made
// later, on this thread or another, would lower it under the launches of those
// that are alive.
static int ctas_per_sm(TileKernel k, int threads, size_t smem) {
  int dev = 0, most = 0, n = 0;
  cudaFuncAttributes fa;
  if (cudaGetDevice(&dev) == cudaSuccess &&
      cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
      cudaFuncGetAttributes(&fa, k) == cudaSuccess) {
    const int room = most - (int)fa.sharedSizeBytes;
    if (smem <= (size_t)room &&
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, room) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, threads, smem) == cudaSuccess)
      return n;
  }
  cudaGetLastError();
  return 0;
}

template <int STORE, int THREADS, int LS>
static TileKernel staged_kernel_st(int mode) {
  switch (mode) {
    case MV_STD_A: return k_mv_staged<STORE, MV_STD_A, THREADS, LS>;
    case MV_CG_FIRST: return k_mv_staged<STORE, MV_CG_FIRST, THREADS, LS>;
    default: return k_mv_staged<STORE, MV_CG1, THREADS, LS>;
  }
}
static TileKernel staged_kernel(const DevView& v, int mode) {
  constexpr int LS16 = StagedDesc::zero_slot(16) + 1;
  if (v.W == 16 && v.tile_threads <= 192)
    return v.A32 ? staged_kernel_st<ST_SYM32, 224, LS16>(mode) : staged_kernel_st<ST_SYM, 224, LS16>(mode);
  return v.A32 ? staged_kernel_st<ST_SYM32, 288, 0>(mode) : staged_kernel_st<ST_SYM, 288, 0>(mode);
}
int staged_per_sm(const DevView& v) {
  if (!v.sym || v.nz == 1 || StagedDesc::zero_slot(v.W) > 255) return 0;
  const StagedShape h = staged_shape(v, v.A32 != nullptr);
  int least = 0;
  for (int mode : {(int)MV_STD_A, (int)MV_CG_FIRST, (int)MV_CG1}) {
    const int n = ctas_per_sm(staged_kernel(v, mode), v.tile_threads + 32, h.bytes);
    if (n == 0) return 0;
    least = least == 0 ? n : (n < least ? n : least);
  }
  return least;
}
void launch_staged_desc(const DevView& v, unsigned char* desc, cudaStream_t s) {
  if (v.ntiles > 0) k_staged_desc<<<v.ntiles, 256, 2 * 9 * v.W * sizeof(int), s>>>(v, desc);
}
void launch_mv(int mode, const DevView& v, cudaStream_t s) {
  if (is_krylov(mode) && v.staged) {
    const int g = v.ntiles < v.grid_k ? v.ntiles : v.grid_k;
    launch_pcg(staged_kernel(v, mode), g, s, v, v.tile_threads + 32, staged_shape(v, v.A32 != nullptr).bytes);
    return;
  }
  if (is_krylov(mode)) {
    int g = v.ntiles > 0 ? v.ntiles : 1;
    if (v.grid_k > 0 && g > v.grid_k) g = v.grid_k;
    launch_pcg(krylov_kernel_for(v, mode, v.minb_k), g, s, v);
    return;
  }
  const int g = tile_grid(v);
  if (!v.sym) launch_resid_minb<ST_FULL>(mode, v, s, g);
  else if (v.A32) launch_resid_minb<ST_SYM32>(mode, v, s, g);
  else launch_resid_minb<ST_SYM>(mode, v, s, g);
}
int krylov_resident_ctas(const DevView& v, int mode, int minb) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, krylov_kernel_for(v, mode, minb), v.tile_threads, 0) !=
      cudaSuccess)
    return 0;
  return n;
}
void launch_std_update(bool check, const DevView& v, cudaStream_t s) {
  launch_pcg(check ? k_std_update<true> : k_std_update<false>, tile_grid(v), s, v);
}
void launch_std_dir(const DevView& v, cudaStream_t s) { launch_pcg(k_std_dir, tile_grid(v), s, v); }
void launch_cg_first_update(const DevView& v, cudaStream_t s) {
  launch_pcg(k_cg_first_update, tile_grid(v), s, v);
}
void launch_cg_update(bool check, const DevView& v, cudaStream_t s) {
  launch_pcg(check ? k_cg_update<true> : k_cg_update<false>, tile_grid(v), s, v);
}
template <int STORE, int PER_SM>
static TileKernel resident_kernel_st(int variant) {
  return variant == 3 ? k_pcg_resident<STORE, 3, PER_SM> : k_pcg_resident<STORE, 2, PER_SM>;
}
static TileKernel resident_kernel(const DevView& v, int variant, size_t* smem) {
  *smem = resident_shape(v, v.sym && v.A32, variant).bytes;
  if (!v.sym) return resident_kernel_st<ST_FULL, 1>(variant);
  if (!v.A32) return resident_kernel_st<ST_SYM, 1>(variant);
  return v.tile_threads <= 192 ? resident_kernel_st<ST_SYM32, 2>(variant) : resident_kernel_st<ST_SYM32, 1>(variant);
}
int resident_ctas(const DevView& v, int variant, int num_sms) {
  size_t smem = 0;
  TileKernel k = resident_kernel(v, variant, &smem);
  return ctas_per_sm(k, v.tile_threads, smem) * num_sms;
}
cudaError_t launch_pcg_resident(const DevView& v, int variant, cudaStream_t s) {
  size_t smem = 0;
  TileKernel k = resident_kernel(v, variant, &smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(v.ntiles);
  cfg.blockDim = dim3(v.tile_threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, v);
}
void launch_picard_check(const DevView& v, cudaStream_t s) {
  k_picard_check<<<tile_grid(v), v.tile_threads, 0, s>>>(v);
}

// Conditions of the device-resident loops (CUDA-graph WHILE nodes).  One
// thread: count this pass in *iter (reset to 0 by `reset`) and keep
// looping while some instance is active (counter *active > 0) and fewer
// than `cap` passes ran, so every loop ends after at most `cap` passes.
__global__ void k_loop_cond(cudaGraphConditionalHandle h, const int* active, int* iter, int cap, int reset) {
  const int it = reset ? (*iter = 0) : ++*iter;
  cudaGraphSetConditional(h, (*active > 0 && it < cap) ? 1u : 0u);
}
void launch_loop_cond(cudaGraphConditionalHandle h, const DevView& v, bool picard, int* iter, int cap, bool reset,
                      cudaStream_t s) {
  const int* active = picard ? &v.cnt->picard_active : &v.cnt->pcg_active;
  k_loop_cond<<<1, 1, 0, s>>>(h, active, iter, cap, reset ? 1 : 0);
}
void launch_make_a32(const DevView& v, cudaStream_t s) { k_make_a32<<<tile_grid(v), v.tile_threads, 0, s>>>(v); }
void launch_sia_factor(const DevView& v, cudaStream_t s) {
  if (v.sia_f && v.ncols > 0) k_sia_factor<<<(unsigned)((2L * v.ncols + 255) / 256), 256, 0, s>>>(v);
}
void launch_matvec_plain(const DevView& v, const double2* x, double2* y, cudaStream_t s) {
  k_matvec_plain<<<tile_grid(v), v.tile_threads, 0, s>>>(v, x, y);
}
void launch_dinv(const DevView& v, int precond, cudaStream_t s) {
  k_dinv<<<tile_grid(v), v.tile_threads, 0, s>>>(v, precond);
}
// Node layout <-> [column][level] in two arrays, the form in which a host
// array's columns are one copy each.  Bandwidth: 32 bytes a node and way; the
// strided side (a column's levels are W nodes apart) is served by L1.
__global__ void __launch_bounds__(256) k_pack(const __grid_constant__ DevView v, const double2* x, double* u, double* w) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)v.ncols * v.nz) return;
  const int col = (int)(t / v.nz), k = (int)(t - (long)col * v.nz);
  const double2 a = x[node_of(v, col, k)];
  u[t] = a.x;
  w[t] = a.y;
}
__global__ void __launch_bounds__(256) k_unpack(const __grid_constant__ DevView v, long t0, long t1, const double* u,
                                                const double* w, double2* x) {
  const long t = t0 + (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= t1) return;
  const int col = (int)(t / v.nz), k = (int)(t - (long)col * v.nz);
  x[node_of(v, col, k)] = make_double2(u[t], w[t]);
}
void launch_pack(const DevView& v, const double2* x, double* u, double* w, cudaStream_t s) {
  const long n = (long)v.ncols * v.nz;
  if (n > 0) k_pack<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(v, x, u, w);
}
void launch_unpack(const DevView& v, int col_begin, int col_end, const double* u, const double* w, double2* x,
                   cudaStream_t s) {
  const long t0 = (long)col_begin * v.nz, t1 = (long)col_end * v.nz;
  if (t1 > t0) k_unpack<<<(unsigned)((t1 - t0 + 255) / 256), 256, 0, s>>>(v, t0, t1, u, w, x);
}

// A caller's matrix rows into the node layout, 32 rows (a warp each block) at
// a time through shared memory: read and written along their own contiguous
// direction.
__global__ void __launch_bounds__(128) k_gather_matrix(const __grid_constant__ DevView v, const double* raw,
                                                       const int* row_node, long row0, long rows) {
  __shared__ double sm[4][32 * 27 + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;  // warp: block uu, uv, vu, vv
  const long r0 = (long)blockIdx.x * 32;
  const int nr = (int)min(32L, rows - r0);
  const double* src = raw + (size_t)warp * rows * 27 + r0 * 27;
  for (int e = lane; e < nr * 27; e += 32) sm[warp][e] = src[e];
  __syncthreads();
  const int n = lane < nr ? row_node[row0 + r0 + lane] : -1;
  if (n < 0) return;
  const size_t np = (size_t)v.npad;
  // warps 0, 1 the u-row's entries, 2, 3 the v-row's
  const int h = warp >> 1;
  for (int m = warp & 1; m < 27; m += 2)
    v.A[(size_t)(h * 27 + m) * np + n] = make_double2(sm[2 * h][lane * 27 + m], sm[2 * h + 1][lane * 27 + m]);
}
void launch_gather_matrix(const DevView& v, const double* raw, const int* row_node, long row0, long rows,
                          cudaStream_t s) {
  if (rows > 0) k_gather_matrix<<<(unsigned)((rows + 31) / 32), 128, 0, s>>>(v, raw, row_node, row0, rows);
}
void launch_bb(const DevView& v, cudaStream_t s) { k_bb<<<tile_grid(v), v.tile_threads, 0, s>>>(v); }
// The 3-D velocity of a shallow-shelf solve (its 2-D solution on every
// level, :3745-3750) for the post-solve diagnostics.
__global__ void __launch_bounds__(256) k_levels_from_2d(DevView v, double2* x3, int L) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < (long)v.ncols * L) x3[t] = v.x[v.col_node[t / L]];
}

// The bed-face corner betas from the columns' beta_internal (0 where a
// corner has no column) for every cell.
__global__ void __launch_bounds__(256) k_corner_beta(DevView v) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= v.ncells) return;
  for (int q = 0; q < 4; ++q) {
    const int col = v.cell_cols[(size_t)q * v.ncells + cell];
    v.cell_beta[(size_t)q * v.ncells + cell] = col >= 0 ? v.col_beta[col] : 0.0;
  }
}

void launch_levels_from_2d(const DevView& v, double2* x3, int L, cudaStream_t s) {
  const long n = (long)v.ncols * L;
  if (n > 0) k_levels_from_2d<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(v, x3, L);
}
void launch_corner_beta(const DevView& v, cudaStream_t s) {
  if (v.ncells > 0) k_corner_beta<<<(unsigned)((v.ncells + 255) / 256), 256, 0, s>>>(v);
}

void launch_diagnostics(const DevView& v, int which_bfric, double* tau, double* bf, cudaStream_t s) {
  if (tau && v.nelem > 0) k_internal_stress<<<(v.nelem + 255) / 256, 256, 0, s>>>(v, tau);
  const int n = which_bfric == 0 ? v.ncells : v.ncols;
  if (bf && n > 0) k_bfric<<<(n + 255) / 256, 256, 0, s>>>(v, which_bfric, bf);
}
int launch_tune_mv(int store, int minb, int grid, const DevView& v, cudaStream_t s) {
  const int g = grid > 0 ? grid : tile_grid(v);
#define TUNE(ST, MB) k_tune_mv<ST, MB><<<g, v.tile_threads, 0, s>>>(v)
  if (store == ST_FULL && !v.sym) {
    if (minb == 8) TUNE(ST_FULL, 8); else if (minb == 6) TUNE(ST_FULL, 6);
    else if (minb == 4) TUNE(ST_FULL, 4); else TUNE(ST_FULL, 0);
  } else if (store == ST_SYM && v.sym) {
    if (minb == 8) TUNE(ST_SYM, 8); else if (minb == 6) TUNE(ST_SYM, 6);
    else if (minb == 4) TUNE(ST_SYM, 4); else TUNE(ST_SYM, 0);
  } else if (store == ST_SYM32 && v.sym && v.A32) {
    if (minb == 8) TUNE(ST_SYM32, 8); else if (minb == 6) TUNE(ST_SYM32, 6);
    else if (minb == 4) TUNE(ST_SYM32, 4); else TUNE(ST_SYM32, 0);
  } else {
    return -1;
  }
#undef TUNE
  return 0;
}

}  // namespace bp
