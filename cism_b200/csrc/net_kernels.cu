// net_kernels.cu -- BF16 kernels of the learned initial guess: a 2-D
// U-Net over the vertex grid, trained and run on the device.
//
// Activations are NHWC ([pixel][channel]) in BF16; every contraction is a
// tensor-core GEMM on tcgen05 (k_gemm_tc: BF16 operands from shared memory,
// FP32 accumulator in tensor memory; the mma.sync kernel k_gemm_tn remains
// for comparison) over K-contiguous operands:
//   forward  Y[P][Cout]  = col(X)[P][K] . W[Cout][K]^T            (K = 9 Cin)
//   dgrad    dcol[P][K]  = dY[P][Cout] . WT[K][Cout]^T, then col2im
//   wgrad    dW[Cout][K] = dYT[Cout][P] . colT[K][P]^T
// with k = tap * Cin + c, tap = (dy + 1) * 3 + (dx + 1).  Borders are
// periodic (the doubly periodic domains) or zero.  Reductions (bias
// gradients, the loss) run in a fixed order, so a training run is
// deterministic.  Every entry point is extern "C" with plain device
// pointers and the CUDA stream to launch on.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <algorithm>
#include <cstdlib>
#include <map>
#include <mutex>
#include <cstring>

namespace {

typedef __nv_bfloat16 bf16;

// ---------------------------------------------------------------------
// GEMM: C[m][n] = sum_k A[m][k] B[n][k] (+ bias[n]) (+ C[m][n] if accum).
// Tiles 64 x 64 x 32, 4 warps of 32 x 32, cp.async double buffering.
// K, lda, ldb multiples of 8 (16-byte rows of the 8-element chunks).
// ---------------------------------------------------------------------
constexpr int BM = 64, BN = 64, BK = 32, PAD = 8;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 16 : 0;  // src-size 0: the 16 bytes are zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__global__ void __launch_bounds__(128) k_gemm_tn(const bf16* __restrict__ A, const bf16* __restrict__ B,
                                                 float* __restrict__ C, const float* __restrict__ bias,
                                                 int M, int N, int K, int lda, int ldb, int ldc,
                                                 int accum) {
  __shared__ __align__(16) bf16 As[2][BM][BK + PAD];
  __shared__ __align__(16) bf16 Bs[2][BN][BK + PAD];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;

  auto load = [&](int buf, int k0) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {  // 64 rows x 4 chunks = 256 chunks per operand
      const int id = tid + c * 128;
      const int r = id >> 2, ch = (id & 3) * 8;
      const int k = k0 + ch;
      const bool va = (m0 + r) < M && k < K;
      const bool vb = (n0 + r) < N && k < K;
      cp_async16(&As[buf][r][ch], va ? (const void*)(A + (size_t)(m0 + r) * lda + k) : (const void*)A, va);
      cp_async16(&Bs[buf][r][ch], vb ? (const void*)(B + (size_t)(n0 + r) * ldb + k) : (const void*)B, vb);
    }
  };

  const int nk = (K + BK - 1) / BK;
  load(0, 0);
  cp_async_commit();
  for (int kt = 0; kt < nk; ++kt) {
    const int buf = kt & 1;
    if (kt + 1 < nk) {
      load(buf ^ 1, (kt + 1) * BK);
      cp_async_commit();
      cp_async_wait1();
    } else {
      cp_async_wait0();
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      uint32_t af[2][4], bfr[4][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = wm + i * 16 + g;
        af[i][0] = *reinterpret_cast<const uint32_t*>(&As[buf][r][kk + 2 * t4]);
        af[i][1] = *reinterpret_cast<const uint32_t*>(&As[buf][r + 8][kk + 2 * t4]);
        af[i][2] = *reinterpret_cast<const uint32_t*>(&As[buf][r][kk + 2 * t4 + 8]);
        af[i][3] = *reinterpret_cast<const uint32_t*>(&As[buf][r + 8][kk + 2 * t4 + 8]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int nn = wn + j * 8 + g;
        bfr[j][0] = *reinterpret_cast<const uint32_t*>(&Bs[buf][nn][kk + 2 * t4]);
        bfr[j][1] = *reinterpret_cast<const uint32_t*>(&Bs[buf][nn][kk + 2 * t4 + 8]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], af[i], bfr[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int m = m0 + wm + i * 16 + g + (q >> 1) * 8;
        const int n = n0 + wn + j * 8 + 2 * t4 + (q & 1);
        if (m < M && n < N) {
          float x = acc[i][j][q];
          if (bias) x += bias[n];
          float* dst = C + (size_t)m * ldc + n;
          *dst = accum ? *dst + x : x;
        }
      }
}

// ---------------------------------------------------------------------
// im2col / col2im over [B][H][W][C] with 3 x 3 taps; periodic != 0 wraps.
// ---------------------------------------------------------------------
__device__ __forceinline__ bool tap_pixel(int b, int y, int x, int dy, int dx, int H, int W, int periodic,
                                          long long* p) {
  int yy = y + dy, xx = x + dx;
  if (periodic) {
    yy = (yy + H) % H;
    xx = (xx + W) % W;
  } else if (yy < 0 || yy >= H || xx < 0 || xx >= W) {
    return false;
  }
  *p = ((long long)b * H + yy) * W + xx;
  return true;
}

// im2col of channel counts that are multiples of 8: one thread per (pixel, 8
// channels) copies the nine taps' 16 bytes, so that the index arithmetic (one
// division chain) is spent once per 288 bytes and not per 2-byte element.
// Bound by the 18 C bytes written per pixel: 131,072 pixels of 32 channels
// 25 us (256 us element by element).
__global__ void __launch_bounds__(256) k_im2col8(const uint4* __restrict__ X, uint4* __restrict__ col, unsigned P,
                                                 int H, int W, unsigned C8, int periodic) {
  const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned p = id / C8, c = id - p * C8;
  if (p >= P) return;
  const unsigned row = p / (unsigned)W;
  const int x = (int)(p - row * W), b = (int)(row / (unsigned)H), y = (int)(row - (unsigned)b * H);
  uint4* out = col + (size_t)p * 9 * C8 + c;
#pragma unroll
  for (int tap = 0; tap < 9; ++tap) {
    long long q;
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (tap_pixel(b, y, x, tap / 3 - 1, tap % 3 - 1, H, W, periodic, &q)) val = __ldg(X + (size_t)q * C8 + c);
    out[tap * C8] = val;
  }
}

// The same for any C (the network's few input fields): one thread per 8
// entries of a row, stored as 16 bytes (VEC) where rows allow it.
template <bool VEC>
__global__ void __launch_bounds__(256) k_im2col_any(const bf16* __restrict__ X, bf16* __restrict__ col, unsigned P,
                                                    int H, int W, int C, int Kp, int periodic) {
  const unsigned Kp8 = (unsigned)(Kp + 7) / 8;
  const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned p = id / Kp8, j = id - p * Kp8;
  if (p >= P) return;
  const unsigned row = p / (unsigned)W;
  const int x = (int)(p - row * W), b = (int)(row / (unsigned)H), y = (int)(row - (unsigned)b * H);
  __align__(16) bf16 v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int k = (int)(8 * j) + e, tap = k / C;
    long long q;
    v[e] = __float2bfloat16(0.f);
    if (k < 9 * C && tap_pixel(b, y, x, tap / 3 - 1, tap % 3 - 1, H, W, periodic, &q)) v[e] = X[q * C + (k - tap * C)];
  }
  bf16* out = col + (size_t)p * Kp + 8 * j;
  if (VEC) {
    *reinterpret_cast<uint4*>(out) = *reinterpret_cast<const uint4*>(v);
  } else {
    for (int e = 0; e < 8 && (int)(8 * j) + e < Kp; ++e) out[e] = v[e];
  }
}

// dX[p][c] = sum over taps of dcol[q][tap * C + c], q the pixel whose tap
// lands on p (gather in tap order); V = 4: four channels a thread.
template <int V>
__global__ void __launch_bounds__(256) k_col2im(const float* __restrict__ dcol, float* __restrict__ dX, unsigned P,
                                                int H, int W, unsigned CV, int Kp, int periodic) {
  const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned p = id / CV, c = id - p * CV;
  if (p >= P) return;
  const unsigned row = p / (unsigned)W;
  const int x = (int)(p - row * W), b = (int)(row / (unsigned)H), y = (int)(row - (unsigned)b * H);
  float s[V];
#pragma unroll
  for (int e = 0; e < V; ++e) s[e] = 0.f;
#pragma unroll
  for (int tap = 0; tap < 9; ++tap) {
    long long q;
    if (!tap_pixel(b, y, x, -(tap / 3 - 1), -(tap % 3 - 1), H, W, periodic, &q)) continue;
    const float* d = dcol + (size_t)q * Kp + (size_t)(tap * CV + c) * V;
    if (V == 4) {
      const float4 g = __ldg(reinterpret_cast<const float4*>(d));
      s[0] += g.x; s[V > 1 ? 1 : 0] += g.y; s[V > 2 ? 2 : 0] += g.z; s[V > 3 ? 3 : 0] += g.w;
    } else {
      s[0] += *d;
    }
  }
  float* out = dX + ((size_t)p * CV + c) * V;
  if (V == 4) *reinterpret_cast<float4*>(out) = make_float4(s[0], s[V > 1 ? 1 : 0], s[V > 2 ? 2 : 0], s[V > 3 ? 3 : 0]);
  else *out = s[0];
}

// [R][Cc] -> [Cc][R] (BF16), 32 x 32 tiles through shared memory.
__global__ void k_transpose(const bf16* __restrict__ in, bf16* __restrict__ out, int R, int Cc) {
  __shared__ bf16 tile[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int r = r0 + i, c = c0 + threadIdx.x;
    if (r < R && c < Cc) tile[i][threadIdx.x] = in[(size_t)r * Cc + c];
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, r = r0 + threadIdx.x;
    if (r < R && c < Cc) out[(size_t)c * R + r] = tile[threadIdx.x][i];
  }
}

// ---------------------------------------------------------------------
// pointwise
// ---------------------------------------------------------------------
__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
  const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
  return cdf + x * pdf;
}

#define GRID_LOOP(id, total) \
  for (long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x; id < (total); id += (long long)gridDim.x * blockDim.x)

// The pointwise kernels move V consecutive channels a thread: 16 bytes of
// FP32 (V = 4) or BF16 (V = 8) where the channel counts, slice offsets, row
// lengths and addresses are multiples of that, single elements (V = 1)
// otherwise.  Element by element with 64-bit divisions they ran at 0.6-1.3
// TB/s; each element's arithmetic is the same for every V.
template <typename T, int V>
struct alignas(sizeof(T) * V) Pack {
  T e[V];
};
template <typename T, int V>
__device__ __forceinline__ Pack<T, V> ld_pack(const T* p) {
  return *reinterpret_cast<const Pack<T, V>*>(p);
}
template <typename T, int V>
__device__ __forceinline__ void st_pack(T* p, const Pack<T, V>& v) {
  *reinterpret_cast<Pack<T, V>*>(p) = v;
}
// id -> (row, first channel) of C channels in groups of V
struct RowCol {
  long long p;
  int c;
};
template <int V>
__device__ __forceinline__ RowCol row_col(long long id, int C) {
  const unsigned g = (unsigned)C / V;
  RowCol r;
  if (id < (1LL << 32)) {
    const unsigned q = (unsigned)id / g;
    r.p = q;
    r.c = (int)((unsigned)id - q * g) * V;
  } else {
    r.p = id / g;
    r.c = (int)(id % g) * V;
  }
  return r;
}
// pixel p of [B][H][W] -> (b, y, x)
struct Pix {
  long long b;
  int y, x;
};
__device__ __forceinline__ Pix pixel(long long p, int H, int W) {
  Pix r;
  if (p < (1LL << 32)) {
    const unsigned row = (unsigned)p / (unsigned)W, b = row / (unsigned)H;
    r.x = (int)((unsigned)p - row * W);
    r.y = (int)(row - b * H);
    r.b = b;
  } else {
    r.x = (int)(p % W);
    r.y = (int)((p / W) % H);
    r.b = p / ((long long)W * H);
  }
  return r;
}

// Y = act(Z) in BF16 into a channel slice [p][c0 .. c0 + C) of rows of ldy.
template <int V>
__global__ void __launch_bounds__(256) k_act(const float* __restrict__ Z, bf16* __restrict__ Y, long long P, int C,
                                             int ldy, int c0, int act) {
  GRID_LOOP(id, P * C / V) {
    const RowCol r = row_col<V>(id, C);
    const Pack<float, V> z = ld_pack<float, V>(Z + id * V);
    Pack<bf16, V> y;
#pragma unroll
    for (int e = 0; e < V; ++e) y.e[e] = __float2bfloat16(act ? gelu(z.e[e]) : z.e[e]);
    st_pack(Y + r.p * ldy + c0 + r.c, y);
  }
}

// dZ = dY * act'(Z), dY read from a channel slice of rows of ldd (FP32).
template <int V>
__global__ void __launch_bounds__(256) k_act_grad(const float* __restrict__ Z, const float* __restrict__ dY,
                                                  float* __restrict__ dZ, long long P, int C, int ldd, int c0,
                                                  int act) {
  GRID_LOOP(id, P * C / V) {
    const RowCol r = row_col<V>(id, C);
    const Pack<float, V> d = ld_pack<float, V>(dY + r.p * ldd + c0 + r.c), z = ld_pack<float, V>(Z + id * V);
    Pack<float, V> o;
#pragma unroll
    for (int e = 0; e < V; ++e) o.e[e] = act ? d.e[e] * gelu_grad(z.e[e]) : d.e[e];
    st_pack(dZ + id * V, o);
  }
}

__global__ void k_f32_to_bf16(const float* __restrict__ x, bf16* __restrict__ y, long long n) {
  GRID_LOOP(id, n) y[id] = __float2bfloat16(x[id]);
}

// A layer's backward start: dZ = dY * act'(Z) in FP32 (for the column sums)
// and in BF16 (the operand of both gradient products) in one pass.
template <int V>
__global__ void __launch_bounds__(256) k_act_grad_both(const float* __restrict__ Z, const float* __restrict__ dY,
                                                       float* __restrict__ dZ, bf16* __restrict__ dZb, long long n,
                                                       int act) {
  GRID_LOOP(id, n / V) {
    Pack<float, V> d = ld_pack<float, V>(dY + id * V);
    if (act) {
      const Pack<float, V> z = ld_pack<float, V>(Z + id * V);
#pragma unroll
      for (int e = 0; e < V; ++e) d.e[e] = d.e[e] * gelu_grad(z.e[e]);
    }
    Pack<bf16, V> b;
#pragma unroll
    for (int e = 0; e < V; ++e) b.e[e] = __float2bfloat16(d.e[e]);
    st_pack(dZ + id * V, d);
    st_pack(dZb + id * V, b);
  }
}

// Column sums in a fixed order: 256 running sums per column, the t-th over the
// rows t, t + 256, ..., then a halving tree over them.  The running sums of
// all columns are independent chains, one thread each (k_colsum_rows: a warp
// reads 32 columns of a row, 16 rows of its chain in flight; one block per
// column, as before, left most of the GPU idle), the tree is a block per column.
__global__ void __launch_bounds__(256) k_colsum_rows(const float* __restrict__ dZ, float* __restrict__ part,
                                                     long long P, int C) {
  const int c = blockIdx.y * 32 + threadIdx.x, t = blockIdx.x * 8 + threadIdx.y;
  if (c >= C) return;
  constexpr int U = 16;
  float s = 0.f;
  long long p = t;
  for (; p + 256LL * (U - 1) < P; p += 256LL * U) {
    float x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = __ldg(dZ + (p + 256LL * u) * C + c);
#pragma unroll
    for (int u = 0; u < U; ++u) s += x[u];
  }
  for (; p < P; p += 256) s += dZ[p * C + c];
  part[t * C + c] = s;
}
__global__ void __launch_bounds__(256) k_colsum_tree(const float* __restrict__ part, float* __restrict__ db, int C) {
  __shared__ float sm[256];
  const int c = blockIdx.x;
  sm[threadIdx.x] = part[threadIdx.x * C + c];
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sm[threadIdx.x] += sm[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) db[c] = sm[0];
}

// The same sums without scratch, one block per column.
__global__ void k_colsum(const float* __restrict__ dZ, float* __restrict__ db, long long P, int C) {
  __shared__ float sm[256];
  const int c = blockIdx.x;
  float s = 0.f;
  for (long long p = threadIdx.x; p < P; p += blockDim.x) s += dZ[p * C + c];
  sm[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sm[threadIdx.x] += sm[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) db[c] = sm[0];
}

// 2 x 2 average pooling, [B][H][W][C] -> [B][H/2][W/2][C] (BF16).
template <int V>
__global__ void __launch_bounds__(256) k_pool(const bf16* __restrict__ X, bf16* __restrict__ Y, int B, int H, int W,
                                              int C) {
  const int h = H / 2, w = W / 2;
  GRID_LOOP(id, (long long)B * h * w * C / V) {
    const RowCol r = row_col<V>(id, C);
    const Pix x = pixel(r.p, h, w);
    const long long q = (x.b * H + 2 * x.y) * W + 2 * x.x;
    const Pack<bf16, V> a = ld_pack<bf16, V>(X + q * C + r.c), b = ld_pack<bf16, V>(X + (q + 1) * C + r.c),
                        c = ld_pack<bf16, V>(X + (q + W) * C + r.c), d = ld_pack<bf16, V>(X + (q + W + 1) * C + r.c);
    Pack<bf16, V> y;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const float s = __bfloat162float(a.e[e]) + __bfloat162float(b.e[e]) + __bfloat162float(c.e[e]) +
                      __bfloat162float(d.e[e]);
      y.e[e] = __float2bfloat16(0.25f * s);
    }
    st_pack(Y + id * V, y);
  }
}

// gradient of the pooling: dX[fine] += dY[coarse] / 4 (FP32, channel slice
// of the coarse rows)
template <int V>
__global__ void __launch_bounds__(256) k_pool_grad(const float* __restrict__ dY, float* __restrict__ dX, int B, int H,
                                                   int W, int C, int ldy, int c0) {
  GRID_LOOP(id, (long long)B * H * W * C / V) {
    const RowCol r = row_col<V>(id, C);
    const Pix x = pixel(r.p, H, W);
    const long long q = (x.b * (H / 2) + x.y / 2) * (W / 2) + x.x / 2;
    const Pack<float, V> d = ld_pack<float, V>(dY + q * ldy + c0 + r.c);
    Pack<float, V> o = ld_pack<float, V>(dX + id * V);
#pragma unroll
    for (int e = 0; e < V; ++e) o.e[e] += 0.25f * d.e[e];
    st_pack(dX + id * V, o);
  }
}

// nearest 2x upsampling of [B][h][w][C] into a channel slice of the fine
// rows (ldy)
template <int V>
__global__ void __launch_bounds__(256) k_up(const bf16* __restrict__ X, bf16* __restrict__ Y, int B, int h, int w,
                                            int C, int ldy, int c0) {
  const int H = 2 * h, W = 2 * w;
  GRID_LOOP(id, (long long)B * H * W * C / V) {
    const RowCol r = row_col<V>(id, C);
    const Pix x = pixel(r.p, H, W);
    const long long q = (x.b * h + x.y / 2) * w + x.x / 2;
    st_pack(Y + r.p * ldy + c0 + r.c, ld_pack<bf16, V>(X + q * C + r.c));
  }
}

// gradient of the upsampling: dX[coarse] = sum of its 4 fine pixels (fixed order)
template <int V>
__global__ void __launch_bounds__(256) k_up_grad(const float* __restrict__ dY, float* __restrict__ dX, int B, int h,
                                                 int w, int C, int ldy, int c0) {
  const int W = 2 * w;
  GRID_LOOP(id, (long long)B * h * w * C / V) {
    const RowCol r = row_col<V>(id, C);
    const Pix x = pixel(r.p, h, w);
    const float* q = dY + ((x.b * 2 * h + 2 * x.y) * W + 2 * x.x) * ldy + c0 + r.c;
    const Pack<float, V> a = ld_pack<float, V>(q), b = ld_pack<float, V>(q + ldy),
                         c = ld_pack<float, V>(q + (long long)W * ldy), d = ld_pack<float, V>(q + (long long)(W + 1) * ldy);
    Pack<float, V> o;
#pragma unroll
    for (int e = 0; e < V; ++e) o.e[e] = a.e[e] + b.e[e] + c.e[e] + d.e[e];
    st_pack(dX + id * V, o);
  }
}

// copy a BF16 [P][C] block into a channel slice of rows of ldy
template <int V>
__global__ void __launch_bounds__(256) k_copy_slice(const bf16* __restrict__ X, bf16* __restrict__ Y, long long P,
                                                    int C, int ldy, int c0) {
  GRID_LOOP(id, P * C / V) {
    const RowCol r = row_col<V>(id, C);
    st_pack(Y + r.p * ldy + c0 + r.c, ld_pack<bf16, V>(X + id * V));
  }
}

// dX += a channel slice of dY (FP32)
template <int V>
__global__ void __launch_bounds__(256) k_add_slice(const float* __restrict__ dY, float* __restrict__ dX, long long P,
                                                   int C, int ldy, int c0) {
  GRID_LOOP(id, P * C / V) {
    const RowCol r = row_col<V>(id, C);
    const Pack<float, V> d = ld_pack<float, V>(dY + r.p * ldy + c0 + r.c);
    Pack<float, V> o = ld_pack<float, V>(dX + id * V);
#pragma unroll
    for (int e = 0; e < V; ++e) o.e[e] += d.e[e];
    st_pack(dX + id * V, o);
  }
}

// Masked mean squared error over [P][C] (mask per pixel): per-block
// partial sums in a fixed order; gradient 2 (y - t) mask / count.
__global__ void k_mse(const float* __restrict__ Y, const float* __restrict__ T, const float* __restrict__ mask,
                      float* __restrict__ dY, float* __restrict__ partial, long long P, int C, float inv_count) {
  __shared__ float sm[256];
  float s = 0.f;
  for (long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x; id < P * C;
       id += (long long)gridDim.x * blockDim.x) {
    const float m = mask[id / C];
    const float e = (Y[id] - T[id]) * m;
    dY[id] = 2.f * e * inv_count;
    s += e * e;
  }
  sm[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sm[threadIdx.x] += sm[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sm[0] * inv_count;
}

// Adam on FP32 master weights; the BF16 GEMM copy W[Cout][Kp] (k < K real,
// the padding stays zero) is refreshed in the same pass.
__global__ void k_adam(float* __restrict__ w, const float* __restrict__ grad, float* __restrict__ m1,
                       float* __restrict__ m2, bf16* __restrict__ wb, long long n, int K, int Kp, float lr,
                       float b1, float b2, float eps, float c1, float c2) {
  GRID_LOOP(id, n) {
    const float gr = grad[id];
    const float a = b1 * m1[id] + (1.f - b1) * gr;
    const float b = b2 * m2[id] + (1.f - b2) * gr * gr;
    m1[id] = a;
    m2[id] = b;
    const float x = w[id] - lr * (a * c1) / (sqrtf(b * c2) + eps);
    w[id] = x;
    if (wb) {
      const long long r = id / K;
      const int k = (int)(id % K);
      wb[r * Kp + k] = __float2bfloat16(x);
    }
  }
}

// gradient of a padded BF16 GEMM weight [Cout][Kp] back to [Cout][K]
__global__ void k_unpad(const float* __restrict__ src, float* __restrict__ dst, long long rows, int K, int Kp) {
  GRID_LOOP(id, rows * K) {
    const long long r = id / K;
    const int k = (int)(id % K);
    dst[id] = src[r * Kp + k];
  }
}

inline bool aligned(const void* p, unsigned n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; }
// whether the channel-slice kernels may move 16 bytes a thread: 8 BF16 or 4
// FP32 channels
inline bool vec8(int C, int ld, int c0, const void* a, const void* b) {
  return C % 8 == 0 && ld % 8 == 0 && c0 % 8 == 0 && aligned(a, 16) && aligned(b, 16);
}
inline bool vec4(int C, int ld, int c0, const void* a, const void* b) {
  return C % 4 == 0 && ld % 4 == 0 && c0 % 4 == 0 && aligned(a, 16) && aligned(b, 16);
}

inline unsigned grid_for(long long n) {
  long long g = (n + 255) / 256;
  if (g > 65535LL * 16) g = 65535LL * 16;
  return (unsigned)(g < 1 ? 1 : g);
}

// ---------------------------------------------------------------------
// The same GEMM on the 5th-generation tensor cores (tcgen05): one CTA of
// four warps per 128 x 64 tile of C, its FP32 accumulator in tensor memory
// (64 of the SM's 512 TMEM columns, lane = row), the operands staged in
// shared memory in the K-major no-swizzle core-matrix layout (8 rows x 16
// bytes per 128-byte core matrix) that the UMMA shared-memory descriptor
// describes, two stages deep: while the tensor core multiplies one 64-deep
// K slice the threads load the next.  One thread issues the four K = 16
// tcgen05.mma of a slice and commits them to the stage's mbarrier; the
// stage is refilled once that barrier completes.  The epilogue reads the
// accumulator with tcgen05.ld (warp w: rows 32w..32w+31) and adds the bias
// (and C) through shared memory, so that stores run along rows.  Every
// wait is bounded: past the limit the kernel raises g_tc_err, stops
// issuing, frees its tensor memory and returns.
// ---------------------------------------------------------------------
constexpr int TC_BM = 128, TC_BK = 64;
constexpr int TC_A_BYTES = TC_BM * TC_BK * 2;
// BN = 64, 32 for the products with at most 32 output columns, or 128
template <int BN>
constexpr int tc_stage_bytes() { return TC_A_BYTES + BN * TC_BK * 2; }  // 20, 24 or 32 KB

__device__ int g_tc_err = 0;  // a wait of k_gemm_tc ran out (read and cleared by bpnet_gemm_status)

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// UMMA shared-memory descriptor, K-major, no swizzle: start address, leading
// byte offset (between the two 16-byte K chunks of one K = 16 step), stride
// byte offset (between 8-row groups), version 1, base offset 0, layout 0.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), A
// and B BF16 (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4
// at bit 24.
template <int BN>
constexpr uint32_t tc_idesc() {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (int i = 0; i < (1 << 24); ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  atomicExch(&g_tc_err, 1);
  return false;
}

// Split K: CTA z of the grid covers K slices [z * kchunk, min(K, (z + 1) *
// kchunk)) (kchunk a multiple of TC_BK) and writes its partial product to
// C + z * cstride; gridDim.z = 1 is the whole K with bias and accumulation.
template <int BN>
__global__ void __launch_bounds__(128) k_gemm_tc(const bf16* __restrict__ A, const bf16* __restrict__ B,
                                                 float* __restrict__ C, const float* __restrict__ bias,
                                                 int M, int N, int K, int lda, int ldb, int ldc,
                                                 int accum, int kchunk, long long cstride) {
  extern __shared__ __align__(1024) uint8_t tc_smem[];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5;
  constexpr int STAGE = tc_stage_bytes<BN>();
  const int m0 = blockIdx.y * TC_BM, n0 = blockIdx.x * BN;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar[0])));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar[1])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const int kbeg = blockIdx.z * kchunk, kend = min(K, kbeg + kchunk);
  C += (size_t)blockIdx.z * cstride;
  const int nk = (kend - kbeg + TC_BK - 1) / TC_BK;
  bool ok = true;
  for (int it = 0; it < nk; ++it) {
    const int st = it & 1;
    uint8_t* As = tc_smem + st * STAGE;
    uint8_t* Bs = As + TC_A_BYTES;
    if (it >= 2) ok = mbar_wait(smem_u32(&bar[st]), ((it - 2) >> 1) & 1);  // the stage's last slice is done
    if (!__syncthreads_and(ok)) {
      ok = false;
      break;
    }
    const int k0 = kbeg + it * TC_BK;
    for (int c = tid; c < TC_BM * 8; c += 128) {  // 128 rows x 8 chunks of 8 K elements
      const int r = c >> 3, kc = c & 7, gm = m0 + r, gk = k0 + kc * 8;
      uint4 val = make_uint4(0u, 0u, 0u, 0u);
      if (gm < M && gk < kend) val = __ldg(reinterpret_cast<const uint4*>(A + (size_t)gm * lda + gk));
      *reinterpret_cast<uint4*>(As + (kc * (TC_BM / 8) + (r >> 3)) * 128 + (r & 7) * 16) = val;
    }
    for (int c = tid; c < BN * 8; c += 128) {
      const int r = c >> 3, kc = c & 7, gn = n0 + r, gk = k0 + kc * 8;
      uint4 val = make_uint4(0u, 0u, 0u, 0u);
      if (gn < N && gk < kend) val = __ldg(reinterpret_cast<const uint4*>(B + (size_t)gn * ldb + gk));
      *reinterpret_cast<uint4*>(Bs + (kc * (BN / 8) + (r >> 3)) * 128 + (r & 7) * 16) = val;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads through the async proxy
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int s = 0; s < TC_BK / 16; ++s) {
        if (k0 + 16 * s >= kend) break;
        const uint64_t ad = umma_desc(smem_u32(As) + 2 * s * (TC_BM / 8) * 128, (TC_BM / 8) * 128, 128);
        const uint64_t bd = umma_desc(smem_u32(Bs) + 2 * s * (BN / 8) * 128, (BN / 8) * 128, 128);
        const uint32_t acc = (it > 0 || s > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
            ::"r"(tmem), "l"(ad), "l"(bd), "r"(tc_idesc<BN>()), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&bar[st]))
                   : "memory");
    }
  }
  // the last commit completes after every multiply of the tile (the host
  // never launches an empty K range)
  if (ok) ok = mbar_wait(smem_u32(&bar[(nk - 1) & 1]), ((nk - 1) >> 1) & 1);
  ok = __syncthreads_and(ok);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) {
    // warp w holds rows 32w..32w+31 of the tile (one row per lane); each
    // 32 x 32 block goes through shared memory (the stages are free now)
    // so that a store instruction writes 32 consecutive columns of a row
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // after the tensor core's reads of the stages
    float* T = reinterpret_cast<float*>(tc_smem) + warp * (32 * 33);
    const int lane = tid & 31;
#pragma unroll
    for (int c0 = 0; c0 < BN; c0 += 32) {
      uint32_t v[32];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
          "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
            "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
            "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
            "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
            "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
          : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; ++j) T[lane * 33 + j] = __uint_as_float(v[j]);
      __syncwarp();
      const int col = n0 + c0 + lane;
      if (col < N) {
        const float bc = bias ? bias[col] : 0.f;
        for (int r = 0; r < 32; ++r) {
          const int row = m0 + warp * 32 + r;
          if (row >= M) break;
          float* dst = C + (size_t)row * ldc + col;
          float x = T[r * 33 + lane] + bc;
          if (accum) x += *dst;
          *dst = x;
        }
      }
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN));
}

// ---------------------------------------------------------------------
// The same product with its operands brought in by the Tensor Memory
// Accelerator: a four-stage ring of shared-memory slices that complete on the
// stage's "full" mbarrier.  One thread issues the loads and the tcgen05.mma
// of every slice; a stage is refilled with the slice four ahead once the
// tensor core's commit for it has arrived on the stage's "done" mbarrier, so
// up to four slices of loads are in flight while the tensor core works.
// Operands lie in shared memory with the 128-byte swizzle, so that a slice is
// one box of 128-byte rows per operand (16-byte boxes of the unswizzled
// layout left the copy engine as the limit: 131,072 x 64 x 576 took 83 us, now
// 47; 32 x 288 x 524,288 362 us, now 148).  Either operand is K-major
// (element (m, k) at [m * ld + k]: a box of 64 K elements by the tile's rows)
// or MN-major ([k * ld + m]: boxes of 64 rows of the product by 64 K), which
// takes the gradient products' operands as the other passes left them, without
// transposed copies.  Out-of-range rows and K read as zero (the tensor maps'
// bounds).  Epilogue as k_gemm_tc; ACT also or instead writes the activation
// of the result in BF16.  Every wait is bounded; on a timeout the issuing
// thread waits (bounded) for its copies and its last multiply in flight,
// raises g_tc_err, and the CTA frees its tensor memory and returns.  Loads
// only: no TMA store, no multicast.
// ---------------------------------------------------------------------
constexpr int TM_STAGES = 4;

// bytes of an operand's slice: rows x 64 K elements; MN-major in whole boxes of 64
template <int ROWS, bool MN>
constexpr int tm_operand_bytes() { return (MN ? (ROWS + 63) / 64 * 64 : ROWS) * TC_BK * 2; }
template <int BN, bool AMN, bool BMN>
constexpr int tm_stage_bytes() { return tm_operand_bytes<TC_BM, AMN>() + tm_operand_bytes<BN, BMN>(); }
template <int BN, bool AMN, bool BMN>
constexpr int tm_smem_bytes() { return TM_STAGES * tm_stage_bytes<BN, AMN, BMN>() + 1024; }  // + room to align the ring

// UMMA shared-memory descriptor with the 128-byte swizzle.  K-major: 8-row
// groups 1024 bytes apart (the leading offset is not used); MN-major: groups
// of 8 K rows 1024 bytes apart, boxes of 64 rows of the product 8192.
template <bool MN>
__device__ __forceinline__ uint64_t umma_desc_sw(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(MN ? 8192 >> 4 : 1) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %0;" ::"r"(bytes), "r"(bar) : "memory");
}

// A box of the 2-D tensor map at (x = K element, y = row) into shared
// memory; x is always a multiple of 8 (16 bytes).
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
          "r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}

template <int BN, bool AMN, bool BMN>
__global__ void __launch_bounds__(128) k_gemm_tma(const __grid_constant__ CUtensorMap tmA,
                                                  const __grid_constant__ CUtensorMap tmB, float* __restrict__ C,
                                                  const float* __restrict__ bias, int M, int N, int K, int ldc,
                                                  int accum, int kchunk, long long cstride, bf16* __restrict__ Y,
                                                  int act) {
  extern __shared__ __align__(1024) uint8_t tc_smem[];
  __shared__ __align__(8) uint64_t full[TM_STAGES], done[TM_STAGES];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_ok;
  constexpr int STAGE = tm_stage_bytes<BN, AMN, BMN>(), A_BYTES = tm_operand_bytes<TC_BM, AMN>();
  const int tid = threadIdx.x, warp = tid >> 5;
  const int m0 = blockIdx.y * TC_BM, n0 = blockIdx.x * BN;
  const int kbeg = blockIdx.z * kchunk, kend = min(K, kbeg + kchunk);
  if (C) C += (size_t)blockIdx.z * cstride;
  const int nk = (kend - kbeg + TC_BK - 1) / TC_BK;
  // the ring starts on a 1024-byte boundary, the swizzle's period
  const uint32_t ring = (smem_u32(tc_smem) + 1023u) & ~1023u;
  uint8_t* ring_ptr = tc_smem + (ring - smem_u32(tc_smem));
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int st = 0; st < TM_STAGES; ++st) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[st])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&done[st])));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_ok = 1;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  if (tid == 0) {
    // MN-major: boxes past the operand's last row are left out (their rows of
    // the product are not stored)
    const int boxa = AMN ? min(TC_BM / 64, (M - m0 + 63) / 64) : 1;
    const int boxb = BMN ? min((BN + 63) / 64, (N - n0 + 63) / 64) : 1;
    const uint32_t bytes = (uint32_t)((AMN ? boxa * 8192 : A_BYTES) + (BMN ? boxb * 8192 : STAGE - A_BYTES));
    auto issue = [&](int j) {  // slice j into stage j % TM_STAGES
      const int st = j % TM_STAGES;
      const uint32_t a = ring + st * STAGE, b = a + A_BYTES, bar = smem_u32(&full[st]);
      mbar_expect_tx(bar, bytes);
      const int k0 = kbeg + j * TC_BK;
      if (AMN) {
        for (int x = 0; x < boxa; ++x) tma_load_2d(a + x * 8192, &tmA, m0 + 64 * x, k0, bar);
      } else {
        tma_load_2d(a, &tmA, k0, m0, bar);
      }
      if (BMN) {
        for (int x = 0; x < boxb; ++x) tma_load_2d(b + x * 8192, &tmB, n0 + 64 * x, k0, bar);
      } else {
        tma_load_2d(b, &tmB, k0, n0, bar);
      }
    };
    bool ok = true;
    int issued = 0, it = 0, last_mma = -1;
    for (; issued < nk && issued < TM_STAGES; ++issued) issue(issued);
    for (; it < nk; ++it) {
      const int st = it % TM_STAGES;
      if (!mbar_wait(smem_u32(&full[st]), (it / TM_STAGES) & 1)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int k0 = kbeg + it * TC_BK;
      const uint32_t a = ring + st * STAGE, b = a + A_BYTES;
#pragma unroll
      for (int s = 0; s < TC_BK / 16; ++s) {
        if (k0 + 16 * s >= kend) break;
        // 16 K elements on: 32 bytes along a K-major row, two groups of 8 K rows MN-major
        const uint64_t ad = umma_desc_sw<AMN>(a + s * (AMN ? 2048 : 32));
        const uint64_t bd = umma_desc_sw<BMN>(b + s * (BMN ? 2048 : 32));
        const uint32_t acc = (it > 0 || s > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(tc_idesc<BN>() | (AMN ? 1u << 15 : 0u) | (BMN ? 1u << 16 : 0u)), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&done[st]))
                   : "memory");
      last_mma = it;
      if (issued < nk) {  // the stage takes the slice TM_STAGES ahead once this multiply has read it
        if (!mbar_wait(smem_u32(&done[st]), (it / TM_STAGES) & 1)) {
          ok = false;
          ++it;
          break;
        }
        issue(issued);
        ++issued;
      }
    }
    if (ok && last_mma >= 0)  // the last commit completes after every multiply of the tile
      ok = mbar_wait(smem_u32(&done[last_mma % TM_STAGES]), (last_mma / TM_STAGES) & 1);
    if (!ok) {  // no copy and no multiply may still be in flight when the CTA exits
      for (int j = it; j < issued; ++j) mbar_wait(smem_u32(&full[j % TM_STAGES]), (j / TM_STAGES) & 1);
      if (last_mma >= 0) mbar_wait(smem_u32(&done[last_mma % TM_STAGES]), (last_mma / TM_STAGES) & 1);
      s_ok = 0;
    }
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (s_ok) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // after the copies and the tensor core's reads
    float* T = reinterpret_cast<float*>(ring_ptr) + warp * (32 * 33);
    const int lane = tid & 31;
#pragma unroll
    for (int c0 = 0; c0 < BN; c0 += 32) {
      uint32_t v[32];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
          "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
            "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
            "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
            "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
            "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
          : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; ++j) T[lane * 33 + j] = __uint_as_float(v[j]);
      __syncwarp();
      const int col = n0 + c0 + lane;
      if (col < N) {
        const float bc = bias ? bias[col] : 0.f;
        for (int r = 0; r < 32; ++r) {
          const int row = m0 + warp * 32 + r;
          if (row >= M) break;
          float x = T[r * 33 + lane] + bc;
          if (C) {
            float* dst = C + (size_t)row * ldc + col;
            if (accum) x += *dst;
            *dst = x;
          }
          if (Y) Y[(size_t)row * ldc + col] = __float2bfloat16(act ? gelu(x) : x);
        }
      }
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN));
}

PFN_cuTensorMapEncodeTiled_v12000 tma_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 enc = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  }();
  return enc;
}
// The 2-D tensor map of a row-major BF16 operand, inner x outer elements with
// rows of ld, in boxes of 64 inner elements (128 bytes, swizzled) by box_outer;
// false where the driver has no encoder or refuses the operand (address or
// stride not 16-byte aligned).
bool tma_map(CUtensorMap* map, const void* ptr, int inner, int outer, int ld, int box_outer) {
  const auto enc = tma_encoder();
  if (!enc || (reinterpret_cast<uintptr_t>(ptr) & 15) || ((size_t)ld * 2) % 16) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_outer};
  const cuuint32_t es[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// k_dgrad3's map, 64-byte swizzle: the weights [cout][Kp] in boxes of 32
// columns by `rows` rows.
bool dgrad_map(CUtensorMap* mw, const void* w, int C, int Kp, int K, int rows) {
  const auto enc = tma_encoder();
  if (!enc || (reinterpret_cast<uintptr_t>(w) & 15) || Kp % 8) return false;
  const cuuint64_t dw[2] = {(cuuint64_t)K, (cuuint64_t)C}, sw[1] = {(cuuint64_t)Kp * 2};
  const cuuint32_t bx[2] = {32, (cuuint32_t)rows}, e2[2] = {1, 1};
  return enc(mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(w), dw, sw, bx, e2,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---------------------------------------------------------------------
// Input gradient of a 3 x 3 convolution: dX[p][c] = sum over taps, in tap
// order, of (sum over o of dZ[q][o] w[o][tap * cin + c]), q the pixel whose
// tap lands on p.
//
// As a product over all taps and a gather, its FP32 result (9 cin columns a
// pixel) is written to memory and read back: 151 MB for 131,072 pixels of 32
// channels.  Here a CTA takes 8 x 16 pixels by 32 NB input channels.  It
// copies dZ's 10 x 18 pixels around them once, as planes of 8 channels (16
// bytes a pixel): in that layout a tap's 128 shifted pixels are the same
// operand from another start address (8 rows of 16 bytes lie together, the
// next 8 one row of the copy on), wrapped or zero at the border as copied.
// The weights, MN-major as they lie, follow in slices of 32 or 64 output channels.
// For every tap the tensor core forms the tap's product in one of BUFS
// accumulators while four warps add the last tap's to their sums in registers.
// Same products in the same order as before: the result is bitwise that of
// the product and the gather.  A fifth warp issues the multiplies, a sixth the copies.
// Waits bounded as in k_gemm_tma.
// Eight 128 x 128 grids with the L2 cold, product and gather -> here: 32 to 32
// channels 132 -> 32 us, 96 to 32 431 -> 64; 64 x 64, 192 to 64 177 -> 38;
// 32 x 32, 384 to 128 99 -> 28.  Its bytes take 4 to 9 us: it is bound by the
// row of waits in a CTA (copy, nine taps, store), hidden by 2 to 4 CTAs an SM.
// ---------------------------------------------------------------------
constexpr int DG_W = 8, DG_H = 16, DG_PLANE = (DG_W + 2) * (DG_H + 2) * 16, DG_RING = 16384, DG_MAX_COUT = 256;
constexpr int DG_BUFS = 2;
constexpr int dg_cols(int nb) { return nb == 3 ? 256 : 64 * nb; }  // accumulator columns, a power of two
// the ring of weights, dZ's planes; at least what keeps the CTAs of an SM
// within its 512 accumulator columns
constexpr int dg_smem_bytes(int nb, int cout) {
  const int n = DG_RING * nb + cout / 8 * DG_PLANE + 1024, least = nb == 3 ? 80 * 1024 : nb == 2 ? 56 * 1024 : 0;
  return n > least ? n : least;
}

// 64-byte swizzle, MN-major: groups of 8 K rows 512 bytes apart, groups of 32
// columns `box`
__device__ __forceinline__ uint64_t umma_desc_sw64(uint32_t addr, uint32_t box) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(box >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
// no swizzle, K-major: 8 channels on = the next plane, 8 rows on = the next row of the copy
__device__ __forceinline__ uint64_t umma_desc_planes(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(DG_PLANE >> 4) << 16) |
         ((uint64_t)((DG_W + 2) * 16 >> 4) << 32) | ((uint64_t)1 << 46);
}

// KR: output channels of a slice of weights; the ring holds DG_RING bytes per 32 columns.
template <int NB, int KR>
__global__ void __launch_bounds__(192, NB == 1 ? 4 : NB == 2 ? 3 : 2) k_dgrad3(const __grid_constant__ CUtensorMap tmW, const bf16* __restrict__ dZ,
                                                float* __restrict__ dX, int H, int W, int cin, int cout,
                                                int periodic) {
  constexpr int BUFS = DG_BUFS, COLS = dg_cols(NB), BOX = KR * 64, STAGE = NB * BOX, STAGES = DG_RING / BOX;
  extern __shared__ __align__(1024) uint8_t tc_smem[];
  __shared__ __align__(8) uint64_t full[STAGES], done[STAGES], tap_done[BUFS], tap_free[BUFS];
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tx = (W + DG_W - 1) / DG_W;
  const int x0 = ((int)blockIdx.x % tx) * DG_W, y0 = ((int)blockIdx.x / tx) * DG_H, b = blockIdx.y;
  const int c0 = blockIdx.z * (32 * NB), ns = cout / KR;
  const uint32_t ring = (smem_u32(tc_smem) + 1023u) & ~1023u, planes = ring + STAGES * STAGE;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 128) {
    for (int i = 0; i < STAGES; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&done[i])));
    }
    for (int i = 0; i < BUFS; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&tap_done[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(smem_u32(&tap_free[i])));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp < 4) {
    // a pixel outside the grid is its wrapped one or zeros
    const int nc = cout >> 3;
    for (int i = tid; i < (DG_W + 2) * (DG_H + 2) * nc; i += 128) {
      const int px = i / nc, c8 = i - px * nc, hy = px / (DG_W + 2);
      int y = y0 + hy - 1, x = x0 + (px - hy * (DG_W + 2)) - 1;
      if (periodic) {
        y = y < 0 ? H - 1 : y == H ? 0 : y;
        x = x < 0 ? W - 1 : x == W ? 0 : x;
      }
      const bool in = y >= 0 && y < H && x >= 0 && x < W;
      const bf16* src = in ? dZ + (((size_t)b * H + y) * W + x) * cout + c8 * 8 : dZ;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(planes + c8 * DG_PLANE + px * 16), "l"(src),
                   "r"(in ? 16 : 0)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  bool ok = true;
  float s[32 * NB];
  if (warp == 5) {  // the copies of the weights
    if (lane == 0) {
      int st = 0, n = 0;  // slice n of stage st; its stage's use before ended at parity `par`
      uint32_t par = 1;
      for (int tap = 0; ok && tap < 9; ++tap)
        for (int o0 = 0; o0 < cout; o0 += KR, ++n) {
          const uint32_t bar = smem_u32(&full[st]);
          if (n >= STAGES && !(ok = mbar_wait(smem_u32(&done[st]), par))) break;
          mbar_expect_tx(bar, STAGE);
#pragma unroll
          for (int i = 0; i < NB; ++i)
            tma_load_2d(ring + st * STAGE + i * BOX, &tmW, tap * cin + c0 + 32 * i, o0, bar);
          if (++st == STAGES) {
            st = 0;
            par ^= 1;
          }
        }
      // no copy may still be in flight when the CTA exits: the last one of each stage issued
      const int last = n < STAGES ? n : STAGES;
      for (int i = 0; i < last; ++i) {
        const int j = n - 1 - i;
        mbar_wait(smem_u32(&full[j % STAGES]), (j / STAGES) & 1);
      }
    }
  } else if (warp == 4) {  // the multiplies
    if (lane == 0) {
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(32 * NB >> 3) << 17) |
                                 ((uint32_t)(128 >> 4) << 24);
      const uint64_t a0 = umma_desc_planes(planes), b0 = umma_desc_sw64(ring, BOX);
      int st = 0, buf = 0, last = -1;
      uint32_t par = 0, free_par = 1;  // (parities of full[st] and, from tap BUFS on, tap_free[buf])
      for (int tap = 0; ok && tap < 9; ++tap) {
        // the accumulator's last tap has been read
        if (tap >= BUFS && !(ok = mbar_wait(smem_u32(&tap_free[buf]), free_par))) break;
        // the tap (ty, tx) of the pixel (y - ty, x - tx) lands on (y, x); the copy
        // starts at (y0 - 1, x0 - 1).  Descriptors count 16 bytes.
        const uint64_t at = a0 + (uint32_t)((1 - (tap / 3 - 1)) * (DG_W + 2) + 1 - (tap % 3 - 1));
        for (int sl = 0; sl < ns; ++sl) {
          if (!(ok = mbar_wait(smem_u32(&full[st]), par))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int k = 0; k < KR / 16; ++k) {  // 16 output channels: two planes, two groups of 8 rows of w
            const uint64_t ad = at + (uint32_t)((sl * (KR / 8) + k * 2) * (DG_PLANE / 16)),
                           bd = b0 + (uint32_t)((st * STAGE + k * 1024) / 16);
            const uint32_t acc = (sl > 0 || k > 0) ? 1u : 0u;
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(tmem +
                                                                                                      32 * NB * buf),
                "l"(ad), "l"(bd), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                           smem_u32(&done[st]))
                       : "memory");
          last = (st << 1) | (int)par;  // (a stage's uses of full and done have the same parity)
          if (++st == STAGES) {
            st = 0;
            par ^= 1;
          }
        }
        if (!ok) break;
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&tap_done[buf]))
                     : "memory");
        if (++buf == BUFS) {
          buf = 0;
          free_par ^= 1;
        }
      }
      // no multiply may still be in flight when the CTA exits
      if (last >= 0 && !mbar_wait(smem_u32(&done[last >> 1]), last & 1)) ok = false;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32 * NB; ++j) s[j] = 0.f;
    const int m = warp * 32 + lane, y = y0 + m / DG_W, x = x0 + m % DG_W;
    for (int tap = 0; tap < 9; ++tap) {
      const int buf = tap % BUFS;
      // one lane asks: 128 of them asking keep shared memory from the fifth warp
      if (lane == 0) ok = mbar_wait(smem_u32(&tap_done[buf]), (tap / BUFS) & 1);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // a pixel outside the grid adds nothing, whatever the weights are
      const int yq = y - (tap / 3 - 1), xq = x - (tap % 3 - 1);
      const bool in = periodic || (yq >= 0 && yq < H && xq >= 0 && xq < W);
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        uint32_t v[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
            "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
              "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
              "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
              "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
            : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(32 * NB * buf + 32 * n)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (n == NB - 1) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tap_free[buf])) : "memory");
        }
        if (in) {
#pragma unroll
          for (int j = 0; j < 32; ++j) s[32 * n + j] += __uint_as_float(v[j]);
        }
      }
    }
  }
  ok = __syncthreads_and(ok);
  if (ok && warp < 4) {
    // warp w: pixels 32w .. 32w + 31 of the rectangle, through the ring's and
    // the planes' memory so that a store writes one pixel's 32 channels
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    float* T = reinterpret_cast<float*>(tc_smem + (ring - smem_u32(tc_smem))) + warp * (32 * 33);
#pragma unroll
    for (int n = 0; n < NB; ++n) {
#pragma unroll
      for (int j = 0; j < 32; ++j) T[lane * 33 + j] = s[32 * n + j];
      __syncwarp();
#pragma unroll 4
      for (int r = 0; r < 32; ++r) {
        const int m = warp * 32 + r, y = y0 + m / DG_W, x = x0 + m % DG_W;
        if (y < H && x < W) dX[(((size_t)b * H + y) * W + x) * cin + c0 + 32 * n + lane] = T[r * 33 + lane];
      }
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
}

template <int NB, int KR>
int launch_dgrad3(const void* dZ, const void* w, float* dX, int B, int H, int W, int cin, int cout, int Kp,
                  int periodic, cudaStream_t st) {
  static_assert(4 * 32 * 33 * 4 <= DG_RING + 4 * DG_PLANE, "room for the result's transposition");
  static const bool ok = cudaFuncSetAttribute(k_dgrad3<NB, KR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              dg_smem_bytes(NB, DG_MAX_COUT)) == cudaSuccess;
  CUtensorMap mw;
  if (!ok) return 6;
  if (!dgrad_map(&mw, w, cout, Kp, 9 * cin, KR)) return 10;
  const dim3 grid((unsigned)(((W + DG_W - 1) / DG_W) * ((H + DG_H - 1) / DG_H)), B, cin / (32 * NB));
  k_dgrad3<NB, KR><<<grid, 192, dg_smem_bytes(NB, cout), st>>>(mw, (const bf16*)dZ, dX, H, W, cin, cout, periodic);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

// C[r][c] = sum over z of part[z][r][c] in z order (+ bias) (+ C): the
// split-K partial products, summed deterministically.
__global__ void k_splitk_sum(const float* __restrict__ part, int S, long long cstride, float* __restrict__ C,
                             const float* __restrict__ bias, int M, int N, int ldc, int accum) {
  GRID_LOOP(id, (long long)M * N) {
    const long long r = id / N;
    const int c = (int)(id % N);
    float v = 0.f;
    for (int z = 0; z < S; ++z) v += part[z * cstride + id];
    if (bias) v += bias[c];
    float* dst = C + r * ldc + c;
    if (accum) v += *dst;
    *dst = v;
  }
}

// Grow-only scratch of the split-K partial products, one per device (the
// current one); a buffer is replaced only after the device has finished
// with it.
float* splitk_scratch(size_t n) {
  static std::mutex mu;
  static std::map<int, std::pair<float*, size_t>> bufs;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  auto& b = bufs[dev];
  if (n > b.second) {
    if (b.first) {
      cudaDeviceSynchronize();
      cudaFree(b.first);
    }
    b = {nullptr, 0};
    if (cudaMalloc(&b.first, n * sizeof(float)) != cudaSuccess) return nullptr;
    b.second = n;
  }
  return b.first;
}

// One product on the TMA-fed kernel.
template <int W, bool AMN, bool BMN>
bool launch_tma(const CUtensorMap& ma, const CUtensorMap& mb, dim3 grid, cudaStream_t st, float* out,
                const float* bout, int M, int N, int K, int ldo, int acc, int kchunk, long long cs, bf16* Y, int act) {
  static const bool ok = cudaFuncSetAttribute(k_gemm_tma<W, AMN, BMN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              tm_smem_bytes<W, AMN, BMN>()) == cudaSuccess;
  if (!ok) return false;
  k_gemm_tma<W, AMN, BMN><<<grid, 128, tm_smem_bytes<W, AMN, BMN>(), st>>>(ma, mb, out, bout, M, N, K, ldo, acc,
                                                                           kchunk, cs, Y, act);
  return true;
}
template <int W>
bool launch_tma_major(int a_mn, int b_mn, const CUtensorMap& ma, const CUtensorMap& mb, dim3 grid, cudaStream_t st,
                      float* out, const float* bout, int M, int N, int K, int ldo, int acc, int kchunk, long long cs,
                      bf16* Y, int act) {
  if (a_mn && b_mn) return launch_tma<W, true, true>(ma, mb, grid, st, out, bout, M, N, K, ldo, acc, kchunk, cs, Y, act);
  if (a_mn) return launch_tma<W, true, false>(ma, mb, grid, st, out, bout, M, N, K, ldo, acc, kchunk, cs, Y, act);
  if (b_mn) return launch_tma<W, false, true>(ma, mb, grid, st, out, bout, M, N, K, ldo, acc, kchunk, cs, Y, act);
  return launch_tma<W, false, false>(ma, mb, grid, st, out, bout, M, N, K, ldo, acc, kchunk, cs, Y, act);
}
template <int W>
bool launch_tc(dim3 grid, cudaStream_t st, const bf16* A, const bf16* B, float* out, const float* bout, int M, int N,
               int K, int lda, int ldb, int ldo, int acc, int kchunk, long long cs) {
  static const bool ok = cudaFuncSetAttribute(k_gemm_tc<W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              2 * tc_stage_bytes<W>()) == cudaSuccess;
  if (!ok) return false;
  k_gemm_tc<W><<<grid, 128, 2 * tc_stage_bytes<W>(), st>>>(A, B, out, bout, M, N, K, lda, ldb, ldo, acc, kchunk, cs);
  return true;
}

// How a product is cut: tile width bn, split S of K in chunks of kchunk.
struct GemmCut {
  int bn, S, kchunk, gx, gy;
};
GemmCut cut_gemm(int M, int N, int K) {
  GemmCut c;
  // tile width: 32 for at most 32 columns (no MMA work on padding); 128
  // for widths that are not a multiple of 64 where it pads no more than 64
  // does (96: one tile instead of 64 + 32, A read once); else 64 (a
  // multiple of 64 keeps twice the CTAs: 128 x 128 tiles measured slower at
  // N = 128 and 1152)
  c.bn = 64;
  if (N <= 32)
    c.bn = 32;
  else if (N % 64 != 0 && (N + 127) / 128 * 128 <= (N + 63) / 64 * 64)
    c.bn = 128;
  const int nslices = (K + TC_BK - 1) / TC_BK;
  c.gx = (N + c.bn - 1) / c.bn;
  c.gy = (M + TC_BM - 1) / TC_BM;
  c.S = 1;
  c.kchunk = nslices * TC_BK;
  // few output tiles and a long K (the weight gradients, K = pixels): split
  // along K over enough CTAs to fill the GPU
  if (c.gx * c.gy < 296 && nslices >= 64)
    c.S = std::min((296 + c.gx * c.gy - 1) / (c.gx * c.gy), nslices / 16);
  if (c.S > 1) {
    c.kchunk = (nslices + c.S - 1) / c.S * TC_BK;
    c.S = (K + c.kchunk - 1) / c.kchunk;  // no empty chunk
  }
  return c;
}

// C = A B^T (+ bias) (+ C) on the tensor cores: tma = 1 the TMA-fed kernel
// (10 where its operands cannot be mapped), 0 the register-staged one (both
// operands K-major).  a_mn, b_mn: the operand is MN-major (element (m, k) at
// [k * ld + m]).  Y (not with a split K or accumulation): act of the result in
// BF16, rows of ldc; C may then be null.
int tensor_gemm(int tma, int a_mn, int b_mn, const bf16* A, const bf16* B, float* C, const float* bias, int M, int N,
                int K, int lda, int ldb, int ldc, int accum, bf16* Y, int act, cudaStream_t st) {
  const GemmCut c = cut_gemm(M, N, K);
  if (Y && (c.S > 1 || accum)) return 10;
  CUtensorMap ma, mb;
  if (tma &&
      !(a_mn ? tma_map(&ma, A, M, K, lda, 64) : tma_map(&ma, A, K, M, lda, TC_BM)))
    return 10;
  if (tma && !(b_mn ? tma_map(&mb, B, N, K, ldb, 64) : tma_map(&mb, B, K, N, ldb, c.bn))) return 10;
  float* out = C;
  const float* bout = bias;
  int ldo = ldc, acc = accum;
  long long cs = 0;
  if (c.S > 1) {  // partial products into the scratch, summed afterwards
    cs = (long long)M * N;
    out = splitk_scratch((size_t)c.S * cs);
    if (!out) return 6;
    bout = nullptr;
    ldo = N;
    acc = 0;
  }
  const dim3 grid(c.gx, c.gy, c.S);
  bool ok;
  if (!tma)
    ok = c.bn == 32   ? launch_tc<32>(grid, st, A, B, out, bout, M, N, K, lda, ldb, ldo, acc, c.kchunk, cs)
         : c.bn == 64 ? launch_tc<64>(grid, st, A, B, out, bout, M, N, K, lda, ldb, ldo, acc, c.kchunk, cs)
                      : launch_tc<128>(grid, st, A, B, out, bout, M, N, K, lda, ldb, ldo, acc, c.kchunk, cs);
  else
    ok = c.bn == 32
             ? launch_tma_major<32>(a_mn, b_mn, ma, mb, grid, st, out, bout, M, N, K, ldo, acc, c.kchunk, cs, Y, act)
         : c.bn == 64
             ? launch_tma_major<64>(a_mn, b_mn, ma, mb, grid, st, out, bout, M, N, K, ldo, acc, c.kchunk, cs, Y, act)
             : launch_tma_major<128>(a_mn, b_mn, ma, mb, grid, st, out, bout, M, N, K, ldo, acc, c.kchunk, cs, Y, act);
  if (!ok) return 6;
  if (c.S > 1) k_splitk_sum<<<grid_for(cs), 256, 0, st>>>(out, c.S, cs, C, bias, M, N, ldc, accum);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

// The default kernel of the products (bpnet_gemm_tn): BPNET_GEMM=tc selects the
// register-staged tcgen05 kernel throughout, BPNET_GEMM=mma the mma.sync one.
int gemm_mode() {
  static const int mode = [] {
    const char* e = std::getenv("BPNET_GEMM");
    if (e && std::strcmp(e, "mma") == 0) return 2;
    if (e && std::strcmp(e, "tc") == 0) return 1;
    return 0;
  }();
  return mode;
}

}  // namespace

extern "C" {

int bpnet_act(const float* Z, void* Y, long long P, int C, int ldy, int c0, int act, void* stream);

// Returns 0, or 10 for arguments the kernels do not take.
// The product with an explicit kernel: mode 0 tcgen05 with TMA-fed operands
// (k_gemm_tma), 1 tcgen05 with register-staged operands (k_gemm_tc), 2 the
// mma.sync kernel.
int bpnet_gemm_tn_mode(int mode, const void* A, const void* B, float* C, const float* bias, int M, int N, int K,
                       int lda, int ldb, int ldc, int accum, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (K % 8) || (lda % 8) || (ldb % 8) || mode < 0 || mode > 2) return 10;
  cudaStream_t st = (cudaStream_t)stream;
  const bf16 *a16 = (const bf16*)A, *b16 = (const bf16*)B;
  if (mode == 2) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    k_gemm_tn<<<grid, 128, 0, st>>>(a16, b16, C, bias, M, N, K, lda, ldb, ldc, accum);
    return cudaGetLastError() == cudaSuccess ? 0 : 6;
  }
  if (mode == 0) {
    const int rc = tensor_gemm(1, 0, 0, a16, b16, C, bias, M, N, K, lda, ldb, ldc, accum, nullptr, 0, st);
    if (rc != 10) return rc;  // operands that TMA cannot map go through registers
  }
  return tensor_gemm(0, 0, 0, a16, b16, C, bias, M, N, K, lda, ldb, ldc, accum, nullptr, 0, st);
}

// Whether the default kernel of a K-major product is the register-staged one: a
// single K slice has no pipeline to fill, and with tiles for two CTAs an SM or
// more the copies of the other CTAs cover a CTA's own (131,072 x 32 x 56: 30.1
// us against 32.3 TMA-fed; 131,072 x 64 x 64 32.4 and 34.4; 65,536 x 64 x 56
// 24.4 and 26.6).  With fewer tiles the one bulk copy is there sooner (16,384
// x 32 x 56, 128 tiles: 21.4 and 20.4; 4,096 x 22 x 32 17.8 and 16.3).
int bpnet_gemm_by_registers(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K > TC_BK) return 0;
  const GemmCut c = cut_gemm(M, N, K);
  return (long long)c.gx * c.gy >= 296 ? 1 : 0;
}

// The product on the default kernel.
int bpnet_gemm_tn(const void* A, const void* B, float* C, const float* bias, int M, int N, int K, int lda,
                  int ldb, int ldc, int accum, void* stream) {
  const int mode = gemm_mode() == 0 && bpnet_gemm_by_registers(M, N, K) ? 1 : gemm_mode();
  return bpnet_gemm_tn_mode(mode, A, B, C, bias, M, N, K, lda, ldb, ldc, accum, stream);
}

// Whether bpnet_gemm_act leaves the activation to its own pass where it is
// given room for Z: with the register-staged kernel, which has no such
// epilogue, and whole 16-byte groups of channels (131,072 x 32 x 56: 41.1 us
// in two kernels, 44.2 fused; 262,144 rows 55.8, 64.1, and 59.4 fused without Z;
// 22 channels, element by element: 45.7 and 40.9).
int bpnet_act_apart(int M, int N, int K) { return N % 4 == 0 && bpnet_gemm_by_registers(M, N, K); }

// The product with its activation: Z = A B^T + bias (FP32, may be null) and Y
// = act(Z) in BF16, both with rows of N.
int bpnet_gemm_act(const void* A, const void* B, float* Z, const float* bias, void* Y, int M, int N, int K, int lda,
                   int ldb, int act, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (K % 8) || (lda % 8) || (ldb % 8) || !Y) return 10;
  cudaStream_t st = (cudaStream_t)stream;
  if (gemm_mode() == 0 && !(Z && bpnet_act_apart(M, N, K))) {
    const int rc = tensor_gemm(1, 0, 0, (const bf16*)A, (const bf16*)B, Z, bias, M, N, K, lda, ldb, N, 0, (bf16*)Y,
                               act, st);
    if (rc != 10) return rc;
  }
  if (!Z) return 10;
  const int rc = bpnet_gemm_tn(A, B, Z, bias, M, N, K, lda, ldb, N, 0, stream);
  return rc ? rc : bpnet_act(Z, Y, M, N, N, 0, act, stream);
}

// The product of operands of either order (a_mn, b_mn: element (m, k) at
// [k * ld + m]) on the TMA-fed kernel: the gradient products.  lda, ldb
// multiples of 8; 10 where the operands cannot be mapped.
int bpnet_gemm_major(int a_mn, int b_mn, const void* A, const void* B, float* C, int M, int N, int K, int lda, int ldb,
                     int ldc, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (lda % 8) || (ldb % 8)) return 10;
  if ((!a_mn || !b_mn) && K % 8) return 10;
  if (gemm_mode() != 0) return 10;
  return tensor_gemm(1, a_mn != 0, b_mn != 0, (const bf16*)A, (const bf16*)B, C, nullptr, M, N, K, lda, ldb, ldc, 0,
                     nullptr, 0, (cudaStream_t)stream);
}

// The mma.sync kernel (the comparison of the tcgen05 one).
int bpnet_gemm_tn_mma(const void* A, const void* B, float* C, const float* bias, int M, int N, int K, int lda,
                      int ldb, int ldc, int accum, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (K % 8) || (lda % 8) || (ldb % 8)) return 10;
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  k_gemm_tn<<<grid, 128, 0, (cudaStream_t)stream>>>((const bf16*)A, (const bf16*)B, C, bias, M, N, K, lda,
                                                     ldb, ldc, accum);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

// 1 if a wait of the tcgen05 GEMM ran out since the last call (and clears
// it), 0 if not, 6 on a CUDA error.
int bpnet_gemm_status(void* stream) {
  int e = 0, z = 0;
  if (cudaMemcpyFromSymbolAsync(&e, g_tc_err, sizeof(int), 0, cudaMemcpyDeviceToHost, (cudaStream_t)stream) !=
          cudaSuccess ||
      cudaMemcpyToSymbolAsync(g_tc_err, &z, sizeof(int), 0, cudaMemcpyHostToDevice, (cudaStream_t)stream) !=
          cudaSuccess ||
      cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess)
    return 6;
  return e;
}

int bpnet_im2col(const void* X, void* col, int B, int H, int W, int C, int Kp, int periodic, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const bool v8 = C % 8 == 0 && Kp == 9 * C && aligned(X, 16) && aligned(col, 16);
  const bool vec = Kp % 8 == 0 && aligned(col, 16);
  // images per launch: thread numbers fit 32 bits
  const long long per = (long long)H * W * (v8 ? C / 8 : (Kp + 7) / 8);
  if (per <= 0) return cudaGetLastError() == cudaSuccess ? 0 : 6;
  const int nb = (int)std::max(1LL, std::min((long long)B, (1LL << 31) / per));
  for (int b0 = 0; b0 < B; b0 += nb) {
    const unsigned P = (unsigned)((long long)std::min(nb, B - b0) * H * W);
    const bf16* x = (const bf16*)X + (size_t)b0 * H * W * C;
    bf16* o = (bf16*)col + (size_t)b0 * H * W * Kp;
    const unsigned blocks = (unsigned)(((long long)P * (v8 ? C / 8 : (Kp + 7) / 8) + 255) / 256);
    if (v8) k_im2col8<<<blocks, 256, 0, st>>>((const uint4*)x, (uint4*)o, P, H, W, C / 8, periodic);
    else if (vec) k_im2col_any<true><<<blocks, 256, 0, st>>>(x, o, P, H, W, C, Kp, periodic);
    else k_im2col_any<false><<<blocks, 256, 0, st>>>(x, o, P, H, W, C, Kp, periodic);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_col2im(const float* dcol, float* dX, int B, int H, int W, int C, int Kp, int periodic, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const bool v4 = C % 4 == 0 && Kp % 4 == 0 && aligned(dcol, 16) && aligned(dX, 16);
  const long long per = (long long)H * W * (v4 ? C / 4 : C);
  if (per <= 0) return cudaGetLastError() == cudaSuccess ? 0 : 6;
  const int nb = (int)std::max(1LL, std::min((long long)B, (1LL << 31) / per));
  for (int b0 = 0; b0 < B; b0 += nb) {
    const unsigned P = (unsigned)((long long)std::min(nb, B - b0) * H * W);
    const float* d = dcol + (size_t)b0 * H * W * Kp;
    float* o = dX + (size_t)b0 * H * W * C;
    const unsigned blocks = (unsigned)(((long long)P * (v4 ? C / 4 : C) + 255) / 256);
    if (v4) k_col2im<4><<<blocks, 256, 0, st>>>(d, o, P, H, W, C / 4, Kp, periodic);
    else k_col2im<1><<<blocks, 256, 0, st>>>(d, o, P, H, W, C, Kp, periodic);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_transpose(const void* in, void* out, int R, int Cc, void* stream) {
  dim3 grid((Cc + 31) / 32, (R + 31) / 32), block(32, 8);
  k_transpose<<<grid, block, 0, (cudaStream_t)stream>>>((const bf16*)in, (bf16*)out, R, Cc);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_act(const float* Z, void* Y, long long P, int C, int ldy, int c0, int act, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (C % 4 == 0 && ldy % 4 == 0 && c0 % 4 == 0 && aligned(Z, 16) && aligned(Y, 8))
    k_act<4><<<grid_for(P * C / 4), 256, 0, st>>>(Z, (bf16*)Y, P, C, ldy, c0, act);
  else
    k_act<1><<<grid_for(P * C), 256, 0, st>>>(Z, (bf16*)Y, P, C, ldy, c0, act);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_act_grad(const float* Z, const float* dY, float* dZ, long long P, int C, int ldd, int c0, int act,
                   void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (C % 4 == 0 && ldd % 4 == 0 && c0 % 4 == 0 && aligned(Z, 16) && aligned(dY, 16) && aligned(dZ, 16))
    k_act_grad<4><<<grid_for(P * C / 4), 256, 0, st>>>(Z, dY, dZ, P, C, ldd, c0, act);
  else
    k_act_grad<1><<<grid_for(P * C), 256, 0, st>>>(Z, dY, dZ, P, C, ldd, c0, act);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

// dZ in BF16 and its column sums db [C] (dY [P][C]; scratch: (P + 256) C
// floats, which receive dZ in FP32 and the running sums).
int bpnet_act_grad_sum(const float* Z, const float* dY, void* dZb, float* db, float* scratch, long long P, int C,
                       int act, void* stream) {
  if (C <= 0) return 10;
  cudaStream_t st = (cudaStream_t)stream;
  const long long n = P * C;
  float* part = scratch + n;
  if (n % 4 == 0 && aligned(Z, 16) && aligned(dY, 16) && aligned(dZb, 8) && aligned(scratch, 16))
    k_act_grad_both<4><<<grid_for(n / 4), 256, 0, st>>>(Z, dY, scratch, (bf16*)dZb, n, act);
  else
    k_act_grad_both<1><<<grid_for(n), 256, 0, st>>>(Z, dY, scratch, (bf16*)dZb, n, act);
  k_colsum_rows<<<dim3(32, (C + 31) / 32), dim3(32, 8), 0, st>>>(scratch, part, P, C);
  k_colsum_tree<<<C, 256, 0, st>>>(part, db, C);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

// dX [B][H][W][cin] (FP32) of a 3 x 3 convolution with weights [cout][Kp] from
// dZ [B][H][W][cout].  10 for what it does not take: channels that are not
// multiples of 32, more output channels than shared memory holds, operands
// that are not 16-byte aligned, another GEMM kernel selected, few pixels.
int bpnet_dgrad3(const void* dZ, const void* w, float* dX, int B, int H, int W, int cin, int cout, int Kp, int periodic,
                 void* stream) {
  if (B <= 0 || H <= 0 || W <= 0 || cin <= 0 || cout <= 0) return 10;
  if (cin % 32 || cout % 32 || cout > DG_MAX_COUT || Kp < 9 * cin || B > 65535 || cin / 32 > 65535) return 10;
  if (!aligned(dZ, 16) || gemm_mode() != 0) return 10;
  const long long tiles = (long long)((W + DG_W - 1) / DG_W) * ((H + DG_H - 1) / DG_H);
  if (tiles > 0x7fffffffLL) return 10;
  // few CTAs with a long row of slices: the product over all taps spreads wider
  // (16 x 16 pixels, 256 to 256 channels: 17 us against 29; at 128 CTAs equal)
  if (cout > 128 && tiles * B * (cin / 32) < 128) return 10;
  // the widest tile that gives every SM a CTA: 128 x 128 x 8 pixels, 96 to 32
  // channels, 64 us with 96 columns and 77 with 32; 64 x 64 x 8, 192 to 64, 38 and 48
  int nb = 1;
  for (int n = 3; n > 1; --n)
    if (cin % (32 * n) == 0 && tiles * B * (cin / (32 * n)) >= 148) {
      nb = n;
      break;
    }
  const auto f = cout % 64 == 0 ? (nb == 3 ? launch_dgrad3<3, 64> : nb == 2 ? launch_dgrad3<2, 64> : launch_dgrad3<1, 64>)
                                : (nb == 3 ? launch_dgrad3<3, 32> : nb == 2 ? launch_dgrad3<2, 32> : launch_dgrad3<1, 32>);
  return f(dZ, w, dX, B, H, W, cin, cout, Kp, periodic, (cudaStream_t)stream);
}

int bpnet_to_bf16(const float* x, void* y, long long n, void* stream) {
  k_f32_to_bf16<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(x, (bf16*)y, n);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_colsum(const float* dZ, float* db, long long P, int C, void* stream) {
  k_colsum<<<C, 256, 0, (cudaStream_t)stream>>>(dZ, db, P, C);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_pool(const void* X, void* Y, int B, int H, int W, int C, void* stream) {
  if ((H % 2) || (W % 2)) return 10;
  cudaStream_t st = (cudaStream_t)stream;
  const long long n = (long long)B * (H / 2) * (W / 2) * C;
  if (C % 8 == 0 && aligned(X, 16) && aligned(Y, 16))
    k_pool<8><<<grid_for(n / 8), 256, 0, st>>>((const bf16*)X, (bf16*)Y, B, H, W, C);
  else
    k_pool<1><<<grid_for(n), 256, 0, st>>>((const bf16*)X, (bf16*)Y, B, H, W, C);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_pool_grad(const float* dY, float* dX, int B, int H, int W, int C, int ldy, int c0, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const long long n = (long long)B * H * W * C;
  if (vec4(C, ldy, c0, dY, dX)) k_pool_grad<4><<<grid_for(n / 4), 256, 0, st>>>(dY, dX, B, H, W, C, ldy, c0);
  else k_pool_grad<1><<<grid_for(n), 256, 0, st>>>(dY, dX, B, H, W, C, ldy, c0);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_up(const void* X, void* Y, int B, int h, int w, int C, int ldy, int c0, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const long long n = (long long)B * 4 * h * w * C;
  if (vec8(C, ldy, c0, X, Y)) k_up<8><<<grid_for(n / 8), 256, 0, st>>>((const bf16*)X, (bf16*)Y, B, h, w, C, ldy, c0);
  else k_up<1><<<grid_for(n), 256, 0, st>>>((const bf16*)X, (bf16*)Y, B, h, w, C, ldy, c0);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_up_grad(const float* dY, float* dX, int B, int h, int w, int C, int ldy, int c0, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const long long n = (long long)B * h * w * C;
  if (vec4(C, ldy, c0, dY, dX)) k_up_grad<4><<<grid_for(n / 4), 256, 0, st>>>(dY, dX, B, h, w, C, ldy, c0);
  else k_up_grad<1><<<grid_for(n), 256, 0, st>>>(dY, dX, B, h, w, C, ldy, c0);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_copy_slice(const void* X, void* Y, long long P, int C, int ldy, int c0, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (vec8(C, ldy, c0, X, Y))
    k_copy_slice<8><<<grid_for(P * C / 8), 256, 0, st>>>((const bf16*)X, (bf16*)Y, P, C, ldy, c0);
  else
    k_copy_slice<1><<<grid_for(P * C), 256, 0, st>>>((const bf16*)X, (bf16*)Y, P, C, ldy, c0);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_add_slice(const float* dY, float* dX, long long P, int C, int ldy, int c0, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (vec4(C, ldy, c0, dY, dX)) k_add_slice<4><<<grid_for(P * C / 4), 256, 0, st>>>(dY, dX, P, C, ldy, c0);
  else k_add_slice<1><<<grid_for(P * C), 256, 0, st>>>(dY, dX, P, C, ldy, c0);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

// partial must hold 256 floats; the loss is the sum of them (host side).
int bpnet_mse(const float* Y, const float* T, const float* mask, float* dY, float* partial, long long P, int C,
              float inv_count, void* stream) {
  k_mse<<<256, 256, 0, (cudaStream_t)stream>>>(Y, T, mask, dY, partial, P, C, inv_count);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_adam(float* w, const float* grad, float* m1, float* m2, void* wb, long long n, int K, int Kp,
               float lr, float b1, float b2, float eps, float c1, float c2, void* stream) {
  k_adam<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(w, grad, m1, m2, (bf16*)wb, n, K, Kp, lr, b1, b2, eps,
                                                        c1, c2);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

int bpnet_unpad(const float* src, float* dst, long long rows, int K, int Kp, void* stream) {
  k_unpad<<<grid_for(rows * K), 256, 0, (cudaStream_t)stream>>>(src, dst, rows, K, Kp);
  return cudaGetLastError() == cudaSuccess ? 0 : 6;
}

}  // extern "C"
