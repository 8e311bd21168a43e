// Small dense helpers of the MoE layer's backward pass (sm_100a, plain CUDA cores):
//
//   transpose_experts   dst[n][j][col0 + i] = src[n][i][j] for a stack of bf16 matrices, through a
//                       64x64 shared-memory tile with 16-byte global accesses on both sides.  Builds the
//                       K-major copies of the local experts that the activation-gradient GEMMs read.
//   swiglu_bwd          per row r and column i, from a = x Wg^T, u = x Wu^T and g = dy Wd (unscaled):
//                         h = silu(a) u;  dgate[r] = sum_i g h;  dh = g w[r]
//                         da = dh u s (1 + a (1 - s)),  du = dh a s   (s = sigmoid(a))
//                       writes [da | du] side by side (one GEMM then yields dx), h*w (for the down
//                       projection's weight gradient) and dgate.
//
//   sgd_update          w (bf16) -= lr * g (fp32), vectorised.
//   adamw_update        one AdamW step of up to kUpdateTensors weights in one pass: fp32 master, moments and gradient in,
//                       master, moments and the rounded bf16 weight out.
//
// The reference has no expert computation; these serve the MoE training-step configuration.
#include <cuda_bf16.h>

#include "common.cuh"
#include "host.h"

namespace moonep {

namespace {

constexpr int kTile = 64;
constexpr int kUpdateTensors = 3;  // weights per launch of the weight updates
constexpr int kUpdateSteps = 4;  // vectors per thread of the weight updates, at most

__global__ void __launch_bounds__(256)
    transpose_experts_kernel(const uint16_t* __restrict__ src, uint16_t* __restrict__ dst, int d0, int d1,
                             long long dst_ld, long long dst_expert_stride, int col0, const int* __restrict__ active) {
  __shared__ uint16_t tile[kTile][kTile + 8];
  const int n = blockIdx.z;
  if (active != nullptr && active[n] < 0) return;  // e.g. a prefetch slot that holds no expert in this step
  const int i0 = blockIdx.y * kTile, j0 = blockIdx.x * kTile;
  const uint16_t* s = src + (long long)n * d0 * d1;
  uint16_t* d = dst + (long long)n * dst_expert_stride;
  // load 64 rows x 64 columns, 8 columns (16 bytes) per thread and step
  for (int v = threadIdx.x; v < kTile * (kTile / 8); v += blockDim.x) {
    const int r = v / (kTile / 8), cv = v % (kTile / 8);
    const int4 x = ld16(s + (long long)(i0 + r) * d1 + j0 + cv * 8);
    const uint16_t* e = reinterpret_cast<const uint16_t*>(&x);
#pragma unroll
    for (int q = 0; q < 8; ++q) tile[r][cv * 8 + q] = e[q];
  }
  __syncthreads();
  // store: output row j (a source column), 8 consecutive i per thread
  for (int v = threadIdx.x; v < kTile * (kTile / 8); v += blockDim.x) {
    const int j = v / (kTile / 8), iv = v % (kTile / 8);
    int4 x;
    uint16_t* e = reinterpret_cast<uint16_t*>(&x);
#pragma unroll
    for (int q = 0; q < 8; ++q) e[q] = tile[iv * 8 + q][j];
    st16(d + (long long)(j0 + j) * dst_ld + col0 + i0 + iv * 8, x);
  }
}

__device__ __forceinline__ float bf(uint16_t u) { return __uint_as_float(((unsigned)u) << 16); }
__device__ __forceinline__ uint16_t tobf(float f) {
  __nv_bfloat16 b = __float2bfloat16_rn(f);
  return *reinterpret_cast<uint16_t*>(&b);
}

// one warp per row; I must be a multiple of 8
__global__ void __launch_bounds__(256)
    swiglu_bwd_kernel(const uint16_t* __restrict__ a, const uint16_t* __restrict__ u, const uint16_t* __restrict__ g,
                      const float* __restrict__ w, const int* __restrict__ total_rows_ptr, int rows_cap, int I,
                      uint16_t* __restrict__ dadu, uint16_t* __restrict__ hsw, float* __restrict__ dgate) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  griddep_wait();
  griddep_launch();
  int rows = total_rows_ptr != nullptr ? *total_rows_ptr : rows_cap;
  if (rows > rows_cap) rows = rows_cap;
  for (int r = blockIdx.x * nwarps + warp; r < rows; r += gridDim.x * nwarps) {
    const float wr = w[r];
    float acc = 0.f;
    const long long base = (long long)r * I;
    for (int c0 = lane * 8; c0 < I; c0 += 32 * 8) {
      const int4 av = ld16(a + base + c0), uv = ld16(u + base + c0), gv = ld16(g + base + c0);
      const uint16_t* ae = reinterpret_cast<const uint16_t*>(&av);
      const uint16_t* ue = reinterpret_cast<const uint16_t*>(&uv);
      const uint16_t* ge = reinterpret_cast<const uint16_t*>(&gv);
      int4 dav, duv, hv;
      uint16_t* dae = reinterpret_cast<uint16_t*>(&dav);
      uint16_t* due = reinterpret_cast<uint16_t*>(&duv);
      uint16_t* he = reinterpret_cast<uint16_t*>(&hv);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float x = bf(ae[q]), y = bf(ue[q]), gg = bf(ge[q]);
        const float s = 1.f / (1.f + __expf(-x));
        const float h = x * s * y;
        acc += gg * h;
        const float dh = gg * wr;
        dae[q] = tobf(dh * y * s * (1.f + x * (1.f - s)));
        due[q] = tobf(dh * x * s);
        he[q] = tobf(h * wr);
      }
      st16(dadu + (long long)r * 2 * I + c0, dav);
      st16(dadu + (long long)r * 2 * I + I + c0, duv);
      st16(hsw + base + c0, hv);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) dgate[r] = acc;
  }
}

// w (bf16) -= lr * g (fp32), 8 elements per thread and step.  Short CTAs as in adamw_kernel: 117 M elements 160 -> 145 us.
// The weights of a layer share a launch: a training step of S=64, H=1024, I=256, 6 experts 98.7 -> 92.7 us, S=1500, H=4096,
// I=1024, 8 experts 469 -> 460.  Placed while the kernel before still ran (PDL), the latter took 499.
struct SgdTensor {
  uint16_t* w;
  const float* g;
  long long n8;  // groups of eight elements
};
struct SgdArgs {
  SgdTensor t[kUpdateTensors];
  float lr;
  int steps;  // vectors per thread
};

__global__ void __launch_bounds__(256) sgd_update_kernel(const __grid_constant__ SgdArgs a) {
  uint16_t* __restrict__ w = a.t[blockIdx.y].w;
  const float* __restrict__ g = a.t[blockIdx.y].g;
  const long long n8 = a.t[blockIdx.y].n8;
  const float lr = a.lr;
  const long long first = (long long)blockIdx.x * (256 * a.steps) + threadIdx.x;
#pragma unroll 1
  for (int s = 0; s < a.steps; ++s) {
    const long long v = first + s * 256;
    if (v >= n8) break;
    int4 wv = ld16(w + v * 8);
    const int4 g0 = ld16(g + v * 8), g1 = ld16(g + v * 8 + 4);
    uint16_t* we = reinterpret_cast<uint16_t*>(&wv);
    const float gf[8] = {__int_as_float(g0.x), __int_as_float(g0.y), __int_as_float(g0.z), __int_as_float(g0.w),
                         __int_as_float(g1.x), __int_as_float(g1.y), __int_as_float(g1.z), __int_as_float(g1.w)};
#pragma unroll
    for (int q = 0; q < 8; ++q) we[q] = tobf(bf(we[q]) - lr * gf[q]);
    st16(w + v * 8, wv);
  }
}

// One AdamW step.  Bound by HBM: 16 bytes in and 14 out per element, where a pass per operation moved 86.  Three weights
// of 33.5 M elements: 1350 us as 30 elementwise launches, 478 us here (6.3 TB/s).  The four loads of a step are 16 bytes
// each and independent.  CTAs are short (kUpdateSteps vectors per thread) and scheduled as they fit: SMs reach HBM at
// rates that differ by a quarter, and a resident grid that strode over the elements took 515 us.
struct AdamTensor {
  float* p;        // fp32 master
  float* m;        // first moment
  float* v;        // second moment
  const float* g;  // gradient
  uint16_t* w;     // bf16 weight
  long long n4;    // groups of four elements
};
struct AdamArgs {
  AdamTensor t[kUpdateTensors];
  int steps;              // vectors per thread
  float decay;            // 1 - lr * weight_decay
  float b1, b2;           // decay rates of the moments
  float one_b1, one_b2;   // 1 - b1, 1 - b2
  float inv_c2, eps;      // 1 / bias correction of the second moment
  float step;             // lr / bias correction of the first moment
};

__global__ void __launch_bounds__(256) adamw_kernel(const AdamArgs a) {
  const AdamTensor t = a.t[blockIdx.y];
  const long long first = (long long)blockIdx.x * (256 * a.steps) + threadIdx.x;
#pragma unroll 1
  for (int s = 0; s < a.steps; ++s) {
    const long long i = first + s * 256;
    if (i >= t.n4) break;
    int4 x[4] = {ld16(t.p + i * 4), ld16(t.m + i * 4), ld16(t.v + i * 4), ld16(t.g + i * 4)};
    float *p = reinterpret_cast<float*>(&x[0]), *m = reinterpret_cast<float*>(&x[1]), *v = reinterpret_cast<float*>(&x[2]);
    const float* g = reinterpret_cast<const float*>(&x[3]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      m[q] = m[q] * a.b1 + a.one_b1 * g[q];
      v[q] = v[q] * a.b2 + a.one_b2 * (g[q] * g[q]);
      p[q] = p[q] * a.decay - a.step * (m[q] / (sqrtf(v[q] * a.inv_c2) + a.eps));
    }
    st16(t.p + i * 4, x[0]);
    st16(t.m + i * 4, x[1]);
    st16(t.v + i * 4, x[2]);
    *reinterpret_cast<uint2*>(t.w + i * 4) = make_uint2(pack_bf16(p[0], p[1]), pack_bf16(p[2], p[3]));
  }
}

}  // namespace

}  // namespace moonep

using namespace moonep;

// Vectors per thread: a thread's steps follow one another, so as long as one step each does not fill the GPU (8 CTAs per SM)
// there is one: up to 1 M elements an SGD update takes 6.2 us, 8.2 with four.
static int update_steps(long long vectors) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long full = vectors / (256ll * 8 * imax(1, sms));
  return (int)(full < 1 ? 1 : full > kUpdateSteps ? kUpdateSteps : full);
}

// count weights: master, m, v, g fp32 and w bf16 of n[i] elements each (a multiple of 4; all 16-byte aligned, w 8-byte).
// step: lr / bias correction of m; decay: 1 - lr * weight_decay; c2: bias correction of v.
extern "C" int moonep_adamw_update(int count, void* const* master, void* const* m, void* const* v, void* const* g,
                                   void* const* w, const long long* n, double step, double b1, double b2, double eps,
                                   double decay, double c2, void* stream) {
  if (count < 1 || count > kUpdateTensors) {
    set_error("moonep_adamw_update: 1 to " + std::to_string(kUpdateTensors) + " weights per call");
    return 1;
  }
  AdamArgs a;
  long long most = 0;
  for (int i = 0; i < count; ++i) {
    const uintptr_t bits = (uintptr_t)master[i] | (uintptr_t)m[i] | (uintptr_t)v[i] | (uintptr_t)g[i];
    if (n[i] % 4 != 0 || (bits & 15u) != 0 || ((uintptr_t)w[i] & 7u) != 0) {
      set_error("moonep_adamw_update: element counts must be multiples of 4 and the tensors 16-byte aligned");
      return 1;
    }
    a.t[i] = {(float*)master[i], (float*)m[i], (float*)v[i], (const float*)g[i], (uint16_t*)w[i], n[i] / 4};
    most = n[i] > most ? n[i] : most;
  }
  if (most == 0) return 0;
  a.decay = (float)decay;
  a.b1 = (float)b1;
  a.b2 = (float)b2;
  a.one_b1 = (float)(1.0 - b1);
  a.one_b2 = (float)(1.0 - b2);
  a.inv_c2 = (float)(1.0 / c2);
  a.eps = (float)eps;
  a.step = (float)step;
  a.steps = update_steps(most / 4 * count);
  const long long per_cta = 256 * 4 * a.steps;
  const dim3 grid((unsigned)((most + per_cta - 1) / per_cta), (unsigned)count);
  adamw_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(a);
  return check_launch("adamw_kernel");
}

// count weights, w: [n[i]] bf16, g: [n[i]] fp32, n[i] a multiple of 8: w -= lr * g.
extern "C" int moonep_sgd_update(int count, void* const* w, void* const* g, const long long* n, float lr, void* stream) {
  if (count < 1 || count > kUpdateTensors) {
    set_error("moonep_sgd_update: 1 to " + std::to_string(kUpdateTensors) + " weights per call");
    return 1;
  }
  SgdArgs a;
  long long most = 0;
  for (int i = 0; i < count; ++i) {
    if (n[i] % 8 != 0) {
      set_error("moonep_sgd_update: element counts must be multiples of 8");
      return 1;
    }
    a.t[i] = {(uint16_t*)w[i], (const float*)g[i], n[i] / 8};
    most = n[i] > most ? n[i] : most;
  }
  if (most == 0) return 0;
  a.lr = lr;
  a.steps = update_steps(most / 8 * count);
  const long long per_cta = 256 * 8 * a.steps;
  const dim3 grid((unsigned)((most + per_cta - 1) / per_cta), (unsigned)count);
  sgd_update_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(a);
  return check_launch("sgd_update_kernel");
}

// src: [n, d0, d1] bf16 -> dst[n][j][col0 + i] with row stride dst_ld and expert stride dst_expert_stride (elements).
// active (optional, device, [n]): matrices with a negative entry are skipped.
extern "C" int moonep_transpose_experts(const void* src, void* dst, int n, int d0, int d1, long long dst_ld,
                                        long long dst_expert_stride, int col0, const int* active, void* stream) {
  if (n <= 0) return 0;
  if (d0 % kTile != 0 || d1 % kTile != 0 || dst_ld % 8 != 0 || col0 % 8 != 0) {
    set_error("moonep_transpose_experts: dimensions must be multiples of 64 and the destination 16-byte aligned");
    return 1;
  }
  dim3 grid(d1 / kTile, d0 / kTile, n);
  transpose_experts_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const uint16_t*)src, (uint16_t*)dst, d0, d1, dst_ld,
                                                                   dst_expert_stride, col0, active);
  return check_launch("transpose_experts_kernel");
}

// a, u, g: [rows_cap, I] bf16; w: [rows_cap] fp32; total_rows: device int (rows in use) or null.
extern "C" int moonep_swiglu_bwd(const void* a, const void* u, const void* g, const float* w, const int* total_rows,
                                 int rows_cap, int I, void* dadu, void* hsw, float* dgate, void* stream) {
  if (I % 8 != 0 || rows_cap <= 0) {
    set_error("moonep_swiglu_bwd: I must be a multiple of 8");
    return 1;
  }
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (int rc = check_cuda(launch_maybe_pdl(swiglu_bwd_kernel, imax(1, sms * 4), 256, 0, (cudaStream_t)stream, expert_pdl(0),
                                           (const uint16_t*)a, (const uint16_t*)u, (const uint16_t*)g, w, total_rows, rows_cap, I,
                                           (uint16_t*)dadu, (uint16_t*)hsw, dgate),
                          "launch swiglu_bwd_kernel"))
    return rc;
  return check_launch("swiglu_bwd_kernel");
}
