// SwiGLU glue between the gate/up and the down projection: a = T(T(silu(g)) * u) and its backward, every
// intermediate rounded to the activation type T (bf16 or fp16) exactly where PyTorch autograd rounds
// `F.silu(g) * u` -- so the op can replace the autograd expression bit for bit in the forward and in du.
// Reference operators: torch.ops.bitlattice.swiglu_fwd / swiglu_bwd (csrc/swiglu.cu:20-80, csrc/bindings.cpp:126-129).
//
// Streaming work: 2 reads + 1 write (forward), 3 reads + 2 writes (backward) of 2-byte elements, 6 and 10 bytes per element;
// one thread handles 8 consecutive elements (16-byte accesses), grid-stride over the tensor, the next vectors' loads issued
// before the current ones are worked on. What bounds it above the bytes is the arithmetic of the sigmoid: one exponential
// and, in IEEE arithmetic, two divisions by the same d = 1 + exp(-g). glu_sigmoid shares one reciprocal between them. On a
// B200, 65536 x 12288 bf16: forward 986 -> 796 us (6.1 TB/s), backward 1585 -> 1325 us (6.1 TB/s); 4096 x 12288 from HBM: 70 ->
// 59 and 106 -> 86 us.
#include "common.cuh"

namespace blb {

constexpr int kGluThreads = 256;
constexpr int kFwdCtas = 5, kBwdCtas = 4;     // CTAs an SM holds (48 and 64 registers); the grids are one wave of them

// ATen's silu in its op-math type: x / (1 + exp(-x)), true division
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }

template <typename T>
struct Pack8 {
  uint4 raw;
  __device__ __forceinline__ float get(int i) const { return to_f<T>(reinterpret_cast<const T*>(&raw)[i]); }
  __device__ __forceinline__ void set(int i, float v) { reinterpret_cast<T*>(&raw)[i] = from_f<T>(v); }
};

template <typename T>
__device__ __forceinline__ float round_to(float v) { return to_f<T>(from_f<T>(v)); }

template <typename T>
__device__ __forceinline__ float glu_forward(float g, float u) { return round_to<T>(silu_f(g)) * u; }

// (dg, du) for one element; the order of operations is ATen's silu_backward: d * sig * (1 + g * (1 - sig))
template <typename T>
__device__ __forceinline__ void glu_backward(float g, float u, float da, float& dg, float& du) {
  du = da * round_to<T>(silu_f(g));
  const float ds = round_to<T>(da * u);
  const float sig = 1.0f / (1.0f + expf(-g));
  dg = ds * sig * (1.0f + g * (1.0f - sig));
}

// -1/d and -g/d of a pair of elements, d = 1 + exp(-g), both rounded to nearest like the plain divisions: the hardware's
// approximate reciprocal takes one Newton step, and the quotient Markstein's correction (div_rn in common.cuh). g has 16
// bits, so d takes at most 2^16 values: the tests compare every one with the plain divisions. Valid for finite g >= -87: d
// stays in [1, 2^126), the reciprocal is normal, and a g so small that the quotient is not has d = 2, an exact half (zeros
// keep their sign: the residual is +0). glu_in_range says so for eight elements; a warp with others takes the plain divisions,
// out of line, as a whole (32768 x 12288 of N(0, 100^2): forward 1343 us by thread, 1130 by warp; gates that are all in range,
// zeros among them or not, 401). The signs come out negated because the reciprocal's operand can be negated for free and
// packed operands cannot.
__device__ __forceinline__ f32x2 newton_neg_rcp(float d0, float d1) {       // -1/d, two lanes
  const f32x2 nr = pk(rcp_approx(-d0), rcp_approx(-d1));
  return fma2p(nr, fma2p(pk(d0, d1), nr, pk(1.0f, 1.0f)), nr);
}
__device__ __forceinline__ void glu_sigmoid(float g0, float g1, f32x2& nsig, f32x2& nsilu) {
  const float d0 = 1.0f + expf(-g0), d1 = 1.0f + expf(-g1);
  const f32x2 d = pk(d0, d1), g = pk(g0, g1);
  nsig = newton_neg_rcp(d0, d1);
  const f32x2 nq = mul2p(g, nsig);
  nsilu = fma2p(fma2p(d, nq, g), nsig, nq);
}
__device__ __forceinline__ bool glu_in_range(const float g[8]) {            // a NaN gives false
  float lo = g[0], hi = g[0];
#pragma unroll
  for (int i = 1; i < 7; i += 2) {
    asm("min.NaN.f32 %0, %0, %1, %2;" : "+f"(lo) : "f"(g[i]), "f"(g[i + 1]));
    asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(hi) : "f"(g[i]), "f"(g[i + 1]));
  }
  asm("min.NaN.f32 %0, %0, %1, %1;" : "+f"(lo) : "f"(g[7]));
  asm("max.NaN.f32 %0, %0, %1, %1;" : "+f"(hi) : "f"(g[7]));
  return lo >= -87.0f && hi <= 3.4028235e38f;
}

template <typename T>
static __device__ __noinline__ uint4 glu_forward8_plain(uint4 g, uint4 u) {
  Pack8<T> pg, pu, pa;
  pg.raw = g;
  pu.raw = u;
#pragma unroll
  for (int i = 0; i < 8; ++i) pa.set(i, glu_forward<T>(pg.get(i), pu.get(i)));
  return pa.raw;
}

template <typename T>
static __device__ __noinline__ void glu_backward8_plain(uint4 g, uint4 u, uint4 d, uint4* og, uint4* ou) {
  Pack8<T> pg, pu, pd, px, py;
  pg.raw = g;
  pu.raw = u;
  pd.raw = d;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float x, y;
    glu_backward<T>(pg.get(i), pu.get(i), pd.get(i), x, y);
    px.set(i, x);
    py.set(i, y);
  }
  *og = px.raw;
  *ou = py.raw;
}

template <typename T>
__device__ __forceinline__ uint4 glu_forward8(const Pack8<T>& pg, const Pack8<T>& pu) {
  Pack8<T> pa;
  float g[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) g[i] = pg.get(i);
  if (__builtin_expect(!__all_sync(__activemask(), glu_in_range(g)), 0)) return glu_forward8_plain<T>(pg.raw, pu.raw);
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    f32x2 nsig, nsilu;
    glu_sigmoid(g[i], g[i + 1], nsig, nsilu);
    float s0, s1;
    upk(nsilu, s0, s1);
    pa.set(i, -round_to<T>(s0) * pu.get(i));
    pa.set(i + 1, -round_to<T>(s1) * pu.get(i + 1));
  }
  return pa.raw;
}

template <typename T>
__device__ __forceinline__ void glu_backward8(const Pack8<T>& pg, const Pack8<T>& pu, const Pack8<T>& pd, uint4* dg, uint4* du) {
  float g[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) g[i] = pg.get(i);
  if (__builtin_expect(!__all_sync(__activemask(), glu_in_range(g)), 0)) {
    glu_backward8_plain<T>(pg.raw, pu.raw, pd.raw, dg, du);
    return;
  }
  Pack8<T> og, ou;
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    f32x2 nsig, nsilu;
    glu_sigmoid(g[i], g[i + 1], nsig, nsilu);
    float ns[2], nl[2];
    upk(nsig, ns[0], ns[1]);
    upk(nsilu, nl[0], nl[1]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float da = pd.get(i + e), sig = -ns[e];
      ou.set(i + e, da * -round_to<T>(nl[e]));
      og.set(i + e, round_to<T>(da * pu.get(i + e)) * sig * (1.0f + g[i + e] * (1.0f - sig)));
    }
  }
  *dg = og.raw;
  *du = ou.raw;
}

template <typename T>
__global__ void __launch_bounds__(kGluThreads, kFwdCtas) swiglu_fwd_kernel(const T* __restrict__ g, const T* __restrict__ u,
                                                                           T* __restrict__ a, int64_t n) {
  const int64_t nvec = n / 8, stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  Pack8<T> pg, pu;
  if (v < nvec) {
    pg.raw = __ldcs(reinterpret_cast<const uint4*>(g) + v);
    pu.raw = __ldcs(reinterpret_cast<const uint4*>(u) + v);
  }
  while (v < nvec) {
    const int64_t next = v + stride;
    Pack8<T> ng, nu;
    if (next < nvec) {
      ng.raw = __ldcs(reinterpret_cast<const uint4*>(g) + next);
      nu.raw = __ldcs(reinterpret_cast<const uint4*>(u) + next);
    }
    reinterpret_cast<uint4*>(a)[v] = glu_forward8<T>(pg, pu);
    pg = ng;
    pu = nu;
    v = next;
  }
  // ragged tail: the last n % 8 elements, one per thread of block 0
  const int64_t t = nvec * 8 + threadIdx.x;
  if (blockIdx.x == 0 && t < n) a[t] = from_f<T>(glu_forward<T>(to_f<T>(g[t]), to_f<T>(u[t])));
}

template <typename T>
__global__ void __launch_bounds__(kGluThreads, kBwdCtas) swiglu_bwd_kernel(const T* __restrict__ g, const T* __restrict__ u,
                                                                           const T* __restrict__ da, T* __restrict__ dg,
                                                                           T* __restrict__ du, int64_t n) {
  const int64_t nvec = n / 8, stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  Pack8<T> pg, pu, pd;
  if (v < nvec) {
    pg.raw = __ldcs(reinterpret_cast<const uint4*>(g) + v);
    pu.raw = __ldcs(reinterpret_cast<const uint4*>(u) + v);
    pd.raw = __ldcs(reinterpret_cast<const uint4*>(da) + v);
  }
  while (v < nvec) {
    const int64_t next = v + stride;
    Pack8<T> ng, nu, nd;
    if (next < nvec) {
      ng.raw = __ldcs(reinterpret_cast<const uint4*>(g) + next);
      nu.raw = __ldcs(reinterpret_cast<const uint4*>(u) + next);
      nd.raw = __ldcs(reinterpret_cast<const uint4*>(da) + next);
    }
    glu_backward8<T>(pg, pu, pd, reinterpret_cast<uint4*>(dg) + v, reinterpret_cast<uint4*>(du) + v);
    pg = ng;
    pu = nu;
    pd = nd;
    v = next;
  }
  const int64_t t = nvec * 8 + threadIdx.x;
  if (blockIdx.x == 0 && t < n) {
    float x, y;
    glu_backward<T>(to_f<T>(g[t]), to_f<T>(u[t]), to_f<T>(da[t]), x, y);
    dg[t] = from_f<T>(x);
    du[t] = from_f<T>(y);
  }
}

static int glu_grid(int64_t n, int device, int per_sm) {
  const int64_t blocks = (n / 8 + kGluThreads - 1) / kGluThreads;
  const int64_t cap = static_cast<int64_t>(sm_count(device)) * per_sm;
  return static_cast<int>(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

}  // namespace blb

using namespace blb;

extern "C" int bl_swiglu_fwd(const void* g, const void* u, void* a, int dtype, int64_t n, int device,
                             bl_stream_t stream) {
  BL_REQUIRE(g && u && a && n > 0, "swiglu_fwd: null or empty buffer");
  BL_REQUIRE(dtype == BL_BF16 || dtype == BL_F16, "swiglu_fwd: activations must be bf16 or fp16, got dtype %d", dtype);
  BL_REQUIRE(aligned16(g) && aligned16(u) && aligned16(a), "swiglu_fwd: buffers must be 16-byte aligned");
  BL_DEVICE(device);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int grid = glu_grid(n, device, kFwdCtas);
  if (dtype == BL_BF16)
    swiglu_fwd_kernel<<<grid, kGluThreads, 0, st>>>(static_cast<const __nv_bfloat16*>(g),
                                                    static_cast<const __nv_bfloat16*>(u),
                                                    static_cast<__nv_bfloat16*>(a), n);
  else
    swiglu_fwd_kernel<<<grid, kGluThreads, 0, st>>>(static_cast<const __half*>(g), static_cast<const __half*>(u),
                                                    static_cast<__half*>(a), n);
  BL_CUDA(cudaGetLastError());
  return 0;
}

extern "C" int bl_swiglu_bwd(const void* g, const void* u, const void* da, void* dg, void* du, int dtype, int64_t n,
                             int device, bl_stream_t stream) {
  BL_REQUIRE(g && u && da && dg && du && n > 0, "swiglu_bwd: null or empty buffer");
  BL_REQUIRE(dtype == BL_BF16 || dtype == BL_F16, "swiglu_bwd: activations must be bf16 or fp16, got dtype %d", dtype);
  BL_REQUIRE(aligned16(g) && aligned16(u) && aligned16(da) && aligned16(dg) && aligned16(du),
             "swiglu_bwd: buffers must be 16-byte aligned");
  BL_DEVICE(device);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int grid = glu_grid(n, device, kBwdCtas);
  if (dtype == BL_BF16)
    swiglu_bwd_kernel<<<grid, kGluThreads, 0, st>>>(
        static_cast<const __nv_bfloat16*>(g), static_cast<const __nv_bfloat16*>(u),
        static_cast<const __nv_bfloat16*>(da), static_cast<__nv_bfloat16*>(dg), static_cast<__nv_bfloat16*>(du), n);
  else
    swiglu_bwd_kernel<<<grid, kGluThreads, 0, st>>>(static_cast<const __half*>(g), static_cast<const __half*>(u),
                                                    static_cast<const __half*>(da), static_cast<__half*>(dg),
                                                    static_cast<__half*>(du), n);
  BL_CUDA(cudaGetLastError());
  return 0;
}
