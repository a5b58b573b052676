// st3d_kernels_copy.cu -- host-boundary layout conversion on the device.
//
// The caller's arrays use the reference layout (IDX = ijk_ofs + k +
// j*jmult + i*imult, stencils.h:5, grid.cpp:20-24); the kernels use the
// library layout (st3d_internal.h).  A strided host<->device copy of ~1M rows
// of a few KB each runs far below the link rate, so transfers go through a
// staging buffer in the reference layout instead:
//   upload:   one contiguous host->device copy of the whole host array, then
//             k_ref_to_dev scatters the region the stencil can read (interior
//             plus up to 4 halo planes/rows and up to `pk` halo points along
//             k) into the library layout;
// (device arrays and pinned host arrays are read and written by these kernels
// themselves, without the staging buffer)
//   download: k_dev_to_ref gathers every interior row together with its k
//             halo into the staging buffer, then one 2-D copy moves, per
//             i-plane, the span of the interior rows (ys rows of jmult
//             points) back to the host.  The j-halo rows and i-halo planes of
//             the host array are not written; the k-halo points inside the
//             span are written with the values uploaded for them.
#include "st3d_internal.h"

namespace st3d {

namespace {

// A transfer works on planes: blockIdx.y is the plane, and the plane's rows
// (each `kv` words of W points, halos included) form one flat run that the
// blocks cut into pieces of kCopyBlock * kCopyUnroll words, so short rows fill
// the blocks as well as long ones (one block a row left 3/4 of the threads
// idle on 200-point rows).  A thread moves kCopyUnroll words, loads first:
// bound by HBM (1024^3 FP32, 16-byte words: 1.45 ms an array, 6.0 TB/s,
// against 1.70 ms for one block a row with 4-byte words) or by the host link,
// which needs several transfers in flight per thread.
constexpr int kCopyUnroll = 4;
constexpr int kCopyBlock = 256;

// Row and word of the flat run's element `first + m`, the block's first
// element split once into (row, rest).
struct RowRun {
  long long row0;
  uint32_t rest, kv;
  __device__ __forceinline__ RowRun(long long first, uint32_t kv_) : kv(kv_) {
    if (first >> 32) {
      row0 = first / kv_;
      rest = (uint32_t)(first - row0 * kv_);
    } else {
      const uint32_t q = (uint32_t)first / kv_;
      row0 = q;
      rest = (uint32_t)first - q * kv_;
    }
  }
  __device__ __forceinline__ void at(uint32_t m, long long* row, uint32_t* word) const {
    const uint32_t x = rest + m, q = x / kv;
    *row = row0 + q;
    *word = x - q * kv;
  }
};

// V: the word moved (T itself or 16 bytes of T), W points of T.
template <typename V, int W>
__global__ void __launch_bounds__(kCopyBlock)
    k_ref_to_dev(Layout L, RefGeom R, const V* __restrict__ stage, V* __restrict__ dst, int hx, int hy,
                 int hz) {
  const uint32_t kv = (uint32_t)(R.zs + 2 * hz) / W;
  const long long n = (long long)(R.ys + 2 * hy) * kv;
  const long long first = (long long)blockIdx.x * (kCopyBlock * kCopyUnroll);
  const int i = (int)blockIdx.y - hx;
  const RowRun run(first, kv);
  const long long splane = R.ijk_ofs + (long long)i * R.imult - (long long)hy * R.jmult - hz;
  const long long dplane =
      ((long long)(i + (int)L.pi) * L.nj + ((int)L.pj - hy)) * L.nk + (int)L.pk - hz;
  V x[kCopyUnroll];
  long long to[kCopyUnroll];
#pragma unroll
  for (int m = 0; m < kCopyUnroll; ++m) {
    const uint32_t y = threadIdx.x + m * kCopyBlock;
    long long row;
    uint32_t word;
    run.at(y, &row, &word);
    to[m] = -1;
    if (first + y < n) {
      x[m] = stage[(splane + row * R.jmult) / W + word];
      to[m] = (dplane + row * (long long)L.nk) / W + word;
    }
  }
#pragma unroll
  for (int m = 0; m < kCopyUnroll; ++m)
    if (to[m] >= 0) dst[to[m]] = x[m];
}

template <typename V, int W>
__global__ void __launch_bounds__(kCopyBlock)
    k_dev_to_ref(Layout L, RefGeom R, const V* __restrict__ src, V* __restrict__ stage, int hz) {
  const uint32_t kv = (uint32_t)(R.zs + 2 * hz) / W;
  const long long n = (long long)R.ys * kv;
  const long long first = (long long)blockIdx.x * (kCopyBlock * kCopyUnroll);
  const int i = (int)blockIdx.y;
  const RowRun run(first, kv);
  const long long splane = ((long long)(i + (int)L.pi) * L.nj + (int)L.pj) * L.nk + (int)L.pk - hz;
  const long long dplane = R.ijk_ofs + (long long)i * R.imult - hz;
  V x[kCopyUnroll];
  long long to[kCopyUnroll];
#pragma unroll
  for (int m = 0; m < kCopyUnroll; ++m) {
    const uint32_t y = threadIdx.x + m * kCopyBlock;
    long long row;
    uint32_t word;
    run.at(y, &row, &word);
    to[m] = -1;
    if (first + y < n) {
      x[m] = src[(splane + row * (long long)L.nk) / W + word];
      to[m] = (dplane + row * R.jmult) / W + word;
    }
  }
#pragma unroll
  for (int m = 0; m < kCopyUnroll; ++m)
    if (to[m] >= 0) stage[to[m]] = x[m];
}

// Whole 16-byte words on both sides: rows of the caller's array a multiple of
// W points long, a k halo that leaves the device rows' starts on a word (the
// pads and pitches are multiples of 128 bytes), both bases 16-byte aligned.
bool rows_in_words(int W, const Layout& L, const RefGeom& R, int hz, const void* a, const void* b) {
  return R.jmult % W == 0 && R.ijk_ofs % W == hz % W && ((int)L.pk - hz) % W == 0 &&
         (R.zs + 2 * hz) % W == 0 &&
         (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) % 16 == 0;
}

dim3 run_grid(long long rows, long long klen, int W, unsigned planes) {
  const long long piece = kCopyBlock * kCopyUnroll;
  return dim3((unsigned)((rows * (klen / W) + piece - 1) / piece), planes, 1);
}

}  // namespace

cudaError_t launch_ref_to_dev(int eb, const Layout& L, const RefGeom& R, const void* stage,
                              void* dst, int hx, int hy, int hz, cudaStream_t stream) {
  if (eb != 4 && eb != 8) return cudaErrorInvalidValue;
  const int W = 16 / eb;
  const unsigned planes = (unsigned)(R.xs + 2 * hx);
  const long long rows = R.ys + 2 * hy, klen = R.zs + 2 * hz;
  if (planes > 65535) return cudaErrorInvalidConfiguration;
  if (rows_in_words(W, L, R, hz, stage, dst)) {
    const dim3 grid = run_grid(rows, klen, W, planes);
    if (eb == 4)
      k_ref_to_dev<float4, 4><<<grid, kCopyBlock, 0, stream>>>(L, R, (const float4*)stage, (float4*)dst, hx, hy, hz);
    else
      k_ref_to_dev<double2, 2><<<grid, kCopyBlock, 0, stream>>>(L, R, (const double2*)stage, (double2*)dst, hx, hy, hz);
  } else {
    const dim3 grid = run_grid(rows, klen, 1, planes);
    if (eb == 4)
      k_ref_to_dev<float, 1><<<grid, kCopyBlock, 0, stream>>>(L, R, (const float*)stage, (float*)dst, hx, hy, hz);
    else
      k_ref_to_dev<double, 1><<<grid, kCopyBlock, 0, stream>>>(L, R, (const double*)stage, (double*)dst, hx, hy, hz);
  }
  return cudaGetLastError();
}

cudaError_t launch_dev_to_ref(int eb, const Layout& L, const RefGeom& R, const void* src,
                              void* stage, int hz, cudaStream_t stream) {
  if (eb != 4 && eb != 8) return cudaErrorInvalidValue;
  const int W = 16 / eb;
  const unsigned planes = (unsigned)R.xs;
  const long long rows = R.ys, klen = R.zs + 2 * hz;
  if (planes > 65535) return cudaErrorInvalidConfiguration;
  if (rows_in_words(W, L, R, hz, src, stage)) {
    const dim3 grid = run_grid(rows, klen, W, planes);
    if (eb == 4)
      k_dev_to_ref<float4, 4><<<grid, kCopyBlock, 0, stream>>>(L, R, (const float4*)src, (float4*)stage, hz);
    else
      k_dev_to_ref<double2, 2><<<grid, kCopyBlock, 0, stream>>>(L, R, (const double2*)src, (double2*)stage, hz);
  } else {
    const dim3 grid = run_grid(rows, klen, 1, planes);
    if (eb == 4)
      k_dev_to_ref<float, 1><<<grid, kCopyBlock, 0, stream>>>(L, R, (const float*)src, (float*)stage, hz);
    else
      k_dev_to_ref<double, 1><<<grid, kCopyBlock, 0, stream>>>(L, R, (const double*)src, (double*)stage, hz);
  }
  return cudaGetLastError();
}

}  // namespace st3d

// ---------------------------------------------------------------------------
// 16-bit storage (st3d_f16.cuh): host arrays stay float; the device keeps a
// 16-bit word per point (plus a low byte in the compensated form) and a
// power-of-two scale per i-plane.
// ---------------------------------------------------------------------------
#include "st3d_f16.cuh"

namespace st3d {

namespace {

template <int KIND>
__device__ __forceinline__ float word_to_float(uint16_t b) {
  if (KIND == 0) return __half2float(__ushort_as_half(b));
  return __uint_as_float((uint32_t)b << 16);
}
template <int KIND>
__device__ __forceinline__ uint16_t float_to_word(float x) {
  if (KIND == 0) return __half_as_ushort(__float2half_rn(x));
  return __bfloat16_as_ushort(__float2bfloat16_rn(x));
}

// Per-plane maxima of |x| over the interior (float bits, atomicMax) and the
// maximum over the halo points the stencil reads; x = stage - stage2 when
// stage2 is given (the halo check then covers both arrays).
__global__ void k_plane_max_ref(RefGeom R, const float* __restrict__ stage,
                                const float* __restrict__ stage2, uint32_t* __restrict__ M,
                                uint32_t* __restrict__ halo_max, int hx, int hy, int hz) {
  const int kk = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = (int)blockIdx.y - hy;
  const int i = (int)blockIdx.z - hx;
  const int k = kk - hz;
  float m_in = 0.0f, m_halo = 0.0f;
  if (kk < R.zs + 2 * hz) {
    const long long s = R.ijk_ofs + (long long)i * R.imult + (long long)j * R.jmult + k;
    const float a = stage[s];
    const float b = stage2 ? stage2[s] : 0.0f;
    const bool inner = i >= 0 && i < R.xs && j >= 0 && j < R.ys && k >= 0 && k < R.zs;
    if (inner) m_in = fabsf(a - b); else m_halo = fmaxf(fabsf(a), fabsf(b));
  }
  const uint32_t a = __reduce_max_sync(0xffffffffu, __float_as_uint(m_in));
  const uint32_t b = __reduce_max_sync(0xffffffffu, __float_as_uint(m_halo));
  if ((threadIdx.x & 31) == 0) {
    if (a && i >= 0 && i < R.xs) atomicMax(&M[i], a);
    if (b) atomicMax(halo_max, b);
  }
}

// Scatter + encode: staging (reference layout, float) -> words (+ low bytes)
// in the library layout, the plane's scale from its maximum.
// With lo16 (FP16 words), the lo word of the hi/lo pair: fp16(xs - hi).
template <int KIND, bool HILO>
__global__ void k_ref_to_dev16(Layout L, RefGeom R, const float* __restrict__ stage,
                               const float* __restrict__ stage2, uint16_t* __restrict__ hi,
                               int8_t* __restrict__ lo, const uint32_t* __restrict__ M,
                               int* __restrict__ E, int hx, int hy, int hz,
                               uint16_t* __restrict__ lo16) {
  const int kk = blockIdx.x * blockDim.x + threadIdx.x;
  if (kk >= R.zs + 2 * hz) return;
  const int j = (int)blockIdx.y - hy;
  const int i = (int)blockIdx.z - hx;
  const int k = kk - hz;
  const bool plane_in = i >= 0 && i < R.xs;
  const int e = plane_in ? scale_exponent(__uint_as_float(M[i])) : 0;
  if (plane_in && kk == 0 && blockIdx.y == 0) E[i] = e;
  const long long s = R.ijk_ofs + (long long)i * R.imult + (long long)j * R.jmult + k;
  const float xs = (stage2 ? stage[s] - stage2[s] : stage[s]) * exp2i(-e);
  const long long d = ((long long)(i + (int)L.pi) * L.nj + (j + (int)L.pj)) * L.nk + (k + (int)L.pk);
  const uint16_t w = float_to_word<KIND>(xs);
  hi[d] = w;
  if (lo16) lo16[d] = float_to_word<KIND>(xs - word_to_float<KIND>(w));
  if (HILO) {
    const float r = xs - word_to_float<KIND>(w);
    int eb = (w >> 10) & 0x1f;
    if (eb == 0) eb = 1;
    int q = __float2int_rn(r * exp2i(33 - eb));
    q = q > 127 ? 127 : (q < -127 ? -127 : q);
    lo[d] = (int8_t)q;
  }
}

// Gather + decode: words (+ low bytes) -> staging (reference layout, float),
// interior rows with their k halo.
template <int KIND, bool HILO>
__global__ void k_dev16_to_ref(Layout L, RefGeom R, const uint16_t* __restrict__ hi,
                               const int8_t* __restrict__ lo, const int* __restrict__ E,
                               float* __restrict__ stage, int hz) {
  const int kk = blockIdx.x * blockDim.x + threadIdx.x;
  if (kk >= R.zs + 2 * hz) return;
  const int j = (int)blockIdx.y;
  const int i = (int)blockIdx.z;
  const int k = kk - hz;
  const long long s = ((long long)(i + (int)L.pi) * L.nj + (j + (int)L.pj)) * L.nk + (k + (int)L.pk);
  const uint16_t w = hi[s];
  float x = word_to_float<KIND>(w);
  if (HILO) x = __fmaf_rn((float)lo[s], ulp256_f16(w), x);
  stage[R.ijk_ofs + (long long)i * R.imult + (long long)j * R.jmult + k] = x * exp2i(E[i]);
}

// Delta form -> float: u = dec(U), or v = dec(U) - dec(D).
template <int KIND>
__global__ void k_delta_to_ref(Layout L, RefGeom R, const uint16_t* __restrict__ u,
                               const int* __restrict__ Eu, const uint16_t* __restrict__ d,
                               const int* __restrict__ Ed, bool minus_d, float* __restrict__ stage,
                               int hz, const uint16_t* __restrict__ ul) {
  const int kk = blockIdx.x * blockDim.x + threadIdx.x;
  if (kk >= R.zs + 2 * hz) return;
  const int j = (int)blockIdx.y;
  const int i = (int)blockIdx.z;
  const int k = kk - hz;
  const long long s = ((long long)(i + (int)L.pi) * L.nj + (j + (int)L.pj)) * L.nk + (k + (int)L.pk);
  float x = word_to_float<KIND>(u[s]);
  if (ul) x = x + word_to_float<KIND>(ul[s]);  // exact: the pair holds <= 22 bits
  x = x * exp2i(Eu[i]);
  if (minus_d) x = x - word_to_float<KIND>(d[s]) * exp2i(Ed[i]);
  stage[R.ijk_ofs + (long long)i * R.imult + (long long)j * R.jmult + k] = x;
}

}  // namespace

cudaError_t launch_plane_max_ref(const RefGeom& R, const float* stage, uint32_t* M,
                                 uint32_t* halo_max, int hx, int hy, int hz, cudaStream_t stream,
                                 const float* stage2) {
  dim3 block(256);
  dim3 grid((R.zs + 2 * hz + 255) / 256, R.ys + 2 * hy, R.xs + 2 * hx);
  if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidConfiguration;
  k_plane_max_ref<<<grid, block, 0, stream>>>(R, stage, stage2, M, halo_max, hx, hy, hz);
  return cudaGetLastError();
}

cudaError_t launch_ref_to_dev16(int storage, const Layout& L, const RefGeom& R, const float* stage,
                                uint16_t* hi, int8_t* lo, const uint32_t* M, int* E, int hx, int hy,
                                int hz, cudaStream_t stream, const float* stage2, uint16_t* lo16) {
  dim3 block(256);
  dim3 grid((R.zs + 2 * hz + 255) / 256, R.ys + 2 * hy, R.xs + 2 * hx);
  if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidConfiguration;
  if (lo16 && storage != ST3D_F16) return cudaErrorInvalidValue;
  if (storage == ST3D_F16)
    k_ref_to_dev16<0, false><<<grid, block, 0, stream>>>(L, R, stage, stage2, hi, lo, M, E, hx, hy, hz, lo16);
  else if (storage == ST3D_BF16)
    k_ref_to_dev16<1, false><<<grid, block, 0, stream>>>(L, R, stage, stage2, hi, lo, M, E, hx, hy, hz, lo16);
  else if (storage == ST3D_F16_HILO)
    k_ref_to_dev16<0, true><<<grid, block, 0, stream>>>(L, R, stage, stage2, hi, lo, M, E, hx, hy, hz, lo16);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_delta_to_ref(int storage, const Layout& L, const RefGeom& R, const uint16_t* u,
                                const int* Eu, const uint16_t* d, const int* Ed, bool minus_d,
                                float* stage, int hz, cudaStream_t stream, const uint16_t* ul) {
  dim3 block(256);
  dim3 grid((R.zs + 2 * hz + 255) / 256, R.ys, R.xs);
  if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidConfiguration;
  if (ul && storage != ST3D_F16) return cudaErrorInvalidValue;
  if (storage == ST3D_F16)
    k_delta_to_ref<0><<<grid, block, 0, stream>>>(L, R, u, Eu, d, Ed, minus_d, stage, hz, ul);
  else if (storage == ST3D_BF16)
    k_delta_to_ref<1><<<grid, block, 0, stream>>>(L, R, u, Eu, d, Ed, minus_d, stage, hz, ul);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_dev16_to_ref(int storage, const Layout& L, const RefGeom& R, const uint16_t* hi,
                                const int8_t* lo, const int* E, float* stage, int hz,
                                cudaStream_t stream) {
  dim3 block(256);
  dim3 grid((R.zs + 2 * hz + 255) / 256, R.ys, R.xs);
  if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidConfiguration;
  if (storage == ST3D_F16)
    k_dev16_to_ref<0, false><<<grid, block, 0, stream>>>(L, R, hi, lo, E, stage, hz);
  else if (storage == ST3D_BF16)
    k_dev16_to_ref<1, false><<<grid, block, 0, stream>>>(L, R, hi, lo, E, stage, hz);
  else if (storage == ST3D_F16_HILO)
    k_dev16_to_ref<0, true><<<grid, block, 0, stream>>>(L, R, hi, lo, E, stage, hz);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

}  // namespace st3d
