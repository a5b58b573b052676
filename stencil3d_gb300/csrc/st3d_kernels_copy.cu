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
// blocks cut into pieces of kCopyBlock * kRunUnroll words, so short rows fill
// the blocks as well as long ones (one block a row left 3/4 of the threads
// idle on 200-point rows).  A thread moves kRunUnroll words, loads first:
// bound by HBM (1024^3 FP32, 16-byte words: 1.45 ms an array, 6.0 TB/s,
// against 1.70 ms for one block a row with 4-byte words) or by the host link,
// which needs several transfers in flight per thread.
constexpr int kCopyUnroll = 4;
constexpr int kCopyBlock = 256;
// Rows that are not whole 16-byte words move element by element, twice as many
// a thread: with four the bytes in flight bound them (525 x 219 x 387 FP32 device
// array, up / down: 4 elements 4110 / 4047 GB/s, 8 5171 / 5121, 12 5491 / 5074,
// 16 5527 / 4533).
template <int W>
constexpr int kRunUnroll = W == 1 ? 2 * kCopyUnroll : kCopyUnroll;

// Row and word of the flat run's element `first + m`, the block's first
// element split once into (row, rest).
struct RowRun {
  long long row0;
  uint32_t rest, kv, inv;  // inv: ceil(2^32 / kv), exact while (kv + 4096) * kv < 2^32; 0: divide
  __device__ __forceinline__ RowRun(long long first, uint32_t kv_)
      : kv(kv_), inv(kv_ > 1 && kv_ < 60000u ? 0xffffffffu / kv_ + 1u : 0u) {
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
    const uint32_t x = rest + m, q = inv ? __umulhi(x, inv) : x / kv;
    *row = row0 + q;
    *word = x - q * kv;
  }
};

// The caller's side of a plane is one contiguous span; the pieces are shifted so
// that their warps' accesses to it start on 128-byte lines (over the host link a
// line written in two parts costs two transfers: 525 x 219 x 387 to a pinned
// array 144 GB/s unshifted).
template <typename V>
__device__ __forceinline__ int line_shift(const V* p) {
  return (int)((reinterpret_cast<uintptr_t>(p) / sizeof(V)) % (128 / sizeof(V)));
}

// V: the word moved (T itself or 16 bytes of T), W points of T.
template <typename V, int W, bool UP>
__device__ __forceinline__ void copy_plane_piece(const Layout& L, const RefGeom& R, V* dev, V* ref, int i, int hy,
                                                 int hz) {
  constexpr int U = kRunUnroll<W>;
  const uint32_t kv = (uint32_t)(R.zs + 2 * hz) / W;
  const long long n = (long long)(R.ys + 2 * hy) * kv;
  V* span = ref + (R.ijk_ofs + (long long)i * R.imult - (long long)hy * R.jmult - hz) / W;
  V* plane = dev + (((long long)(i + (int)L.pi) * L.nj + ((int)L.pj - hy)) * L.nk + (int)L.pk - hz) / W;
  const long long at = (long long)blockIdx.x * (kCopyBlock * U) - line_shift(span);
  const long long first = at > 0 ? at : 0;
  const int lead = (int)(first - at);
  const RowRun run(first, kv);
  V x[U];
  long long to[U];
#pragma unroll
  for (int m = 0; m < U; ++m) {
    const int y = (int)threadIdx.x + m * kCopyBlock - lead;
    to[m] = -1;
    if (y >= 0 && first + y < n) {
      long long row;
      uint32_t word;
      run.at((uint32_t)y, &row, &word);
      const long long d = row * (long long)(L.nk / W) + word;
      if (UP) {
        x[m] = span[first + y];
        to[m] = d;
      } else {
        x[m] = plane[d];
        to[m] = first + y;
      }
    }
  }
#pragma unroll
  for (int m = 0; m < U; ++m)
    if (to[m] >= 0) (UP ? plane : span)[to[m]] = x[m];
}

template <typename V, int W>
__global__ void __launch_bounds__(kCopyBlock)
    k_ref_to_dev(Layout L, RefGeom R, const V* __restrict__ stage, V* __restrict__ dst, int hx, int hy,
                 int hz) {
  copy_plane_piece<V, W, true>(L, R, dst, const_cast<V*>(stage), (int)blockIdx.y - hx, hy, hz);
}

template <typename V, int W>
__global__ void __launch_bounds__(kCopyBlock)
    k_dev_to_ref(Layout L, RefGeom R, const V* __restrict__ src, V* __restrict__ stage, int hz) {
  copy_plane_piece<V, W, false>(L, R, const_cast<V*>(src), stage, (int)blockIdx.y, 0, hz);
}

// Whole 16-byte words on both sides: rows of the caller's array a multiple of
// W points long, a k halo that leaves the device rows' starts on a word (the
// pads and pitches are multiples of 128 bytes), both bases 16-byte aligned.
bool rows_in_words(int W, const Layout& L, const RefGeom& R, int hz, const void* a, const void* b) {
  return R.jmult % W == 0 && R.ijk_ofs % W == hz % W && ((int)L.pk - hz) % W == 0 &&
         (R.zs + 2 * hz) % W == 0 &&
         (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) % 16 == 0;
}

dim3 run_grid(long long rows, long long klen, int W, unsigned planes, int unroll = kCopyUnroll) {
  const long long piece = kCopyBlock * unroll, shift = 31;  // words a piece may be shifted by
  return dim3((unsigned)((rows * (klen / W) + shift + piece - 1) / piece), planes, 1);
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
    const dim3 grid = run_grid(rows, klen, 1, planes, kRunUnroll<1>);
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
    const dim3 grid = run_grid(rows, klen, 1, planes, kRunUnroll<1>);
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

// The 16-bit transfers run on the same flat runs of a plane's rows, W = 4
// points a word (16 bytes of floats, 8 of 16-bit words) where the rows are
// whole words, else W = 1.
template <int W>
struct Floats {
  float x[W];
};
template <int W>
__device__ __forceinline__ Floats<W> load_floats(const float* p) {
  Floats<W> f;
  if constexpr (W == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f.x[0] = v.x; f.x[1] = v.y; f.x[2] = v.z; f.x[3] = v.w;
  } else {
    f.x[0] = *p;
  }
  return f;
}
template <int W>
__device__ __forceinline__ void store_floats(float* p, const Floats<W>& f) {
  if constexpr (W == 4)
    *reinterpret_cast<float4*>(p) = make_float4(f.x[0], f.x[1], f.x[2], f.x[3]);
  else
    *p = f.x[0];
}
template <int W>
struct Words {
  uint16_t w[W];
};
template <int W>
__device__ __forceinline__ Words<W> load_words(const uint16_t* p) {
  Words<W> r;
  if constexpr (W == 4) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    r.w[0] = (uint16_t)v.x; r.w[1] = (uint16_t)(v.x >> 16);
    r.w[2] = (uint16_t)v.y; r.w[3] = (uint16_t)(v.y >> 16);
  } else {
    r.w[0] = *p;
  }
  return r;
}
template <int W>
__device__ __forceinline__ void store_words(uint16_t* p, const Words<W>& r) {
  if constexpr (W == 4)
    *reinterpret_cast<uint2*>(p) = make_uint2((uint32_t)r.w[0] | ((uint32_t)r.w[1] << 16),
                                              (uint32_t)r.w[2] | ((uint32_t)r.w[3] << 16));
  else
    *p = r.w[0];
}

// Words a thread of the maximum kernel reads: one atomic per warp and 2048
// points.  512^3: 127 us (4.4 TB/s) against 1317 us with an atomic per 32
// points, which all met on one address a plane.  The encoder of the same
// fields takes 177 us (677 with one point a thread), the decoder 199 (618).
constexpr int kMaxUnroll = 16;

// Per-plane maxima of |x| over the interior (float bits, atomicMax) and the
// maximum over the halo points the stencil reads; x = stage - stage2 when
// stage2 is given (the halo check then covers both arrays).  With pair.Ma also
// those of |stage| alone; with pair.to / to2 the points read go on into the
// staging slots, so that a device array is read once for both (a copy of each
// array and two passes over them took 1.3 ms more of a 1024^3 upload).
template <int W>
__global__ void __launch_bounds__(kCopyBlock)
    k_plane_max_ref(RefGeom R, const float* __restrict__ stage, const float* __restrict__ stage2,
                    uint32_t* __restrict__ M, uint32_t* __restrict__ halo_max, PairMax pair, int hx, int hy,
                    int hz) {
  const uint32_t kv = (uint32_t)(R.zs + 2 * hz) / W;
  const long long n = (long long)(R.ys + 2 * hy) * kv;
  const long long first = (long long)blockIdx.x * (kCopyBlock * kMaxUnroll);
  const int i = (int)blockIdx.y - hx;
  const RowRun run(first, kv);
  const long long plane = R.ijk_ofs + (long long)i * R.imult - (long long)hy * R.jmult - hz;
  const bool in_plane = i >= 0 && i < R.xs;
  uint32_t m_in = 0u, m_a = 0u, m_halo = 0u, m_halo_a = 0u;
#pragma unroll 4
  for (int m = 0; m < kMaxUnroll; ++m) {
    const uint32_t y = threadIdx.x + m * kCopyBlock;
    if (first + y >= n) break;
    long long row;
    uint32_t word;
    run.at(y, &row, &word);
    const long long s = plane + row * R.jmult + (long long)word * W;
    const Floats<W> a = load_floats<W>(stage + s);
    Floats<W> b;
    if (stage2) {
      b = load_floats<W>(stage2 + s);
    } else {
#pragma unroll
      for (int c = 0; c < W; ++c) b.x[c] = 0.0f;
    }
    if (pair.to) store_floats<W>(pair.to + s, a);
    if (pair.to2) store_floats<W>(pair.to2 + s, b);
    const bool in_row = in_plane && row >= hy && row < hy + R.ys;
#pragma unroll
    for (int c = 0; c < W; ++c) {
      const int k = (int)(word * W) + c - hz;
      if (in_row && k >= 0 && k < R.zs) {
        m_in = max(m_in, __float_as_uint(fabsf(a.x[c] - b.x[c])));
        m_a = max(m_a, __float_as_uint(fabsf(a.x[c])));
      } else {
        m_halo = max(m_halo, __float_as_uint(fmaxf(fabsf(a.x[c]), fabsf(b.x[c]))));
        m_halo_a = max(m_halo_a, __float_as_uint(fmaxf(fabsf(a.x[c]), 0.0f)));  // a NaN passes, as in m_halo
      }
    }
  }
  const uint32_t a = __reduce_max_sync(0xffffffffu, m_in);
  const uint32_t b = __reduce_max_sync(0xffffffffu, m_halo);
  const bool lead = (threadIdx.x & 31) == 0;
  if (lead) {
    if (a && in_plane) atomicMax(&M[i], a);
    if (b) atomicMax(halo_max, b);
  }
  if (pair.Ma) {
    const uint32_t ua = __reduce_max_sync(0xffffffffu, m_a);
    const uint32_t ub = __reduce_max_sync(0xffffffffu, m_halo_a);
    if (lead && ua && in_plane) atomicMax(&pair.Ma[i], ua);
    if (lead && ub) atomicMax(halo_max + 1, ub);
  }
}

// U from stage (with ulo the lo words of the hi/lo pair too, fp16(xs - hi)) and
// D = stage - stage2 in one pass over the slots: what k_ref_to_dev16 writes for each.
template <int KIND, int W>
__global__ void __launch_bounds__(kCopyBlock)
    k_pair_to_dev16(Layout L, RefGeom R, const float* __restrict__ stage, const float* __restrict__ stage2,
                    uint16_t* __restrict__ uhi, uint16_t* __restrict__ ulo, uint16_t* __restrict__ dw,
                    const uint32_t* __restrict__ Mu, const uint32_t* __restrict__ Md, int* __restrict__ Eu,
                    int* __restrict__ Ed, int hx, int hy, int hz) {
  const uint32_t kv = (uint32_t)(R.zs + 2 * hz) / W;
  const long long n = (long long)(R.ys + 2 * hy) * kv;
  const long long first = (long long)blockIdx.x * (kCopyBlock * kCopyUnroll);
  const int i = (int)blockIdx.y - hx;
  const RowRun run(first, kv);
  const bool plane_in = i >= 0 && i < R.xs;
  const int eu = plane_in ? scale_exponent(__uint_as_float(Mu[i])) : 0;
  const int ed = plane_in ? scale_exponent(__uint_as_float(Md[i])) : 0;
  if (plane_in && blockIdx.x == 0 && threadIdx.x == 0) {
    Eu[i] = eu;
    Ed[i] = ed;
  }
  const float inv_u = exp2i(-eu), inv_d = exp2i(-ed);
  const long long splane = R.ijk_ofs + (long long)i * R.imult - (long long)hy * R.jmult - hz;
  const long long dplane =
      ((long long)(i + (int)L.pi) * L.nj + ((int)L.pj - hy)) * L.nk + (int)L.pk - hz;
#pragma unroll
  for (int m = 0; m < kCopyUnroll; ++m) {
    const uint32_t y = threadIdx.x + m * kCopyBlock;
    if (first + y >= n) break;
    long long row;
    uint32_t word;
    run.at(y, &row, &word);
    const long long s = splane + row * R.jmult + (long long)word * W;
    const long long d = dplane + row * (long long)L.nk + (long long)word * W;
    const Floats<W> a = load_floats<W>(stage + s), b = load_floats<W>(stage2 + s);
    Words<W> h, l, q;
#pragma unroll
    for (int c = 0; c < W; ++c) {
      const float xs = a.x[c] * inv_u;
      h.w[c] = float_to_word<KIND>(xs);
      l.w[c] = float_to_word<KIND>(xs - word_to_float<KIND>(h.w[c]));
      q.w[c] = float_to_word<KIND>((a.x[c] - b.x[c]) * inv_d);
    }
    store_words<W>(uhi + d, h);
    if (ulo) store_words<W>(ulo + d, l);
    store_words<W>(dw + d, q);
  }
}

// Scatter + encode: staging (reference layout, float) -> words (+ low bytes)
// in the library layout, the plane's scale from its maximum.
template <int KIND, bool HILO, int W>
__global__ void __launch_bounds__(kCopyBlock)
    k_ref_to_dev16(Layout L, RefGeom R, const float* __restrict__ stage,
                   const float* __restrict__ stage2, uint16_t* __restrict__ hi, int8_t* __restrict__ lo,
                   const uint32_t* __restrict__ M, int* __restrict__ E, int hx, int hy, int hz) {
  const uint32_t kv = (uint32_t)(R.zs + 2 * hz) / W;
  const long long n = (long long)(R.ys + 2 * hy) * kv;
  const long long first = (long long)blockIdx.x * (kCopyBlock * kCopyUnroll);
  const int i = (int)blockIdx.y - hx;
  const RowRun run(first, kv);
  const bool plane_in = i >= 0 && i < R.xs;
  const int e = plane_in ? scale_exponent(__uint_as_float(M[i])) : 0;
  if (plane_in && blockIdx.x == 0 && threadIdx.x == 0) E[i] = e;
  const float inv = exp2i(-e);
  const long long splane = R.ijk_ofs + (long long)i * R.imult - (long long)hy * R.jmult - hz;
  const long long dplane =
      ((long long)(i + (int)L.pi) * L.nj + ((int)L.pj - hy)) * L.nk + (int)L.pk - hz;
#pragma unroll
  for (int m = 0; m < kCopyUnroll; ++m) {
    const uint32_t y = threadIdx.x + m * kCopyBlock;
    if (first + y >= n) break;
    long long row;
    uint32_t word;
    run.at(y, &row, &word);
    const long long s = splane + row * R.jmult + (long long)word * W;
    const long long d = dplane + row * (long long)L.nk + (long long)word * W;
    Floats<W> x = load_floats<W>(stage + s);
    if (stage2) {
      const Floats<W> b = load_floats<W>(stage2 + s);
#pragma unroll
      for (int c = 0; c < W; ++c) x.x[c] = x.x[c] - b.x[c];
    }
    Words<W> h;
    int8_t q8[W];
#pragma unroll
    for (int c = 0; c < W; ++c) {
      const float xs = x.x[c] * inv;
      const uint16_t w = float_to_word<KIND>(xs);
      const float r = xs - word_to_float<KIND>(w);
      h.w[c] = w;
      if (HILO) {
        int eb = (w >> 10) & 0x1f;
        if (eb == 0) eb = 1;
        int q = __float2int_rn(r * exp2i(33 - eb));
        q = q > 127 ? 127 : (q < -127 ? -127 : q);
        q8[c] = (int8_t)q;
      }
    }
    store_words<W>(hi + d, h);
    if (HILO) {
      if constexpr (W == 4) {
        *reinterpret_cast<char4*>(lo + d) = make_char4(q8[0], q8[1], q8[2], q8[3]);
      } else {
        lo[d] = q8[0];
      }
    }
  }
}

// Gather + decode: words (+ low bytes) -> the reference layout (float),
// interior rows with their k halo.
template <int KIND, bool HILO, int W>
__global__ void __launch_bounds__(kCopyBlock)
    k_dev16_to_ref(Layout L, RefGeom R, const uint16_t* __restrict__ hi, const int8_t* __restrict__ lo,
                   const int* __restrict__ E, float* __restrict__ stage, int hz) {
  const uint32_t kv = (uint32_t)(R.zs + 2 * hz) / W;
  const long long n = (long long)R.ys * kv;
  const long long first = (long long)blockIdx.x * (kCopyBlock * kCopyUnroll);
  const int i = (int)blockIdx.y;
  const RowRun run(first, kv);
  const float sc = exp2i(E[i]);
  const long long splane = ((long long)(i + (int)L.pi) * L.nj + (int)L.pj) * L.nk + (int)L.pk - hz;
  const long long dplane = R.ijk_ofs + (long long)i * R.imult - hz;
#pragma unroll
  for (int m = 0; m < kCopyUnroll; ++m) {
    const uint32_t y = threadIdx.x + m * kCopyBlock;
    if (first + y >= n) break;
    long long row;
    uint32_t word;
    run.at(y, &row, &word);
    const long long s = splane + row * (long long)L.nk + (long long)word * W;
    const Words<W> w = load_words<W>(hi + s);
    Floats<W> x;
#pragma unroll
    for (int c = 0; c < W; ++c) {
      x.x[c] = word_to_float<KIND>(w.w[c]);
      if (HILO) x.x[c] = __fmaf_rn((float)lo[s + c], ulp256_f16(w.w[c]), x.x[c]);
      x.x[c] = x.x[c] * sc;
    }
    store_floats<W>(stage + dplane + row * R.jmult + (long long)word * W, x);
  }
}

// Delta form -> float: u = dec(U), or v = dec(U) - dec(D).
template <int KIND, int W>
__global__ void __launch_bounds__(kCopyBlock)
    k_delta_to_ref(Layout L, RefGeom R, const uint16_t* __restrict__ u, const int* __restrict__ Eu,
                   const uint16_t* __restrict__ d, const int* __restrict__ Ed, bool minus_d,
                   float* __restrict__ stage, int hz, const uint16_t* __restrict__ ul) {
  const uint32_t kv = (uint32_t)(R.zs + 2 * hz) / W;
  const long long n = (long long)R.ys * kv;
  const long long first = (long long)blockIdx.x * (kCopyBlock * kCopyUnroll);
  const int i = (int)blockIdx.y;
  const RowRun run(first, kv);
  const float su = exp2i(Eu[i]);
  const float sd = exp2i(Ed[i]);
  const long long splane = ((long long)(i + (int)L.pi) * L.nj + (int)L.pj) * L.nk + (int)L.pk - hz;
  const long long dplane = R.ijk_ofs + (long long)i * R.imult - hz;
#pragma unroll
  for (int m = 0; m < kCopyUnroll; ++m) {
    const uint32_t y = threadIdx.x + m * kCopyBlock;
    if (first + y >= n) break;
    long long row;
    uint32_t word;
    run.at(y, &row, &word);
    const long long s = splane + row * (long long)L.nk + (long long)word * W;
    const Words<W> wu = load_words<W>(u + s);
    Words<W> wl, wd;
    if (ul) wl = load_words<W>(ul + s);
    if (minus_d) wd = load_words<W>(d + s);
    Floats<W> x;
#pragma unroll
    for (int c = 0; c < W; ++c) {
      x.x[c] = word_to_float<KIND>(wu.w[c]);
      if (ul) x.x[c] = x.x[c] + word_to_float<KIND>(wl.w[c]);  // exact: the pair holds <= 22 bits
      x.x[c] = x.x[c] * su;
      if (minus_d) x.x[c] = x.x[c] - word_to_float<KIND>(wd.w[c]) * sd;
    }
    store_floats<W>(stage + dplane + row * R.jmult + (long long)word * W, x);
  }
}

// Whole words of four points (the 16-bit rows' pads and pitches are multiples
// of 64 points; their buffers are allocations of the context).
bool rows_in_fours(const Layout& L, const RefGeom& R, int hz, const float* a, const float* b) {
  return rows_in_words(4, L, R, hz, a, b ? b : a);
}

dim3 max_grid(long long rows, long long klen, int W, unsigned planes) {
  const long long piece = kCopyBlock * kMaxUnroll;
  return dim3((unsigned)((rows * (klen / W) + piece - 1) / piece), planes, 1);
}

}  // namespace

cudaError_t launch_plane_max_ref(const RefGeom& R, const float* stage, uint32_t* M,
                                 uint32_t* halo_max, int hx, int hy, int hz, cudaStream_t stream,
                                 const float* stage2, const PairMax& pair) {
  const unsigned planes = (unsigned)(R.xs + 2 * hx);
  const long long rows = R.ys + 2 * hy, klen = R.zs + 2 * hz;
  if (planes > 65535) return cudaErrorInvalidConfiguration;
  const uintptr_t at = reinterpret_cast<uintptr_t>(stage) | reinterpret_cast<uintptr_t>(stage2) |
                       reinterpret_cast<uintptr_t>(pair.to) | reinterpret_cast<uintptr_t>(pair.to2);
  if (R.jmult % 4 == 0 && R.ijk_ofs % 4 == hz % 4 && klen % 4 == 0 && at % 16 == 0)
    k_plane_max_ref<4><<<max_grid(rows, klen, 4, planes), kCopyBlock, 0, stream>>>(R, stage, stage2, M, halo_max,
                                                                                   pair, hx, hy, hz);
  else
    k_plane_max_ref<1><<<max_grid(rows, klen, 1, planes), kCopyBlock, 0, stream>>>(R, stage, stage2, M, halo_max,
                                                                                   pair, hx, hy, hz);
  return cudaGetLastError();
}

cudaError_t launch_pair_to_dev16(int storage, const Layout& L, const RefGeom& R, const float* stage,
                                 const float* stage2, uint16_t* uhi, uint16_t* ulo, uint16_t* dw,
                                 const uint32_t* Mu, const uint32_t* Md, int* Eu, int* Ed, int hx, int hy,
                                 int hz, cudaStream_t stream) {
  const unsigned planes = (unsigned)(R.xs + 2 * hx);
  const long long rows = R.ys + 2 * hy, klen = R.zs + 2 * hz;
  if (planes > 65535) return cudaErrorInvalidConfiguration;
  if (ulo && storage != ST3D_F16) return cudaErrorInvalidValue;
  const bool fours = rows_in_fours(L, R, hz, stage, stage2);
  const dim3 grid = run_grid(rows, klen, fours ? 4 : 1, planes);
#define ST3D_ENCODE(KIND, W)                                                                          \
  k_pair_to_dev16<KIND, W><<<grid, kCopyBlock, 0, stream>>>(L, R, stage, stage2, uhi, ulo, dw, Mu, Md, \
                                                            Eu, Ed, hx, hy, hz)
  if (storage == ST3D_F16 && fours)
    ST3D_ENCODE(0, 4);
  else if (storage == ST3D_F16)
    ST3D_ENCODE(0, 1);
  else if (storage == ST3D_BF16 && fours)
    ST3D_ENCODE(1, 4);
  else if (storage == ST3D_BF16)
    ST3D_ENCODE(1, 1);
  else
    return cudaErrorInvalidValue;
#undef ST3D_ENCODE
  return cudaGetLastError();
}

cudaError_t launch_ref_to_dev16(int storage, const Layout& L, const RefGeom& R, const float* stage,
                                uint16_t* hi, int8_t* lo, const uint32_t* M, int* E, int hx, int hy,
                                int hz, cudaStream_t stream, const float* stage2) {
  const unsigned planes = (unsigned)(R.xs + 2 * hx);
  const long long rows = R.ys + 2 * hy, klen = R.zs + 2 * hz;
  if (planes > 65535) return cudaErrorInvalidConfiguration;
  const bool fours = rows_in_fours(L, R, hz, stage, stage2);
  const dim3 grid = run_grid(rows, klen, fours ? 4 : 1, planes);
#define ST3D_ENCODE(KIND, HILO)                                                                       \
  do {                                                                                                \
    if (fours)                                                                                        \
      k_ref_to_dev16<KIND, HILO, 4><<<grid, kCopyBlock, 0, stream>>>(L, R, stage, stage2, hi, lo, M,  \
                                                                     E, hx, hy, hz);                  \
    else                                                                                              \
      k_ref_to_dev16<KIND, HILO, 1><<<grid, kCopyBlock, 0, stream>>>(L, R, stage, stage2, hi, lo, M,  \
                                                                     E, hx, hy, hz);                  \
  } while (0)
  if (storage == ST3D_F16)
    ST3D_ENCODE(0, false);
  else if (storage == ST3D_BF16)
    ST3D_ENCODE(1, false);
  else if (storage == ST3D_F16_HILO)
    ST3D_ENCODE(0, true);
  else
    return cudaErrorInvalidValue;
#undef ST3D_ENCODE
  return cudaGetLastError();
}

cudaError_t launch_delta_to_ref(int storage, const Layout& L, const RefGeom& R, const uint16_t* u,
                                const int* Eu, const uint16_t* d, const int* Ed, bool minus_d,
                                float* stage, int hz, cudaStream_t stream, const uint16_t* ul) {
  const unsigned planes = (unsigned)R.xs;
  if (planes > 65535) return cudaErrorInvalidConfiguration;
  if (ul && storage != ST3D_F16) return cudaErrorInvalidValue;
  const bool fours = rows_in_fours(L, R, hz, stage, nullptr);
  const dim3 grid = run_grid(R.ys, R.zs + 2 * hz, fours ? 4 : 1, planes);
  if (storage == ST3D_F16 && fours)
    k_delta_to_ref<0, 4><<<grid, kCopyBlock, 0, stream>>>(L, R, u, Eu, d, Ed, minus_d, stage, hz, ul);
  else if (storage == ST3D_F16)
    k_delta_to_ref<0, 1><<<grid, kCopyBlock, 0, stream>>>(L, R, u, Eu, d, Ed, minus_d, stage, hz, ul);
  else if (storage == ST3D_BF16 && fours)
    k_delta_to_ref<1, 4><<<grid, kCopyBlock, 0, stream>>>(L, R, u, Eu, d, Ed, minus_d, stage, hz, ul);
  else if (storage == ST3D_BF16)
    k_delta_to_ref<1, 1><<<grid, kCopyBlock, 0, stream>>>(L, R, u, Eu, d, Ed, minus_d, stage, hz, ul);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_dev16_to_ref(int storage, const Layout& L, const RefGeom& R, const uint16_t* hi,
                                const int8_t* lo, const int* E, float* stage, int hz,
                                cudaStream_t stream) {
  const unsigned planes = (unsigned)R.xs;
  if (planes > 65535) return cudaErrorInvalidConfiguration;
  const bool fours = rows_in_fours(L, R, hz, stage, nullptr);
  const dim3 grid = run_grid(R.ys, R.zs + 2 * hz, fours ? 4 : 1, planes);
#define ST3D_DECODE(KIND, HILO)                                                                     \
  do {                                                                                              \
    if (fours)                                                                                      \
      k_dev16_to_ref<KIND, HILO, 4><<<grid, kCopyBlock, 0, stream>>>(L, R, hi, lo, E, stage, hz);   \
    else                                                                                            \
      k_dev16_to_ref<KIND, HILO, 1><<<grid, kCopyBlock, 0, stream>>>(L, R, hi, lo, E, stage, hz);   \
  } while (0)
  if (storage == ST3D_F16)
    ST3D_DECODE(0, false);
  else if (storage == ST3D_BF16)
    ST3D_DECODE(1, false);
  else if (storage == ST3D_F16_HILO)
    ST3D_DECODE(0, true);
  else
    return cudaErrorInvalidValue;
#undef ST3D_DECODE
  return cudaGetLastError();
}

}  // namespace st3d
