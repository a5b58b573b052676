// st3d_kernels_brick.cu -- many FP32 wave steps of a small grid in one launch,
// the fields kept in shared memory.
//
// A grid of up to about 110 points a side is bound by what a step costs beside
// its work: one launch a step is 6.4 us at 64^3, and in the multi-step wave
// kernel each level waits some 6 us for the one before.  Here each CTA (one an
// SM, all resident: a cooperative launch) keeps a brick of the grid -- bi planes
// x bj rows x all of k -- of u, v and s in shared memory for all steps of the
// launch.  A step is:
//   1. wait until the four neighbouring bricks have published the step before
//      (one word each, 128 bytes apart; acquire, gpu scope);
//   2. read R planes and R rows of theirs from the field into the brick's halo;
//   3. form the new values in place of v (u and v swap roles), and write to the
//      field the planes and rows the neighbours need (every point in the last
//      two steps, whose levels are the result);
//   4. publish (release, gpu scope).
// A neighbour's cells of level t are overwritten by level t + 2, which it forms
// after this brick has published level t + 1, that is after step 2 above: no
// further waiting.  The chain store, publish, poll, read is what a step costs,
// about 2 us, beside the brick's points (20 steps, before -> now: 7 points 64^3
// 128.5 -> 52.0 us, 96^3 147 -> 76; 25 points 64^3 199 -> 73).  Bricks are at least R planes and rows, so a halo comes from one
// neighbour.
//
// Same operations on every point as the one-step kernel, in the same order: bit
// for bit its result.  Waits give up after `limit_ns` (status word, and an abort
// word the other bricks look at).
#include "st3d_internal.h"
#include "st3d_p4.cuh"
#include "st3d_tma.cuh"

namespace st3d {

namespace {

constexpr int kBrThreads = 512;
constexpr int kBrPad = 32;  // ints between two bricks' words

struct BrickArgs {
  Geom g;
  Coefs<float> cf;
  float* buf[2];
  const float* s;
  int ub0, steps;
  const int* ub_dev;     // see StepFeed
  const float* amps_dev;
  int amp_stride;
  int bi, bj, nbi, nbj;  // brick extents, bricks along i and j
  int zq, pitch;         // quads of a row; floats of a row in shared memory
  int src_i, src_j, src_k;
  int* words;            // [brick]: levels published, kBrPad apart
  int* abort_word;
  uint64_t limit_ns;
  uint32_t* status;
  float amps[kWaveSteps];
};

__device__ __forceinline__ int b_ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void b_st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// x / d for x * d < 2^32 (quads of a brick: x < 2^15, d < 2^11): the product
// with ceil(2^32 / d), upper word.
struct Div {
  uint32_t d, m;
  __device__ __forceinline__ explicit Div(int by) : d((uint32_t)by), m(by > 1 ? 0xffffffffu / (uint32_t)by + 1u : 0u) {}
  __device__ __forceinline__ int of(int x) const { return d > 1 ? (int)__umulhi((uint32_t)x, m) : x; }
};

template <int P>
__global__ void __launch_bounds__(kBrThreads, 1) k_brick(const __grid_constant__ BrickArgs a) {
  constexpr int R = (P == 25) ? 4 : (P == 13) ? 2 : 1;
  constexpr int NP = npairs_of(P);
  extern __shared__ __align__(16) float fields[];
  __shared__ int s_fail;
  const Geom& g = a.g;
  const int tid = threadIdx.x;
  const int bi_id = blockIdx.x / a.nbj, bj_id = blockIdx.x - bi_id * a.nbj;
  const int i0 = bi_id * a.bi, j0 = bj_id * a.bj;
  const int ni = min(a.bi, g.xs - i0), nj = min(a.bj, g.ys - j0);
  const int pitch = a.pitch;                  // a row: 4 halo points, zq quads, 4 halo points
  const int plane = (a.bj + 2 * R) * pitch;   // of u and v, with R halo rows either side
  const int level = (a.bi + 2 * R) * plane;
  float* U = fields;
  float* V = U + level;
  float* Sx = V + level;                      // [bi][bj][zq quads]
  if (tid == 0) s_fail = 0;
  const int ub0 = a.ub_dev ? a.ub0 ^ __ldg(a.ub_dev) : a.ub0;

  // u and v with R planes and rows around, s; rows past the field's halo are not read
  const int wq = pitch / 4;
  for (int x = tid; x < (ni + 2 * R) * (nj + 2 * R) * wq; x += kBrThreads) {
    const int row = x / wq, q = x - row * wq;
    const int ii = row / (nj + 2 * R), jj = row - ii * (nj + 2 * R);
    const long long at = g.org + (long long)(i0 + ii - R) * g.si + (long long)(j0 + jj - R) * g.sj + 4 * q - 4;
    const int to = ii * plane + jj * pitch + 4 * q;
    *reinterpret_cast<float4*>(U + to) = __ldcg(reinterpret_cast<const float4*>(a.buf[ub0] + at));
    *reinterpret_cast<float4*>(V + to) = __ldcg(reinterpret_cast<const float4*>(a.buf[ub0 ^ 1] + at));
  }
  for (int x = tid; x < ni * nj * a.zq; x += kBrThreads) {
    const int row = x / a.zq, q = x - row * a.zq;
    const int ii = row / nj, jj = row - ii * nj;
    const long long at = g.org + (long long)(i0 + ii) * g.si + (long long)(j0 + jj) * g.sj + 4 * q;
    *reinterpret_cast<float4*>(Sx + ((ii * a.bj + jj) * a.zq + q) * 4) =
        __ldcg(reinterpret_cast<const float4*>(a.s + at));
  }
  const bool has_im = bi_id > 0, has_ip = bi_id + 1 < a.nbi, has_jm = bj_id > 0, has_jp = bj_id + 1 < a.nbj;
  // the neighbour this thread polls for, if any
  const int nb = tid == 0 && has_im ? (int)blockIdx.x - a.nbj
               : tid == 1 && has_ip ? (int)blockIdx.x + a.nbj
               : tid == 2 && has_jm ? (int)blockIdx.x - 1
               : tid == 3 && has_jp ? (int)blockIdx.x + 1 : -1;
  const int zq = a.zq;
  // halo rows: R planes below and above, then R rows before and behind
  const int hi_rows = R * nj, hj_rows = R * ni;
  const int halo_quads = 2 * (hi_rows + hj_rows) * zq;
  const Div by_zq(zq), by_nj(nj), by_ni(ni);
  __syncthreads();

  for (int t = 0; t < a.steps; ++t) {
    const float* ug = a.buf[ub0 ^ (t & 1)];
    float* vg = a.buf[ub0 ^ (t & 1) ^ 1];
    if (t > 0) {
      if (nb >= 0) {
        const int* word = a.words + (size_t)nb * kBrPad;
        if (b_ld_acquire(word) < t) {
          const uint64_t start = global_ns();
          for (uint32_t it = 1; b_ld_acquire(word) < t; ++it) {
            if ((it & 255u) == 0 &&
                (global_ns() - start > a.limit_ns || b_ld_acquire(a.abort_word) != 0)) {
              atomicCAS(a.status, 0u, (uint32_t)kDevTimeoutDep);
              atomicExch(a.abort_word, 1);
              s_fail = 1;
              break;
            }
          }
        }
      }
      __syncthreads();
      if (s_fail) return;
      for (int x = tid; x < halo_quads; x += kBrThreads) {
        int row = by_zq.of(x);
        const int q = x - row * zq;
        int ii, jj;
        bool have;
        if (row < 2 * hi_rows) {
          const bool up = row >= hi_rows;
          row -= up ? hi_rows : 0;
          const int m = by_nj.of(row);
          ii = up ? ni + m : m - R;
          jj = row - m * nj;
          have = up ? has_ip : has_im;
        } else {
          row -= 2 * hi_rows;
          const bool up = row >= hj_rows;
          row -= up ? hj_rows : 0;
          const int m = by_ni.of(row);
          jj = up ? nj + m : m - R;
          ii = row - m * ni;
          have = up ? has_jp : has_jm;
        }
        if (have) {
          const long long at = g.org + (long long)(i0 + ii) * g.si + (long long)(j0 + jj) * g.sj + 4 * q;
          *reinterpret_cast<float4*>(U + (ii + R) * plane + (jj + R) * pitch + 4 + 4 * q) =
              __ldcg(reinterpret_cast<const float4*>(ug + at));
        }
      }
      __syncthreads();
    }
    const bool all = t + 2 >= a.steps;
    const float amp = a.amps_dev ? __ldg(a.amps_dev + (size_t)t * a.amp_stride) : a.amps[t];
    for (int x = tid; x < ni * nj * zq; x += kBrThreads) {
      const int row = by_zq.of(x), qd = x - row * zq;
      const int ii = by_nj.of(row), jj = row - ii * nj;
      const float* uc = U + (ii + R) * plane + (jj + R) * pitch + 4 + 4 * qd;
      const float4 c4 = *reinterpret_cast<const float4*>(uc);
      const float4 l4 = *reinterpret_cast<const float4*>(uc - 4);
      const float4 r4 = *reinterpret_cast<const float4*>(uc + 4);
      const float w[12] = {l4.x, l4.y, l4.z, l4.w, c4.x, c4.y, c4.z, c4.w, r4.x, r4.y, r4.z, r4.w};
      const P4 cu = {make_float2(c4.x, c4.y), make_float2(c4.z, c4.w)};
      const P4 u2 = add4(cu, cu);
      const P4 nu2 = {make_float2(-u2.a.x, -u2.a.y), make_float2(-u2.b.x, -u2.b.y)};
      P4 acc;
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const int ax = pair_axis(P, p);
        const int rr = pair_r(P, p);
        P4 sum;
        if (ax == 2) {
          sum = {make_float2(w[4 - rr] + w[4 + rr], w[5 - rr] + w[5 + rr]),
                 make_float2(w[6 - rr] + w[6 + rr], w[7 - rr] + w[7 + rr])};
        } else {
          const int step = rr * (ax == 1 ? pitch : plane);
          const float4 A = *reinterpret_cast<const float4*>(uc - step);
          const float4 B = *reinterpret_cast<const float4*>(uc + step);
          sum = add4({make_float2(A.x, A.y), make_float2(A.z, A.w)},
                     {make_float2(B.x, B.y), make_float2(B.z, B.w)});
        }
        const P4 d = add4(sum, nu2);
        acc = p == 0 ? mul4(d, splat(a.cf.cf[0])) : fma4(splat(a.cf.cf[p]), d, acc);
      }
      float* vc = V + (ii + R) * plane + (jj + R) * pitch + 4 + 4 * qd;
      const float4 v4 = *reinterpret_cast<const float4*>(vc);
      const float4 s4 = *reinterpret_cast<const float4*>(Sx + ((ii * a.bj + jj) * zq + qd) * 4);
      P4 ss = {make_float2(s4.x, s4.y), make_float2(s4.z, s4.w)};
      const int i = i0 + ii, j = j0 + jj, k = 4 * qd;
      if (i == a.src_i && j == a.src_j && (unsigned)(a.src_k - k) < 4u) {
        const int c = a.src_k - k;
        if (c == 0) ss.a.x = ss.a.x + amp;
        if (c == 1) ss.a.y = ss.a.y + amp;
        if (c == 2) ss.b.x = ss.b.x + amp;
        if (c == 3) ss.b.y = ss.b.y + amp;
      }
      P4 y = add4(u2, {make_float2(-v4.x, -v4.y), make_float2(-v4.z, -v4.w)});
      y = fma4(splat(a.cf.c1), acc, y);
      y = fma4(splat(a.cf.c2), ss, y);
      const bool give = all || (ii < R && has_im) || (ii >= ni - R && has_ip) || (jj < R && has_jm) ||
                        (jj >= nj - R && has_jp);
      float* dst = vg + g.org + (long long)i * g.si + (long long)j * g.sj + k;
      if (k + 3 < g.zs) {
        const float4 o = make_float4(y.a.x, y.a.y, y.b.x, y.b.y);
        *reinterpret_cast<float4*>(vc) = o;
        if (give) *reinterpret_cast<float4*>(dst) = o;
      } else {
        // a row's last quad: the points past zs are halo
        const float o[4] = {y.a.x, y.a.y, y.b.x, y.b.y};
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (k + c < g.zs) {
            vc[c] = o[c];
            if (give) dst[c] = o[c];
          }
      }
    }
    __syncthreads();
    if (tid == 0) b_st_release(a.words + (size_t)blockIdx.x * kBrPad, t + 1);
    float* x = U;
    U = V;
    V = x;
  }
}

size_t brick_smem(const BrickPlan& p, int R) {
  return ((size_t)2 * (p.bi + 2 * R) * (p.bj + 2 * R) * p.pitch + (size_t)p.bi * p.bj * p.zq * 4) * 4;
}

template <int P>
cudaError_t launch_p(const BrickPlan& p, const BrickArgs& a, cudaStream_t stream) {
  const size_t smem = brick_smem(p, radius_of(P));
  cudaError_t e = cudaFuncSetAttribute(k_brick<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  void* args[] = {(void*)&a};
  return cudaLaunchCooperativeKernel((const void*)k_brick<P>, dim3(p.nbi * p.nbj), dim3(kBrThreads), args,
                                     smem, stream);
}

}  // namespace

size_t brick_words(int bricks) { return (size_t)(bricks + 1) * kBrPad; }

// Bricks for the grid: of the splits that fit the SMs and shared memory, the
// one with the fewest quads a step (own and halo) in the largest brick.
bool plan_brick(const Geom& g, int R, int sms, size_t max_smem, BrickPlan* best) {
  long long cost = -1;
  BrickPlan p;
  p.zq = (g.zs + 3) / 4;
  p.pitch = 4 * p.zq + 8;
  if (g.xs > 4096 || g.ys > 4096 || g.zs > 4096) return false;
  for (int nbi = 1; nbi <= sms && nbi <= g.xs; ++nbi) {
    p.bi = (g.xs + nbi - 1) / nbi;
    p.nbi = (g.xs + p.bi - 1) / p.bi;
    if (p.nbi > 1 && g.xs - (p.nbi - 1) * p.bi < R) continue;
    for (int nbj = 1; nbj * p.nbi <= sms && nbj <= g.ys; ++nbj) {
      p.bj = (g.ys + nbj - 1) / nbj;
      p.nbj = (g.ys + p.bj - 1) / p.bj;
      if (p.nbj > 1 && g.ys - (p.nbj - 1) * p.bj < R) continue;
      if (brick_smem(p, R) > max_smem) continue;
      const long long c = (long long)p.zq * (2LL * p.bi * p.bj + 2 * R * (p.bi + p.bj));
      if (cost < 0 || c < cost) {
        cost = c;
        *best = p;
      }
    }
  }
  return cost >= 0;
}

// A step costs its chain and the brick's points: 7 points 64^3 (2048 points a
// brick) 2.6 us, 110^3 (9900) 5.3; 25 points 64^3 3.7, 80^3 (3920) 5.1.
double brick_us(const BrickPlan& p, int R, int steps) {
  const double kpts = 0.004 * p.bi * p.bj * p.zq;
  return steps * (R == 1 ? 1.9 + 0.33 * kpts : R == 2 ? 2.1 + 0.4 * kpts : 2.5 + 0.65 * kpts) + 10.0;
}

cudaError_t launch_brick(const BrickPlan& p, int points, const Geom& g, const Coefs<float>& cf,
                         float* const* fld, int steps, const Source& src, const StepFeed& feed, int* words,
                         uint32_t* dev_status, cudaStream_t stream) {
  if (steps < 1 || steps > kWaveSteps) return cudaErrorInvalidValue;
  BrickArgs a;
  a.g = g;
  a.cf = cf;
  a.buf[0] = fld[0];
  a.buf[1] = fld[1];
  a.s = fld[2];
  a.ub0 = feed.ub;
  a.ub_dev = feed.ub_dev;
  a.amps_dev = feed.amps_dev;
  a.amp_stride = feed.amp_stride;
  a.steps = steps;
  a.bi = p.bi;
  a.bj = p.bj;
  a.nbi = p.nbi;
  a.nbj = p.nbj;
  a.zq = p.zq;
  a.pitch = p.pitch;
  a.src_i = src.i;
  a.src_j = src.j;
  a.src_k = src.k;
  a.abort_word = words;
  a.words = words + kBrPad;
  a.limit_ns = 4000000000ull;
  a.status = dev_status;
  for (int n = 0; n < kWaveSteps; ++n) a.amps[n] = n < steps && feed.amps ? feed.amps[n] : 0.0f;
  cudaError_t e = cudaMemsetAsync(words, 0, brick_words(p.nbi * p.nbj) * sizeof(int), stream);
  if (e != cudaSuccess) return e;
  switch (points) {
    case 7: return launch_p<7>(p, a, stream);
    case 13: return launch_p<13>(p, a, stream);
    case 25: return launch_p<25>(p, a, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace st3d
