// st3d_kernels_wave.cu -- many FP32 wave steps in one launch, their planes
// meeting in L2.
//
// One step a launch (st3d_kernels_tma.cu) moves 16 bytes a point and is bound
// by HBM.  Here the steps of a call run as a pipeline along i: the persistent
// CTAs form T levels of S columns; a column is one tile (16 rows x 128 points
// or 32 x 64) over all planes, and a CTA of level t takes its column's planes
// through step p*T + t, a dozen planes behind the CTAs that take the same and
// the neighbouring columns through the step before.  The planes one level
// writes are read by the next from L2, a few microseconds later, so HBM moves
// u, v and s in and two levels out about once for T steps and the other loads
// come at L2 rate.  The update is in place, as step after step: no second
// pair of fields, any halo, the same operations on every point (bit for bit
// the one-step kernel's result).
//
// Order.  Level t runs the columns q = 0, 1, ... of pass 0, 1, ... as one
// sequence, x = p*Q + q, `shift` columns late per level: CTA (t, s) takes
// x + t*shift = s, s + S, s + 2S, ...  A tile's rows lie `skew` rows lower at
// each level, so with skew = R a column needs nothing of the row of tiles after
// its own and a level may follow one column behind (shift = 1, the neighbour
// along k).  When all columns are at work at once there is no skew and no shift.
// Step n of a column at plane i reads U^n up to plane i + R of the tiles that
// hold its rows with R either side and of those beside it along k (the cross
// needs no corner), and overwrites U^{n-1}, which step n - 1 of the same tiles
// read; both are safe once those tiles have stored plane i + R of step n - 1.
// A step waits for the step before only, and each CTA takes its units pass by
// pass: by induction over (pass, level) every wait ends, the launch being
// cooperative (all CTAs resident).
//
// What bounds it is whether L2 (126 MB, 20 TB/s read) still holds a plane
// when the next level comes for it.  The columns of level 0 depend on nothing
// near and drift apart; the levels behind wait for the slowest neighbour, the
// lag grows, and past about 20 us of lag at 430 Gpts/s the planes are gone
// before they are read (7 points, 1024^2 planes: 11.5 bytes read from HBM a
// point and step).  So level 0 is held to `couple` planes of its neighbours:
// 7 points 512^3 437 -> 568 Gpts/s, 25 points 1024^2 planes 392 -> 463; the skew
// (before it a level followed a row of tiles behind, and a fifth of the columns
// found their planes gone at the next turn) 1024^3 at 7 / 25 points 528 -> 576 and
// 458 -> 469.  The
// columns' progress words lie 128 bytes apart: packed, all CTAs polled one L2
// slice and every tile load met that queue (7 points 256^3: 1150 us against
// 590; 25 points 528^3: 18.0 ms against 15.2).  The limit above that is
// shared-memory bandwidth at 25 points (135 KB a plane of 2048 points: 505
// Gpts/s without any waiting) and L2 at 7 points (860).
//
// Inside a CTA: 16 consumer warps and a producer as in the one-step kernel,
// and two more warps that keep the hand-over off their paths:
//   - the publisher reads the plane each consumer warp last stored (shared
//     memory, released per warp) and releases the least of them, gpu scope,
//     as the column's progress: one fence for as many planes as have been
//     finished since the last, not one a plane;
//   - the watcher polls the progress words, fences (acquire, gpu scope, and
//     generic to async proxy) when they have moved, and leaves the planes that
//     may be loaded in shared memory, where the producer finds them.
// Every wait ends: past `limit_ns` it sets the status word and an abort word
// that all other waits look at.
//
// The streamed drop-in call (pinned host arrays, STREAM = true) runs as the same
// pipeline with its transfers: `n_up` more CTAs copy u, v and s in, a row of
// tiles (slab) after the other over all planes, `n_down` copy the last two
// levels of a slab out once its columns have stored them.  A column's first step
// waits until its slab and the two beside it are in; everything later follows
// by the columns' own order.  With as many levels as steps the first slabs leave
// while the last are still coming.
#include <type_traits>

#include "st3d_internal.h"
#include "st3d_p4.cuh"
#include "st3d_tma.cuh"

namespace st3d {

namespace {

constexpr int kWWarps = 16;                      // consumer warps
constexpr int kWThreads = (kWWarps + 3) * 32;    // + producer, publisher, watcher
constexpr int kWNV = 4;                          // pipeline stages (6: no faster)
constexpr int kWPad = 32;                        // ints between two progress words (128 bytes)

// Tile shapes of the same 2048 points: a warp serves one row of 128 points or
// two of 64.
template <bool NARROW>
struct Tile {
  static constexpr int TJ = NARROW ? 32 : 16;
  static constexpr int TK = NARROW ? 64 : 128;
  static constexpr int UKW = TK + 2 * kTmaKHalo;
};

struct WaveArgs {
  Geom g;
  Coefs<float> cf;
  float* buf[2];
  int ub0;               // buffer of U^n at the launch's first step, or, with ub_dev,
  const int* ub_dev;     //   what *ub_dev is exclusive-ored with
  int steps;             // of this launch
  int T, S, Q, shift;    // levels, columns at work per level, columns, delay of a level
  int skew;              // rows a tile lies lower at each level
  int ntk;
  int couple;            // level 0: planes a column may be ahead of its neighbours
  int* prog;             // [step][Q], kWPad apart: planes stored
  int* abort_word;
  int src_i, src_j, src_k;
  uint64_t limit_ns;
  uint32_t* status;
  const float* amps_dev;  // step m's amplitude at [m * amp_stride] instead of amps[m]
  int amp_stride;
  float amps[kWaveSteps];
  WaveXfer x;
  int* up_cnt;           // per slab (kWPad apart): items copied in
  int* heads;            // upload and download queue
};

__device__ __forceinline__ void w_st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int w_lds_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void w_sts_release(int* p, int v) {
  asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ int w_ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void w_acquire_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void w_proxy_fence() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// The end of a wait's patience: past the limit, or another wait gave up.
struct Patience {
  uint64_t start, limit;
  const int* abort_word;
  __device__ __forceinline__ Patience(const WaveArgs& a) : start(global_ns()), limit(a.limit_ns), abort_word(a.abort_word) {}
  __device__ __forceinline__ bool over() const {
    return w_ld_relaxed(abort_word) != 0 || global_ns() - start > limit;
  }
};

__device__ __forceinline__ void give_up(const WaveArgs& a, uint32_t why) {
  atomicCAS(a.status, 0u, why);
  atomicExch(a.abort_word, 1);
}

__device__ __forceinline__ bool wait_bar(const WaveArgs& a, uint64_t* bar, uint32_t parity, uint32_t why) {
  if (mbar_try_wait(bar, parity)) return true;
  const Patience pat(a);
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 63u) == 0 && pat.over()) {
      give_up(a, why);
      return false;
    }
  }
}

// The CTA's units in order: unit(r) is its r-th turn.  False past the end.
struct Turn {
  int q, step, pass;
  int jt, kt, j0;  // tile and its first row (may lie outside the grid)
  bool live;  // a column to work on (a level waits `shift` columns at first, skips steps past
              // the last and tiles without a row of the grid)
};
template <int TJ>
__device__ __forceinline__ bool turn(const WaveArgs& a, int t, int s, int r, Turn* u) {
  const int x = r * a.S + s - t * a.shift;
  u->live = false;
  if (x < 0) return true;
  u->pass = x / a.Q;
  u->q = x - u->pass * a.Q;
  if ((long long)u->pass * a.T >= a.steps) return false;
  u->step = u->pass * a.T + t;
  u->jt = u->q / a.ntk;
  u->kt = u->q - u->jt * a.ntk;
  u->j0 = u->jt * TJ - a.skew * t;
  u->live = u->step < a.steps && u->j0 < a.g.ys && u->j0 + TJ > 0;
  return true;
}

__device__ __forceinline__ void w_red_release(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Rows [ja, jb) of plane i between the host span and the field: one contiguous
// run on the host side, whole words of W points, warps on 128-byte lines.
template <int W, bool UP>
__device__ __forceinline__ void copy_rows(const WaveArgs& a, float* dev, float* host, int i, int ja, int jb) {
  using V = typename std::conditional<W == 4, float4, float>::type;
  const WaveXfer& x = a.x;
  const int kv = (x.R.zs + 2 * x.hz) / W;
  const int n = (jb - ja) * kv;
  V* span = reinterpret_cast<V*>(host + x.R.ijk_ofs + (long long)i * x.R.imult + (long long)ja * x.R.jmult - x.hz);
  V* rows = reinterpret_cast<V*>(dev + a.g.org + (long long)i * a.g.si + (long long)ja * a.g.sj - x.hz);
  const int pitch = (int)(a.g.sj / W);
  const int shift = (int)((reinterpret_cast<uintptr_t>(span) / sizeof(V)) % (128 / sizeof(V)));
  constexpr int UN = W == 4 ? 4 : 8;
  for (int y0 = (int)threadIdx.x - shift; y0 < n; y0 += UN * kWThreads) {
    V v[UN];
#pragma unroll
    for (int m = 0; m < UN; ++m) {
      const int y = y0 + m * kWThreads;
      if (y >= 0 && y < n) {
        const int r = y / kv;
        v[m] = UP ? span[y] : __ldcg(rows + (long long)r * pitch + (y - r * kv));
      }
    }
#pragma unroll
    for (int m = 0; m < UN; ++m) {
      const int y = y0 + m * kWThreads;
      if (y >= 0 && y < n) {
        const int r = y / kv;
        if (UP)
          rows[(long long)r * pitch + (y - r * kv)] = v[m];
        else
          span[y] = v[m];
      }
    }
  }
}

// One transfer CTA: items (slab, block of planes, field) from its queue.
template <int TJ>
__device__ void transfer(const WaveArgs& a, int ub0, int* s_item) {
  const WaveXfer& x = a.x;
  const bool up = (int)blockIdx.x < a.T * a.S + x.n_up;
  // (downloads by the tiles of the two last levels, which the skew may move)
  const int slabs = up ? (a.g.ys + TJ - 1) / TJ : a.Q / a.ntk, fields = up ? 3 : 2;
  const int blocks = (a.g.xs + x.planes - 1) / x.planes, per = blocks * fields;
  while (true) {
    if (threadIdx.x == 0) {
      int it = atomicAdd(a.heads + (up ? 0 : 1), 1);
      if (it >= slabs * per) it = -1;
      if (it >= 0 && !up) {
        // v is the level before the last, u the last
        const int slab = it / per, f = it % fields;
        const int* word = a.prog + ((size_t)(a.steps - 2 + f) * a.Q + slab * a.ntk) * kWPad;
        const int j0 = slab * TJ - a.skew * ((a.steps - 2 + f) % a.T);
        const int cols = j0 < a.g.ys && j0 + TJ > 0 ? a.ntk : 0;
        const Patience pat(a);
        for (int q = 0; q < cols && it >= 0; ++q)
          for (uint32_t n = 1; w_ld_relaxed(word + (size_t)q * kWPad) < a.g.xs; ++n) {
            __nanosleep(200);
            if ((n & 255u) == 0 && pat.over()) {
              give_up(a, kDevTimeoutDep);
              it = -1;
              break;
            }
          }
        w_acquire_fence();
      }
      *s_item = it;
    }
    __syncthreads();
    const int it = *s_item;
    if (it < 0) return;
    const int slab = it / per, rest = it - slab * per;
    const int f = rest % fields, pb = rest / fields;
    int ia = pb * x.planes, ib = min(ia + x.planes, a.g.xs);
    int ja = slab * TJ, jb = min(ja + TJ, a.g.ys);
    if (!up) {
      const int j0 = ja - a.skew * ((a.steps - 2 + f) % a.T);
      ja = max(j0, 0);
      jb = min(j0 + TJ, a.g.ys);
      if (jb <= ja) {
        __syncthreads();
        continue;
      }
    }
    if (up) {
      // the halo planes and rows come with the outermost items
      if (pb == 0) ia -= x.hx;
      if (ib == a.g.xs) ib += x.hx;
      if (slab == 0) ja -= x.hy;
      if (slab == slabs - 1) jb += x.hy;
    }
    // uploads: u, v, s; downloads: v (f = 0), u (f = 1) of the end
    const int ue = ub0 ^ (a.steps & 1);
    float* dev = up ? (f == 2 ? x.s : a.buf[f == 0 ? ub0 : ub0 ^ 1]) : a.buf[f == 1 ? ue : ue ^ 1];
    float* host = up ? const_cast<float*>(x.hin[f]) : x.hout[f];
    for (int i = ia; i < ib; ++i) {
      if (up) {
        if (x.vec) copy_rows<4, true>(a, dev, host, i, ja, jb);
        else copy_rows<1, true>(a, dev, host, i, ja, jb);
      } else {
        if (x.vec) copy_rows<4, false>(a, dev, host, i, ja, jb);
        else copy_rows<1, false>(a, dev, host, i, ja, jb);
      }
    }
    __syncthreads();
    if (up && threadIdx.x == 0) {
      w_proxy_fence();
      w_red_release(a.up_cnt + (size_t)slab * kWPad, 1);
    }
  }
}

template <int P, bool NARROW, bool STREAM>
__global__ void __launch_bounds__(kWThreads, 1)
    k_wave(const __grid_constant__ CUtensorMap um0, const __grid_constant__ CUtensorMap um1,
           const __grid_constant__ CUtensorMap vm0, const __grid_constant__ CUtensorMap vm1,
           const __grid_constant__ CUtensorMap smap, const __grid_constant__ WaveArgs a) {
  constexpr int R = (P == 25) ? 4 : (P == 13) ? 2 : 1;
  constexpr int QN = 2 * R + 1;
  constexpr int NV = kWNV;
  constexpr int NW = kWWarps;
  constexpr int TJ = Tile<NARROW>::TJ;
  constexpr int TK = Tile<NARROW>::TK;
  constexpr int UKW = Tile<NARROW>::UKW;
  constexpr int NU = NV + R;
  constexpr int NP = npairs_of(P);
  constexpr int USLOT = (UKW * (TJ + 2 * R) + 31) / 32 * 32;
  constexpr int VSLOT = TK * TJ;
  constexpr uint32_t UBYTES = UKW * (TJ + 2 * R) * 4;
  constexpr uint32_t VBYTES = VSLOT * 4;

  extern __shared__ __align__(128) unsigned char smem_raw[];
  float* ur = reinterpret_cast<float*>(smem_raw);
  float* vr = ur + NU * USLOT;
  float* sr = vr + NV * VSLOT;
  uint64_t* full = reinterpret_cast<uint64_t*>(sr + NV * VSLOT);
  uint64_t* empty = full + NV;
  int* stored = reinterpret_cast<int*>(empty + NV);  // planes stored per consumer warp, all units together
  int* avail = stored + NW;                          // planes the unit's inputs are ready for, likewise

  const Geom& g = a.g;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x / a.S, s = blockIdx.x - t * a.S;
  const int ub0 = a.ub_dev ? a.ub0 ^ __ldg(a.ub_dev) : a.ub0;
  if (STREAM && (int)blockIdx.x >= a.T * a.S) {
    transfer<TJ>(a, ub0, stored);
    return;
  }
  if (threadIdx.x < NW + 1) stored[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int st = 0; st < NV; ++st) {
      mbar_init(&full[st], 1);
      mbar_init(&empty[st], NW);
    }
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  __syncthreads();

  if (warp == NW) {
    // ---------------- producer ----------------
    if (lane != 0) return;
    tma_prefetch_desc(&um0);
    tma_prefetch_desc(&um1);
    tma_prefetch_desc(&vm0);
    tma_prefetch_desc(&vm1);
    tma_prefetch_desc(&smap);
    uint32_t h = 0;
    int done = 0;  // planes of the units before
    int seen = 0;
    bool ok = true;
    Turn u;
    for (int r = 0; ok && turn<TJ>(a, t, s, r, &u); ++r) {
      if (!u.live) continue;
      const int k0 = u.kt * TK, j0 = u.j0;
      const int ub = ub0 ^ (u.step & 1);
      const CUtensorMap* um = ub ? &um1 : &um0;
      const CUtensorMap* vm = ub ? &vm0 : &vm1;
      const int nsteps = g.xs + 2 * R;
      for (int n = 0; n < nsteps; ++n, ++h) {
        const int stage = (int)(h % NV);
        if (h >= (uint32_t)NV && !wait_bar(a, &empty[stage], ((h / NV) - 1) & 1u, kDevTimeoutEmpty)) {
          ok = false;
          break;
        }
        const int p = n - R;  // u plane of this stage
        // (a streamed call's halo planes come with the column's slabs)
        const int need = done + min(max(p + 1, STREAM ? 1 : 0), g.xs);
        if (seen < need) {
          seen = w_lds_acquire(avail);
          if (seen < need) {
            const Patience pat(a);
            for (uint32_t it = 1; (seen = w_lds_acquire(avail)) < need; ++it) {
              if ((it & 255u) == 0 && pat.over()) {
                give_up(a, kDevTimeoutDep);
                ok = false;
                break;
              }
            }
            if (!ok) break;
          }
          w_proxy_fence();  // the async proxy's loads come after it
        }
        const bool has_vs = n >= 2 * R;
        mbar_arrive_expect_tx(&full[stage], UBYTES + (has_vs ? 2 * VBYTES : 0u));
        tma_load_3d(ur + (h % NU) * USLOT, um, &full[stage], g.pk + k0 - kTmaKHalo, g.pj + j0 - R, g.pi + p);
        if (has_vs) {
          const int i = n - 2 * R;
          tma_load_3d(vr + stage * VSLOT, vm, &full[stage], g.pk + k0, g.pj + j0, g.pi + i);
          tma_load_3d(sr + stage * VSLOT, &smap, &full[stage], g.pk + k0, g.pj + j0, g.pi + i);
        }
      }
      done += g.xs;
    }
    // Leave no copy in flight: wait for the stages issued last.
    for (uint32_t m = (h > (uint32_t)NV ? h - NV : 0u); m < h; ++m)
      (void)mbar_wait_bounded(&full[m % NV], (m / NV) & 1u, 4000000000ull);
    return;
  }

  if (warp == NW + 1) {
    // ---------------- publisher ----------------
    int done = 0;
    Turn u;
    for (int r = 0; turn<TJ>(a, t, s, r, &u); ++r) {
      if (!u.live) continue;
      int* word = a.prog + ((size_t)u.step * a.Q + u.q) * kWPad;
      int out = 0;  // planes published
      const Patience pat(a);
      for (uint32_t it = 1; out < g.xs; ++it) {
        const int mine = lane < NW ? w_lds_acquire(stored + lane) : 0x7fffffff;
        const int planes = min(__reduce_min_sync(0xffffffffu, mine) - done, g.xs);
        if (planes > out) {
          __syncwarp();  // every lane's acquire before lane 0's release
          if (lane == 0) {
            w_proxy_fence();
            w_st_release(word, planes);
          }
          __syncwarp();
          out = planes;
        } else {
          __nanosleep(20);
          if ((it & 1023u) == 0) {
            const bool over = __any_sync(0xffffffffu, pat.over());
            if (over) return;  // the waits that matter report
          }
        }
      }
      done += g.xs;
    }
    return;
  }

  if (warp == NW + 2) {
    // ---------------- watcher ----------------
    // lanes 0..8: the step before, of the tiles (up to three) that hold the
    // column's rows with R either side, and of those beside it along k that
    // hold its rows; lanes 16..19: level 0, the neighbours at work in the same
    // turn, which this column may be `couple` planes ahead of
    const bool before = lane < 9;
    const int l = before ? lane % 3 : (lane & 3) + 1;
    const int lt = t > 0 ? t - 1 : a.T - 1;      // level of the step before
    const int off = a.skew * lt;                 // row j lies in its tile (j + off) / TJ
    int done = 0;
    Turn u;
    for (int r = 0; turn<TJ>(a, t, s, r, &u); ++r) {
      if (!u.live) continue;
      const int jt = u.jt;
      int col = u.q;
      bool look = false;
      if (before) {
        const int kt = u.kt + (l == 1 ? -1 : l == 2 ? 1 : 0), reach = l == 0 ? R : 0;
        const int first = max(u.j0 - reach, 0), last = min(u.j0 + TJ + reach, g.ys) - 1;
        const int tile = (first + off) / TJ + lane / 3;
        look = u.step > 0 && kt >= 0 && kt < a.ntk && tile <= (last + off) / TJ;
        if (look) col = tile * a.ntk + kt;
      } else if (lane >= 16 && lane < 20 && t == 0) {
        const int dq = l == 1 ? -1 : l == 2 ? 1 : l == 3 ? -a.ntk : a.ntk;
        look = s + dq >= 0 && s + dq < a.S &&
               (l == 1 ? u.kt > 0 : l == 2 ? u.kt < a.ntk - 1 : l == 3 ? jt > 0 : (jt + 1) * TJ < g.ys);
        if (look) col = u.q + dq;
      }
      const int ahead = before ? 0 : a.couple;
      const int* word = a.prog + ((size_t)(before && look ? u.step - 1 : u.step) * a.Q + col) * kWPad;
      int ready = 0;
      const Patience pat(a);
      if (STREAM && u.step == 0) {
        // the column's slab and the two beside it are in
        const int slab = jt + lane - 1;
        const bool wait = lane < 3 && slab >= 0 && slab * TJ < g.ys;
        const int* cnt = a.up_cnt + (size_t)(wait ? slab : jt) * kWPad;
        const int need = 3 * ((g.xs + a.x.planes - 1) / a.x.planes);
        for (uint32_t it = 1; !__all_sync(0xffffffffu, !wait || w_ld_relaxed(cnt) >= need); ++it) {
          __nanosleep(200);
          if ((it & 255u) == 0 && __any_sync(0xffffffffu, pat.over())) return;
        }
        w_acquire_fence();
        w_proxy_fence();
        __syncwarp();
      }
      for (uint32_t it = 1; ready < g.xs; ++it) {
        const int mine = look ? w_ld_relaxed(word) + ahead : g.xs;
        const int planes = min(__reduce_min_sync(0xffffffffu, mine), g.xs);
        if (planes > ready) {
          ready = planes;
          w_acquire_fence();
          w_proxy_fence();
          __syncwarp();
          if (lane == 0) w_sts_release(avail, done + ready);
        } else {
          __nanosleep(20);
          if ((it & 255u) == 0) {
            const bool over = __any_sync(0xffffffffu, pat.over());
            if (over) return;  // the producer's wait reports
          }
        }
      }
      done += g.xs;
    }
    return;
  }

  // ---------------- consumers ----------------
  const int row = NARROW ? 2 * warp + (lane >> 4) : warp;
  const int kl = NARROW ? (lane & 15) : lane;
  uint32_t h = 0;
  int done = 0;
  float4 q[QN];
  Turn u;
  for (int r = 0; turn<TJ>(a, t, s, r, &u); ++r) {
    if (!u.live) continue;
    const int j = u.j0 + row;
    const int k = u.kt * TK + 4 * kl;
    const int nsteps = g.xs + 2 * R;
    const bool row_ok = (unsigned)j < (unsigned)g.ys;
    const int ub = ub0 ^ (u.step & 1);
    float* vrow = a.buf[ub ^ 1] + g.org + (long long)j * g.sj + k;
    const float amp = a.amps_dev ? __ldg(a.amps_dev + (size_t)u.step * a.amp_stride) : a.amps[u.step];
    const int src_i = (j == a.src_j && (unsigned)(a.src_k - k) < 4u) ? a.src_i : -1;
    for (int n0 = 0; n0 < nsteps; n0 += QN) {
#pragma unroll
      for (int ph = 0; ph < QN; ++ph) {
        const int n = n0 + ph;
        if (n >= nsteps) break;
        const uint32_t hh = h + (uint32_t)n;
        const int stage = (int)(hh % NV);
        if (!wait_bar(a, &full[stage], (hh / NV) & 1u, kDevTimeoutFull)) return;
        q[ph] = *reinterpret_cast<const float4*>(ur + (hh % NU) * USLOT + (row + R) * UKW + kTmaKHalo + 4 * kl);
        if (n >= 2 * R) {
          const int i = n - 2 * R;
          const float* uc = ur + ((hh - R) % NU) * USLOT + (row + R) * UKW;
          const float4 c4 = q[(ph + QN - R) % QN];
          const float4 l4 = *reinterpret_cast<const float4*>(uc + 4 * kl);
          const float4 r4 = *reinterpret_cast<const float4*>(uc + 2 * kTmaKHalo + 4 * kl);
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
            if (ax == 2 && (rr & 1)) {
              sum = {make_float2(w[4 - rr] + w[4 + rr], w[5 - rr] + w[5 + rr]),
                     make_float2(w[6 - rr] + w[6 + rr], w[7 - rr] + w[7 + rr])};
            } else if (ax == 2) {
              sum = add4({make_float2(w[4 - rr], w[5 - rr]), make_float2(w[6 - rr], w[7 - rr])},
                         {make_float2(w[4 + rr], w[5 + rr]), make_float2(w[6 + rr], w[7 + rr])});
            } else if (ax == 1) {
              const float4 A = *reinterpret_cast<const float4*>(uc - rr * UKW + kTmaKHalo + 4 * kl);
              const float4 B = *reinterpret_cast<const float4*>(uc + rr * UKW + kTmaKHalo + 4 * kl);
              sum = add4({make_float2(A.x, A.y), make_float2(A.z, A.w)},
                         {make_float2(B.x, B.y), make_float2(B.z, B.w)});
            } else {
              const float4 A = q[(ph + 2 * QN - R - rr) % QN];
              const float4 B = q[(ph + QN - R + rr) % QN];
              sum = add4({make_float2(A.x, A.y), make_float2(A.z, A.w)},
                         {make_float2(B.x, B.y), make_float2(B.z, B.w)});
            }
            const P4 d = add4(sum, nu2);
            acc = p == 0 ? mul4(d, splat(a.cf.cf[0])) : fma4(splat(a.cf.cf[p]), d, acc);
          }
          const float4 v4 = *reinterpret_cast<const float4*>(vr + stage * VSLOT + row * TK + 4 * kl);
          const float4 s4 = *reinterpret_cast<const float4*>(sr + stage * VSLOT + row * TK + 4 * kl);
          P4 ss = {make_float2(s4.x, s4.y), make_float2(s4.z, s4.w)};
          if (i == src_i) {
            const int c = a.src_k - k;
            if (c == 0) ss.a.x = ss.a.x + amp;
            if (c == 1) ss.a.y = ss.a.y + amp;
            if (c == 2) ss.b.x = ss.b.x + amp;
            if (c == 3) ss.b.y = ss.b.y + amp;
          }
          P4 x = add4(u2, {make_float2(-v4.x, -v4.y), make_float2(-v4.z, -v4.w)});
          x = fma4(splat(a.cf.c1), acc, x);
          x = fma4(splat(a.cf.c2), ss, x);
          if (row_ok) {
            float* dst = vrow + (long long)i * g.si;
            if (k + 3 < g.zs) {
              *reinterpret_cast<float4*>(dst) = make_float4(x.a.x, x.a.y, x.b.x, x.b.y);
            } else {
              const float o[4] = {x.a.x, x.a.y, x.b.x, x.b.y};
#pragma unroll
              for (int c = 0; c < 4; ++c)
                if (k + c < g.zs) dst[c] = o[c];
            }
          }
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&empty[stage]);
          if (n >= 2 * R) w_sts_release(stored + warp, done + n - 2 * R + 1);
        }
      }
    }
    h += (uint32_t)nsteps;
    done += g.xs;
  }
}

template <int P, bool NARROW>
size_t wave_smem() {
  constexpr int R = (P == 25) ? 4 : (P == 13) ? 2 : 1;
  const size_t uslot = ((size_t)Tile<NARROW>::UKW * (Tile<NARROW>::TJ + 2 * R) + 31) / 32 * 32 * 4;
  const size_t vslot = (size_t)Tile<NARROW>::TK * Tile<NARROW>::TJ * 4;
  return (size_t)(kWNV + R) * uslot + 2 * (size_t)kWNV * vslot + 2 * (size_t)kWNV * 8 + (kWWarps + 1) * 4 + 128;
}

template <int P, bool NARROW>
int occupancy_of() {
  auto kern = k_wave<P, NARROW, false>;
  const size_t smem = wave_smem<P, NARROW>();
  int n = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, kWThreads, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

template <int P, bool NARROW, bool STREAM>
cudaError_t launch_as(const WavePlan& w, const WaveArgs& a, cudaStream_t stream) {
  auto kern = k_wave<P, NARROW, STREAM>;
  const size_t smem = wave_smem<P, NARROW>();
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const WaveShape& sh = w.shape[NARROW ? 1 : 0];
  void* args[] = {(void*)&sh.umap[0], (void*)&sh.umap[1], (void*)&sh.vmap[0],
                  (void*)&sh.vmap[1], (void*)&sh.vmap[2], (void*)&a};
  const int ctas = a.T * a.S + (STREAM ? a.x.n_up + a.x.n_down : 0);
  return cudaLaunchCooperativeKernel((const void*)kern, dim3(ctas), dim3(kWThreads), args, smem, stream);
}

template <int P, bool NARROW>
cudaError_t launch_p(const WavePlan& w, const WaveArgs& a, cudaStream_t stream) {
  return a.x.n_up > 0 ? launch_as<P, NARROW, true>(w, a, stream) : launch_as<P, NARROW, false>(w, a, stream);
}

}  // namespace

int wave_tile_rows(bool narrow) { return narrow ? Tile<true>::TJ : Tile<false>::TJ; }
int wave_tile_cols(bool narrow) { return narrow ? Tile<true>::TK : Tile<false>::TK; }

int wave_blocks_per_sm(int points, bool narrow) {
  switch (points) {
    case 7: return narrow ? occupancy_of<7, true>() : occupancy_of<7, false>();
    case 13: return narrow ? occupancy_of<13, true>() : occupancy_of<13, false>();
    case 25: return narrow ? occupancy_of<25, true>() : occupancy_of<25, false>();
    default: return 0;
  }
}

// abort word, progress, and for a streamed call its slabs' counters and queues
size_t wave_words(int steps, int columns) { return ((size_t)steps * columns + columns + 3) * kWPad; }

cudaError_t launch_wave(const WavePlan& w, int points, const Geom& g, const Coefs<float>& cf,
                        float* const* fld, int steps, const Source& src, const StepFeed& feed,
                        uint32_t* dev_status, cudaStream_t stream, const WaveXfer* xfer) {
  if (steps < 1 || steps > w.max_steps || w.T < 1 || w.S < 1) return cudaErrorInvalidValue;
  WaveArgs a;
  a.g = g;
  a.cf = cf;
  a.buf[0] = fld[0];
  a.buf[1] = fld[1];
  a.ub0 = feed.ub;
  a.ub_dev = feed.ub_dev;
  a.amps_dev = feed.amps_dev;
  a.amp_stride = feed.amp_stride;
  for (int n = 0; n < kWaveSteps; ++n) a.amps[n] = n < steps && feed.amps ? feed.amps[n] : 0.0f;
  a.steps = steps;
  a.T = w.T;
  a.S = w.S;
  a.Q = w.Q;
  a.shift = w.shift;
  a.skew = w.skew;
  a.ntk = w.shape[w.narrow].ntk;
  a.couple = w.couple;
  a.abort_word = w.words;
  a.prog = w.words + kWPad;
  a.src_i = src.i;
  a.src_j = src.j;
  a.src_k = src.k;
  a.limit_ns = w.limit_ns;
  a.status = dev_status;
  a.x = xfer ? *xfer : WaveXfer();
  a.up_cnt = a.prog + (size_t)steps * a.Q * kWPad;
  a.heads = a.up_cnt + (size_t)a.Q * kWPad;
  cudaError_t e = cudaMemsetAsync(w.words, 0, wave_words(steps, a.Q) * sizeof(int), stream);
  if (e != cudaSuccess) return e;
  switch (points) {
    case 7: return w.narrow ? launch_p<7, true>(w, a, stream) : launch_p<7, false>(w, a, stream);
    case 13: return w.narrow ? launch_p<13, true>(w, a, stream) : launch_p<13, false>(w, a, stream);
    case 25: return w.narrow ? launch_p<25, true>(w, a, stream) : launch_p<25, false>(w, a, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace st3d
