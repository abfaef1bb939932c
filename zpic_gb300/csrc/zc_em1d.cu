// zc_em1d.cu -- the em1d step on the GPU (libzpic_cuda, C-ABI zc1_*).
//
// Restates the reference's em1d time step (em1d/simulation.c:45-56):
// current_zero; per species the push -- gather (interpolate_fld,
// em1d/particles.c:864-894), relativistic Boris, move, 1-D zigzag deposit
// (dep_current_zamb, particles.c:707-790), window shift + cold injection and
// absorbing / periodic boundaries (particles.c:1040-1062, 594-612), cell
// sort every n_sort steps; then current_update (guard fold + binomial /
// compensated passes, em1d/current.c:111-330) and emf_advance (yee_b, yee_e,
// Mur, yee_b, guard cells, window shift, em1d/emf.c:379-580).
//
// Layout: particles are SoA arrays (ix, x, ux, uy, uz) in two buffers per
// species, kept in cell order by a counting sort every few steps so that the
// lanes of a warp share cells; E, B, J are the reference's float3 buffers
// (one lower and two upper guard cells).
//
// A run of steps up to the next cell sort is one cooperative launch (k1_run)
// where the particles fit the multiprocessors' shared memory; else, and when
// kernels are timed one by one, a step is two kernels.  The push runs one particle per lane: the current
// of a motion that stays in its cell is summed over the lanes of the cell
// (segmented warp reduction) and added to J with one float reduction per
// node (performed in L2); cell-crossing motions add their two segments
// directly.  With open boundaries or a moving window the survivors are
// appended to the other buffer (one atomic per warp), and the last CTA to
// finish injects the column the window uncovered and updates the species'
// device-resident state (buffer, counts, iteration, window moves, kinetic
// energy).  The fields kernel (one CTA; grids up to a few thousand cells
// in shared memory) folds and filters the current, advances E and B, moves
// the window and clears the deposit buffer for the next step.  Every
// decision of the step is taken on the device, so a block of n_sort steps
// ending with the cell sort is one CUDA graph, captured once and replayed.
//
// Compiled with --fmad=false: every float operation rounds as in the
// reference C, so particles advanced from the same fields land on the same
// bits.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <new>
#include <vector>

#include "../../include/zpic_cuda.h"
#include "zc_internal.cuh"
#include "zc_kernels.h"

namespace zc1 {

constexpr int GC0 = 1, GC1 = 2;  // guard cells (em1d/emf.c:59)
// copies of the deposit buffer: the push's CTAs spread their float
// reductions over them (a 1-D grid is a few KB, held by few L2 slices), and
// the fields kernel sums them in a fixed order
constexpr int kJCopies = 8;
constexpr int kFieldUnroll = 2;  // grid elements per thread per load round of the fields kernel
enum { ERR1_ESCAPE = 1, ERR1_OVERFLOW = 2, ERR1_TIMEOUT = 4 };

struct Parts {
  int *ix;
  float *x, *ux, *uy, *uz;
};

// a species' state on the device, read and written only by the step's
// kernels (the host mirrors the counters, which it can predict)
struct SpecState1 {
  int np[2];        // particles in each buffer
  int cur;          // the buffer that holds the particles
  int iter;         // completed advances (spec->iter)
  int n_move;       // window moves (spec->n_move)
  unsigned done;    // CTAs finished in the running launch (0 between launches)
  double ekin_acc;  // kinetic-energy sum of the running advance
  double ekin;      // the sum of the last completed advance
  long long pushed;  // particles pushed so far (particle-steps)
};

struct Push1 {
  float tem, dt_dx, qnx, q;
  float dt, dx;  // window-move test (spec_move_window, particles.c:594-612)
  int nx;
  int mw;    // moving window
  int open;  // particles leaving [0, nx) are removed (open boundaries or window)
  int cap;   // capacity of each particle buffer
  int jstride;  // floats per deposit-buffer copy
};

// cold injection into column nx-1 after a window move (spec_set_x for
// uniform / step / slab profiles, particles.c:250-300; the momenta are ufl,
// the thermal part being zero)
struct Inject1 {
  int ppc, type;  // density type: 0 uniform, 1 empty, 2 step, 3 slab
  float start, end, dx;
  float ufl[3];
};

__device__ __forceinline__ float lerp1(const float *F, int i, int c, float w) {
  return F[(i + GC0) * 3 + c] * (1.0f - w) + F[(i + 1 + GC0) * 3 + c] * w;
}

// fire-and-forget float add performed in L2 (no value returned)
__device__ __forceinline__ void red(float *J, int i, int c, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(J + (i + GC0) * 3 + c), "f"(v) : "memory");
}

// the five contributions of one segment inside cell ix (particles.c:770-788):
// Jx at ix, Jy and Jz at ix and ix+1
struct Seg1 {
  float jx, y0, y1, z0, z1;
};

__device__ __forceinline__ Seg1 seg_current(float x0, float x1, float dx, float qvy, float qvz, float qnx) {
  const float s00 = 1.0f - x0, s01 = x0;
  const float s10 = 1.0f - x1, s11 = x1;
  Seg1 r;
  r.jx = qnx * dx;
  r.y0 = qvy * (s00 + s10 + (s00 - s10) / 2.0f);
  r.y1 = qvy * (s01 + s11 + (s01 - s11) / 2.0f);
  r.z0 = qvz * (s00 + s10 + (s00 - s10) / 2.0f);
  r.z1 = qvz * (s01 + s11 + (s01 - s11) / 2.0f);
  return r;
}

// adds a segment's contributions (an exact zero adds nothing and is skipped)
__device__ __forceinline__ void add_seg(float *J, int ix, const Seg1 &s) {
  if (s.jx != 0.f) red(J, ix, 0, s.jx);
  if (s.y0 != 0.f) red(J, ix, 1, s.y0);
  if (s.y1 != 0.f) red(J, ix + 1, 1, s.y1);
  if (s.z0 != 0.f) red(J, ix, 2, s.z0);
  if (s.z1 != 0.f) red(J, ix + 1, 2, s.z1);
}

// sums v over the lanes of each run of equal keys (lanes lane..run_last),
// leaving each run's sum in its first lane; maxlen: the longest run
__device__ __forceinline__ void run_sum(Seg1 &v, int run_last, unsigned maxlen) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    if ((unsigned)off >= maxlen) break;
    const bool take = lane + off <= run_last;
    const float o0 = __shfl_down_sync(0xffffffffu, v.jx, off);
    const float o1 = __shfl_down_sync(0xffffffffu, v.y0, off);
    const float o2 = __shfl_down_sync(0xffffffffu, v.y1, off);
    const float o3 = __shfl_down_sync(0xffffffffu, v.z0, off);
    const float o4 = __shfl_down_sync(0xffffffffu, v.z1, off);
    if (take) {
      v.jx += o0;
      v.y0 += o1;
      v.y1 += o2;
      v.z0 += o3;
      v.z1 += o4;
    }
  }
}


// one particle's gather, push and move (momenta in place)
struct Move1 {
  float kin, dx, x1, qvy, qvz;
  int di;
};
__device__ __forceinline__ Move1 push_lane(const float *E, const float *B, int ix, float x, float &ux, float &uy,
                                           float &uz, const Push1 &C) {
  Move1 m;
  // staggered linear gather (particles.c:864-894)
  const int ih = ix + ((x < 0.5f) ? -1 : 0);
  const float w1h = x + ((x < 0.5f) ? 0.5f : -0.5f);
  float ex = lerp1(E, ih, 0, w1h), ey = lerp1(E, ix, 1, x), ez = lerp1(E, ix, 2, x);
  float bx = lerp1(B, ix, 0, x), by = lerp1(B, ih, 1, w1h), bz = lerp1(B, ih, 2, w1h);
  // Boris (particles.c:960-1010)
  ex *= C.tem;
  ey *= C.tem;
  ez *= C.tem;
  float utx = ux + ex, uty = uy + ey, utz = uz + ez;
  const float u2 = utx * utx + uty * uty + utz * utz;
  const float gamma = sqrtf(1 + u2);
  m.kin = u2 / (1 + gamma);
  const float gtem = C.tem / gamma;
  bx *= gtem;
  by *= gtem;
  bz *= gtem;
  const float otsq = 2.0f / (1.0f + bx * bx + by * by + bz * bz);
  ux = utx + uty * bz - utz * by;
  uy = uty + utz * bx - utx * bz;
  uz = utz + utx * by - uty * bx;
  bx *= otsq;
  by *= otsq;
  bz *= otsq;
  utx += uy * bz - uz * by;
  uty += uz * bx - ux * bz;
  utz += ux * by - uy * bx;
  ux = utx + ex;
  uy = uty + ey;
  uz = utz + ez;
  // move (particles.c:1012-1022)
  const float rg = 1.0f / sqrtf(1.0f + ux * ux + uy * uy + uz * uz);
  m.dx = C.dt_dx * rg * ux;
  m.x1 = x + m.dx;
  m.di = (m.x1 >= 1.0f) - (m.x1 < 0.0f);
  m.x1 -= m.di;
  m.qvy = C.q * uy * rg;
  m.qvz = C.q * uz * rg;
  return m;
}

// Sums of 16 values over the warp's 32 lanes: every exchange halves the
// values a lane holds (16 shuffles in all, where 16 sums of their own take
// 80), until lane l has half of the sum of value order(l); one more exchange
// completes it.
__device__ __forceinline__ float sum16(float (&v)[16], int lane) {
#pragma unroll
  for (int h = 8, bit = 16; h >= 1; h >>= 1, bit >>= 1) {
    const bool up = lane & bit;
#pragma unroll
    for (int q = 0; q < h; ++q) {
      const float give = up ? v[q] : v[q + h], keep = up ? v[q + h] : v[q];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// the current of a warp's particles, one a lane
__device__ __forceinline__ void deposit_warp(float *J, bool valid, int ix, float x, const Move1 &m, const Push1 &C) {
  const int lane = threadIdx.x & 31, di = m.di;
  const float dx = m.dx, qvy = m.qvy, qvz = m.qvz;
  // deposit (dep_current_zamb): qvy, qvz halved, split at the cell edge.
  // a: the motion inside cell ix (all of it, or its part up to the edge);
  // b: for a crossing, the part inside cell ix + di
  const float hy = qvy / 2.0f, hz = qvz / 2.0f;
  const bool split = valid && di != 0;
  Seg1 a, b = Seg1{0.f, 0.f, 0.f, 0.f, 0.f};
  if (split) {
    const int ib = (di == 1);
    const float delta = (x + dx - ib) / dx;
    b = seg_current(1 - ib, (x + dx) - di, dx * delta, hy * delta, hz * delta, C.qnx);
    a = seg_current(x, (float)ib, dx * (1.0f - delta), hy * (1.0f - delta), hz * (1.0f - delta), C.qnx);
  } else {
    a = seg_current(x, x + dx, dx, hy, hz, C.qnx);
  }
  // the lanes of a cell are contiguous (cell order): each part is summed
  // over the lanes of the cell and one lane per cell adds the sums, a to
  // cell ix, b to ix + 1 or ix - 1 (one sum per direction)
  {
    const int ix0 = __shfl_sync(0xffffffffu, ix, 0);  // (by every lane, valid or not)
    if (__all_sync(0xffffffffu, valid && ix == ix0)) {
      // one cell (the usual case: 128 particles a cell): the sums of the part
      // inside it and of the parts past its two edges, 5 values each; the
      // value of lane pair p goes to its node with one reduction a lane
      const float zu = di == 1 ? 1.f : 0.f, zd = di == -1 ? 1.f : 0.f;
      float v[16] = {a.jx, a.y0, a.y1, a.z0, a.z1, zu * b.jx, zu * b.y0, zu * b.y1, zu * b.z0, zu * b.z1,
                     zd * b.jx, zd * b.y0, zd * b.y1, zd * b.z0, zd * b.z1, 0.f};
      const float sum = sum16(v, lane);
      const int q = lane >> 1, part = q / 5, e = q % 5;  // (order: value q in lanes 2 q, 2 q + 1)
      const int node = ix + (part == 1 ? 1 : (part == 2 ? -1 : 0)) + ((e == 2 || e == 4) ? 1 : 0);
      if ((lane & 1) == 0 && q < 15 && sum != 0.f) red(J, node, e == 0 ? 0 : (e <= 2 ? 1 : 2), sum);
      return;
    }
    const int key = valid ? ix : -1 - lane;
    const int knext = __shfl_down_sync(0xffffffffu, key, 1);
    const int kprev = __shfl_up_sync(0xffffffffu, key, 1);
    const unsigned lastmask = __ballot_sync(0xffffffffu, lane == 31 || knext != key);
    const int run_last = __ffs(lastmask & (0xffffffffu << lane)) - 1;
    const unsigned maxlen = __reduce_max_sync(0xffffffffu, (unsigned)(run_last - lane + 1));
    const bool head = valid && (lane == 0 || kprev != key);
    const unsigned up = __ballot_sync(0xffffffffu, split && di == 1);
    const unsigned down = __ballot_sync(0xffffffffu, split && di == -1);
    Seg1 sa = valid ? a : Seg1{0.f, 0.f, 0.f, 0.f, 0.f};
    run_sum(sa, run_last, maxlen);
    if (head) add_seg(J, ix, sa);
    if (up) {
      Seg1 sb = (di == 1) ? b : Seg1{0.f, 0.f, 0.f, 0.f, 0.f};
      run_sum(sb, run_last, maxlen);
      if (head) add_seg(J, ix + 1, sb);
    }
    if (down) {
      Seg1 sb = (di == -1) ? b : Seg1{0.f, 0.f, 0.f, 0.f, 0.f};
      run_sum(sb, run_last, maxlen);
      if (head) add_seg(J, ix - 1, sb);
    }
  }
}

// ---------------------------------------------------------------------------
// push + deposit, one particle per lane, warps over consecutive particles;
// boundaries, compaction by append, and (last CTA) injection + bookkeeping
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256, 4) k1_push(Parts b0, Parts b1, SpecState1 *st, const float *E, const float *B,
                                               float *Jall, Push1 C, Inject1 I, int *err) {
  __shared__ double sred[8];
  float *J = Jall + (size_t)(blockIdx.x % kJCopies) * C.jstride;
  __shared__ int s_last;
  const int cur = st->cur;
  const int n = st->np[cur];
  const int iter0 = st->iter, nmove0 = st->n_move;
  const int shift = (C.mw && ((float)(iter0 + 1) * C.dt) > (C.dx * (float)(nmove0 + 1))) ? 1 : 0;
  const Parts src = cur ? b1 : b0;
  const Parts dst = C.open ? (cur ? b0 : b1) : src;
  int *np_out = &st->np[1 - cur];
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  float ks = 0.f, kc = 0.f;
  int errbits = 0;
  for (int base = gw * 32; base < n; base += nw * 32) {
    const int i = base + lane;
    const bool valid = i < n;
    int ix = 0;
    float x = 0.f, ux = 0.f, uy = 0.f, uz = 0.f;
    if (valid) {
      ix = src.ix[i];
      x = src.x[i];
      ux = src.ux[i];
      uy = src.uy[i];
      uz = src.uz[i];
      if (ix < 0 || ix >= C.nx) {
        errbits |= ERR1_ESCAPE;
        ix = min(max(ix, 0), C.nx - 1);
      }
    }
    const Move1 m = push_lane(E, B, ix, x, ux, uy, uz, C);
    const float x1 = m.x1;
    const int di = m.di;
    if (valid) {
      const float y = m.kin - kc;
      const float t = ks + y;
      kc = (t - ks) - y;
      ks = t;
      if (!(fabsf(m.dx) < 1.0f)) errbits |= ERR1_ESCAPE;
    }
    deposit_warp(J, valid, ix, x, m, C);
    // boundaries (particles.c:1040-1062); with open boundaries the survivors
    // are appended to the other buffer, a warp at a time
    int nix = ix + di - shift;
    if (C.open) {
      const bool live = valid && nix >= 0 && nix < C.nx;
      const unsigned lm = __ballot_sync(0xffffffffu, live);
      int obase = 0;
      if (lane == 0 && lm) obase = atomicAdd(np_out, __popc(lm));
      obase = __shfl_sync(0xffffffffu, obase, 0);
      if (live) {
        const int o = obase + __popc(lm & ((1u << lane) - 1));
        if (o < C.cap) {
          dst.ix[o] = nix;
          dst.x[o] = x1;
          dst.ux[o] = ux;
          dst.uy[o] = uy;
          dst.uz[o] = uz;
        } else {
          errbits |= ERR1_OVERFLOW;
        }
      }
    } else if (valid) {
      nix += ((nix < 0) ? C.nx : 0) - ((nix >= C.nx) ? C.nx : 0);
      src.ix[i] = nix;
      src.x[i] = x1;
      src.ux[i] = ux;
      src.uy[i] = uy;
      src.uz[i] = uz;
    }
  }
  const double e = zc::block_sum_double<256>((double)ks - (double)kc, sred);
  if (threadIdx.x == 0 && e != 0.0) atomicAdd(&st->ekin_acc, e);
  if (errbits) atomicOr(err, errbits);
  // the last CTA to finish: every other CTA's stores and appends are done.
  // The barrier orders the CTA's writes before thread 0's fence, which is
  // cumulative, so one fence per CTA publishes them before the count.
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = (atomicAdd(&st->done, 1u) == gridDim.x - 1) ? 1 : 0;
  }
  __syncthreads();
  if (!s_last || threadIdx.x >= 32) return;
  __threadfence();
  int nn = C.open ? atomicAdd(np_out, 0) : n;
  if (shift && I.type != 1) {
    // spec_inject_particles into column nx-1 with the window's new offset
    const int ic = C.nx - 1;
    const float start = I.start / I.dx - (nmove0 + 1);
    const float end = I.end / I.dx - (nmove0 + 1);
    for (int k0 = 0; k0 < I.ppc; k0 += 32) {
      const int k = k0 + lane;
      const float pos = (float)((k + 0.5) / I.ppc);
      bool take = k < I.ppc;
      if (I.type == 2) take = take && ic + pos > start;
      if (I.type == 3) take = take && ic + pos > start && ic + pos < end;
      const unsigned m = __ballot_sync(0xffffffffu, take);
      if (take) {
        const int o = nn + __popc(m & ((1u << lane) - 1));
        if (o < C.cap) {
          dst.ix[o] = ic;
          dst.x[o] = pos;
          dst.ux[o] = I.ufl[0];
          dst.uy[o] = I.ufl[1];
          dst.uz[o] = I.ufl[2];
        } else {
          atomicOr(err, ERR1_OVERFLOW);
        }
      }
      nn += __popc(m);
    }
  }
  if (lane == 0) {
    if (nn > C.cap) {
      nn = C.cap;
      atomicOr(err, ERR1_OVERFLOW);
    }
    if (C.open) {
      st->np[1 - cur] = nn;
      st->np[cur] = 0;
      st->cur = 1 - cur;
    } else if (nn != n) {
      st->np[cur] = nn;
    }
    st->ekin = *(volatile double *)&st->ekin_acc;
    st->ekin_acc = 0.0;
    st->iter = iter0 + 1;
    st->n_move = nmove0 + shift;
    st->pushed += n;
    __threadfence();
    st->done = 0u;
  }
}

// ---------------------------------------------------------------------------
// counting sort by cell (spec_sort, particles.c:796-843) from the current
// buffer into the other: counts and cursors over nx cells, warp-aggregated
// atomics (the input is mostly sorted already); the scatter's last CTA
// switches the buffers
// ---------------------------------------------------------------------------
__global__ void k1_cell_count(Parts b0, Parts b1, const SpecState1 *st, int *cnt) {
  const int cur = st->cur;
  const int n = st->np[cur];
  const int *ix = cur ? b1.ix : b0.ix;
  for (int b = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; b < n; b += gridDim.x * blockDim.x) {
    const int i = b + (threadIdx.x & 31);
    const int key = i < n ? ix[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (i < n && (threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&cnt[key], __popc(peers));
  }
}

__global__ void k1_cell_scan(int *cnt, int nx, SpecState1 *st) {
  __shared__ int sw[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int b0 = 0; b0 < nx; b0 += 1024) {
    const int v = (b0 + (int)threadIdx.x < nx) ? cnt[b0 + threadIdx.x] : 0;
    int tot;
    const int pre = zc::block_exclusive_scan<1024>(v, tot, sw);
    if (b0 + (int)threadIdx.x < nx) cnt[b0 + threadIdx.x] = carry + pre;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) st->np[1 - st->cur] = st->np[st->cur];
}

__global__ void k1_cell_scatter(Parts b0, Parts b1, SpecState1 *st, int *cursor) {
  __shared__ int s_last;
  const int cur = st->cur;
  const int n = st->np[cur];
  const Parts src = cur ? b1 : b0, dst = cur ? b0 : b1;
  const int lane = threadIdx.x & 31;
  for (int b = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; b < n; b += gridDim.x * blockDim.x) {
    const int i = b + lane;
    const int key = i < n ? src.ix[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (i < n && lane == leader) base = atomicAdd(&cursor[key], __popc(peers));
    base = __shfl_sync(peers, base, leader);
    if (i < n) {
      const int o = base + __popc(peers & ((1u << lane) - 1));
      dst.ix[o] = key;
      dst.x[o] = src.x[i];
      dst.ux[o] = src.ux[i];
      dst.uy[o] = src.uy[i];
      dst.uz[o] = src.uz[i];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = (atomicAdd(&st->done, 1u) == gridDim.x - 1) ? 1 : 0;
  }
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    st->np[cur] = 0;
    st->cur = 1 - cur;
    __threadfence();
    st->done = 0u;
  }
}

// ---------------------------------------------------------------------------
// current update + field advance, one CTA (current.c:111-330, emf.c:379-580)
// ---------------------------------------------------------------------------
struct Smooth1 {
  int n;
  float sa[16], sb[16];
};

struct Fields1 {
  int nx;
  float dt, dx;
  int bc;            // 0 none, 1 periodic, 2 open (Mur)
  int cur_periodic;  // periodic guard fold of the current
  int mw;            // moving window
  Smooth1 S;
};

// the field's own counters on the device (emf->iter, emf->n_move)
struct FieldState1 {
  int iter, n_move;
};

__device__ __forceinline__ void yee_b1(const float *E, float *B, int nx, float dt_dx) {
  for (int i = (int)threadIdx.x - 1; i <= nx; i += blockDim.x) {
    const int k = (i + GC0) * 3;
    B[k + 1] += (dt_dx * (E[k + 3 + 2] - E[k + 2]));
    B[k + 2] += (-dt_dx * (E[k + 3 + 1] - E[k + 1]));
  }
}

__device__ __forceinline__ void yee_e1(float *E, const float *B, const float *J, int nx, float dt, float dt_dx) {
  for (int i = threadIdx.x; i <= nx + 1; i += blockDim.x) {
    const int k = (i + GC0) * 3;
    E[k + 0] += (-dt * J[k + 0]);
    E[k + 1] += (-dt_dx * (B[k + 2] - B[k - 3 + 2]) - dt * J[k + 1]);
    E[k + 2] += (+dt_dx * (B[k + 1] - B[k - 3 + 1]) - dt * J[k + 2]);
  }
}

// periodic guard cells of E and B (emf_update_gc, emf.c:476-500): -1 <- nx-1
// and nx <- 0 only; the second upper guard cell nx+1 keeps the value yee_e
// gave it.  Threads 0..11 of the CTA.
__device__ __forceinline__ void periodic_gc1(float *E, float *B, int nx) {
  if (threadIdx.x < 12) {
    float *F = (threadIdx.x < 6) ? E : B;
    const int t = threadIdx.x % 6, g = t / 3, c = t % 3;
    const int gi = (g == 0) ? -1 : nx;
    const int src = (g == 0) ? nx - 1 : 0;
    F[(gi + GC0) * 3 + c] = F[(src + GC0) * 3 + c];
  }
}

__device__ __forceinline__ void mur1(float *e, float *mur, int nx, float dt, float dx) {
  // first-order Mur (mur_abc, emf.c:379-415); mur = fld[2][3], tmp[2][3]
  float *fld = mur, *tmp = mur + 6;
  const float S = (dt - dx) / (dt + dx);
  const int lo = (0 + GC0) * 3, hi = (nx - 1 + GC0) * 3;
  fld[1] = tmp[1] + S * (e[lo + 1] - fld[1]);
  fld[2] = tmp[2] + S * (e[lo + 2] - fld[2]);
  e[(-1 + GC0) * 3 + 1] = fld[1];
  e[(-1 + GC0) * 3 + 2] = fld[2];
  tmp[1] = e[lo + 1];
  tmp[2] = e[lo + 2];
  fld[4] = tmp[4] + S * (e[hi + 1] - fld[4]);
  fld[5] = tmp[5] + S * (e[hi + 2] - fld[5]);
  e[(nx + GC0) * 3 + 1] = fld[4];
  e[(nx + GC0) * 3 + 2] = fld[5];
  tmp[4] = e[hi + 1];
  tmp[5] = e[hi + 2];
}

// SM: the four grids (two current buffers, E, B) live in shared memory for
// the whole kernel, else the kernel works on the global buffers (Jdep and
// Jout then serve as the filter's two buffers).  Jdep (kJCopies copies,
// summed first) is left zero for the next step's deposit; Jout holds the
// filtered current.
template <bool SM>
__global__ void __launch_bounds__(1024) k1_fields(float *E, float *B, float *Jdep, float *Jout, float *mur,
                                                  FieldState1 *fs, Fields1 M) {
  extern __shared__ float smem[];
  const int nx = M.nx;
  const int nf = (nx + GC0 + GC1) * 3;
  const int iter = fs->iter + 1, nmove0 = fs->n_move;
  float *ja, *jb, *e, *b;
  if (SM) {
    ja = smem;
    jb = smem + nf;
    e = smem + 2 * nf;
    b = smem + 3 * nf;
    // every load of a round is issued before its stores (one L2 round trip
    // per kFieldUnroll x blockDim.x elements)
    for (int k0 = threadIdx.x; k0 < nf; k0 += kFieldUnroll * blockDim.x) {
      float v[kFieldUnroll][kJCopies], ve[kFieldUnroll], vb[kFieldUnroll];
#pragma unroll
      for (int r = 0; r < kFieldUnroll; ++r) {
        const int k = k0 + r * blockDim.x;
        const bool in = k < nf;
#pragma unroll
        for (int c = 0; c < kJCopies; ++c) v[r][c] = in ? Jdep[c * nf + k] : 0.f;
        ve[r] = in ? E[k] : 0.f;
        vb[r] = in ? B[k] : 0.f;
      }
#pragma unroll
      for (int r = 0; r < kFieldUnroll; ++r) {
        const int k = k0 + r * blockDim.x;
        if (k < nf) {
          float sum = 0.f;
#pragma unroll
          for (int c = 0; c < kJCopies; ++c) {
            sum += v[r][c];
            Jdep[c * nf + k] = 0.f;
          }
          ja[k] = sum;
          e[k] = ve[r];
          b[k] = vb[r];
        }
      }
    }
  } else {
    ja = Jdep;
    jb = Jout;
    e = E;
    b = B;
    for (int k = threadIdx.x; k < nf; k += blockDim.x) {
      float v = 0.f;
#pragma unroll
      for (int c = 0; c < kJCopies; ++c) {
        v += Jdep[c * nf + k];
        if (c) Jdep[c * nf + k] = 0.f;
      }
      Jdep[k] = v;
    }
  }
  __syncthreads();
  // current_update_gc: J[i] += J[nx + i] for i = -1, 0, 1, then the upper
  // cells copy the lower (current.c:112-132)
  float *J = ja, *O = jb;
  if (M.cur_periodic) {
    if (threadIdx.x < 9) {
      const int i = (int)threadIdx.x / 3 - 1, c = threadIdx.x % 3;
      J[(i + GC0) * 3 + c] += J[(nx + i + GC0) * 3 + c];
    }
    __syncthreads();
    if (threadIdx.x < 9) {
      const int i = (int)threadIdx.x / 3 - 1, c = threadIdx.x % 3;
      J[(nx + i + GC0) * 3 + c] = J[(i + GC0) * 3 + c];
    }
    __syncthreads();
  }
  // the filter passes [sa, sb, sa] (kernel_x, current.c:265-297), out of place
  for (int p = 0; p < M.S.n; ++p) {
    const float sa = M.S.sa[p], sb = M.S.sb[p];
    for (int k = threadIdx.x; k < nx * 3; k += blockDim.x) {
      const int i = k / 3, c = k % 3;
      O[(i + GC0) * 3 + c] =
          sa * J[(i - 1 + GC0) * 3 + c] + sb * J[(i + GC0) * 3 + c] + sa * J[(i + 1 + GC0) * 3 + c];
    }
    __syncthreads();
    // guard cells: periodic copies of the filtered cells, else as they were
    if (threadIdx.x < 9) {
      const int g = threadIdx.x / 3, c = threadIdx.x % 3;  // g: guard -1, nx, nx+1
      const int gi = (g == 0) ? -1 : nx + g - 1;
      const int src = (g == 0) ? nx - 1 : g - 1;
      O[(gi + GC0) * 3 + c] = M.cur_periodic ? O[(src + GC0) * 3 + c] : J[(gi + GC0) * 3 + c];
    }
    __syncthreads();
    float *t = J;
    J = O;
    O = t;
  }
  // the filtered current for reports
  if (SM) {
    for (int k = threadIdx.x; k < nf; k += blockDim.x) Jout[k] = J[k];
  } else if (J != Jout) {
    for (int k = threadIdx.x; k < nf; k += blockDim.x) Jout[k] = J[k];
    __syncthreads();
    J = Jout;
  }
  // emf_advance (emf.c:548-566)
  const float hdt = M.dt / 2.0f;
  yee_b1(e, b, nx, hdt / M.dx);
  __syncthreads();
  yee_e1(e, b, J, nx, M.dt, M.dt / M.dx);
  __syncthreads();
  if (M.bc == 2 && threadIdx.x == 0) {
    mur1(e, mur, nx, M.dt, M.dx);
  }
  __syncthreads();
  yee_b1(e, b, nx, hdt / M.dx);
  __syncthreads();
  if (M.bc == 1) periodic_gc1(e, b, nx);
  if (!SM)
    for (int k = threadIdx.x; k < nf; k += blockDim.x) Jdep[k] = 0.f;
  __syncthreads();
  // window shift (emf_move_window, emf.c:513-540): cells move left by one,
  // cells nx-1 .. nx+1 become zero
  const int shift = (M.mw && ((float)iter * M.dt) > (M.dx * (float)(nmove0 + 1))) ? 1 : 0;
  if (SM) {
    for (int k = threadIdx.x; k < nf; k += blockDim.x) {
      E[k] = shift ? ((k < nx * 3) ? e[k + 3] : 0.f) : e[k];
      B[k] = shift ? ((k < nx * 3) ? b[k + 3] : 0.f) : b[k];
    }
  } else if (shift) {
    for (int base = 0; base < nf; base += blockDim.x) {
      // E[k] <- E[k + 3] for k < nf - 3, every value read before any write
      const int k = base + threadIdx.x;
      float ve = 0.f, vb = 0.f;
      if (k < nf - 3) {
        ve = E[k + 3];
        vb = B[k + 3];
      }
      __syncthreads();
      if (k < nf - 3) {
        E[k] = ve;
        B[k] = vb;
      }
      __syncthreads();
    }
    for (int k = nx * 3 + threadIdx.x; k < nf; k += blockDim.x) {
      E[k] = 0.f;
      B[k] = 0.f;
    }
  }
  if (threadIdx.x == 0) {
    fs->iter = iter;
    fs->n_move = nmove0 + shift;
  }
}

// ---------------------------------------------------------------------------
// Several steps in one launch: a cooperative grid that stays on the GPU, one
// grid-wide barrier a step.  A step of the two kernels above takes 31 us (13
// for the push, 9 for one CTA's fields, the rest between launches) for work
// that fits the chip; nothing in it is bound by bandwidth.  Here
//   - every CTA keeps its share of the particles in shared memory for all the
//     steps (a particle that leaves the grid leaves a hole);
//   - every CTA keeps E and B there too and advances them by itself, all CTAs
//     alike: after the barrier each reads the deposited current (from L2) and
//     makes the filter and the field advance of a few thousand cells, which is
//     cheaper than a second barrier;
//   - the deposits go to one of three buffers in turn: the one that was read a
//     step ago is cleared while nobody uses it;
//   - the column that a window move uncovers goes to the CTAs in turn;
//   - waits are bounded: past the limit an error bit is set and every CTA
//     leaves (the others run into theirs).
// A step takes 10.5 to 11.6 us (1000 cells, 72 to 127 thousand particles, the
// cell sort every 16 steps included): about 2 each for the push with its
// deposit, the barrier, the filter and the advance.  With the particles in
// global memory, compacted every step, it took 16.
// ---------------------------------------------------------------------------
constexpr int kRunSpecies = 4;   // species of a run
constexpr int kRunCopies = 4;    // copies of a deposit buffer
constexpr int kRunThreads = 1024;
constexpr int kBarrierPolls = 1 << 21;

// floats of a grid, rounded up to whole 16-byte units
__host__ __device__ constexpr int grid_stride1(int nx) { return ((nx + GC0 + GC1) * 3 + 3) & ~3; }

struct RunSpecies1 {
  Parts b0, b1;
  SpecState1 *st;
  const float *lat;          // in-cell positions of the injected lattice
  int slots;                 // particles a CTA has room for (a multiple of kRunThreads)
  Push1 C;
  Inject1 I;
};
struct Run1 {
  int nsp, steps, phase;     // phase: the first step's deposit buffer
  unsigned bar0;             // the barrier's count before this launch
  unsigned *bar;
  float *Jrun;               // deposits [3][kRunCopies][grid_stride1]
  float *E, *B, *Jout, *mur;
  FieldState1 *fs;
  int *err;
  Fields1 M;
  RunSpecies1 sp[kRunSpecies];
};

// all CTAs of the grid; false when the limit ran out
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned target) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    int ok = 0;
    for (int it = 0; it < kBarrierPolls && !ok; ++it) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      ok = (int)(v - target) >= 0;
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// The injected lattice points of a window move that pass the density test
// (spec_set_x, particles.c:250-300): [*first, *first + result).  All threads
// of the CTA; the usual cases (all of them, none) need no look at the points.
__device__ __forceinline__ int lattice_range(const Inject1 &I, const float *lat, int nx, int n_move, int *first) {
  const int ic = nx - 1;
  *first = 0;
  if (I.type == 1) return 0;
  if (I.type == 0) return I.ppc;
  const float start = I.start / I.dx - n_move, end = I.end / I.dx - n_move;
  if ((float)nx <= start) return 0;
  if ((float)ic > start && (I.type == 2 || (float)nx < end)) return I.ppc;
  int below = 0, inside = 0;
  for (int q0 = 0; q0 < I.ppc; q0 += kRunThreads) {
    const int q = q0 + (int)threadIdx.x;
    const float pos = q < I.ppc ? lat[q] : 0.f;
    const bool past = ic + pos > start;
    below += __syncthreads_count(q < I.ppc && !past);
    inside += __syncthreads_count(q < I.ppc && past && (I.type == 2 || ic + pos < end));
  }
  *first = below;
  return inside;
}

__global__ void __launch_bounds__(kRunThreads, 1) k1_run(const __grid_constant__ Run1 R) {
  extern __shared__ __align__(16) float sm[];
  __shared__ double sred[kRunThreads / 32];
  __shared__ int s_n[kRunThreads / 32], s_at;
  __shared__ float s_mur[12];
  // per species: slots in use (holes among them), first particle, the buffer
  // that holds them, counters, particles pushed
  __shared__ int s_used[kRunSpecies], s_i0[kRunSpecies], s_cur[kRunSpecies], s_iter[kRunSpecies], s_move[kRunSpecies];
  __shared__ unsigned s_pushed[kRunSpecies];
  const Fields1 &M = R.M;
  const int nx = M.nx, nf = grid_stride1(nx), nv = (nx + GC0 + GC1) * 3;  // (values past nv: unused)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int oe = 0, ob = nf, oj = 2 * nf, oo = 3 * nf;  // E, B, J and a second buffer
  for (int k = tid; k < nf; k += kRunThreads) {
    sm[oe + k] = k < nv ? R.E[k] : 0.f;
    sm[ob + k] = k < nv ? R.B[k] : 0.f;
  }
  if (tid < 12) s_mur[tid] = R.mur[tid];
  // the species' particles: arrays of `slots` cells, positions and momenta,
  // after the grids
  if (tid < R.nsp) {
    const RunSpecies1 &S = R.sp[tid];
    const int cur = S.st->cur, n = S.st->np[cur], share = (n + (int)gridDim.x - 1) / (int)gridDim.x;
    const int i0 = min(n, (int)blockIdx.x * share);
    s_cur[tid] = cur;
    s_iter[tid] = S.st->iter;
    s_move[tid] = S.st->n_move;
    s_i0[tid] = i0;
    s_used[tid] = min(min(share, n - i0), S.slots);
    s_pushed[tid] = 0;
  }
  __syncthreads();
  for (int k = 0, at = 4 * nf; k < R.nsp; ++k) {
    const RunSpecies1 &S = R.sp[k];
    const Parts src = s_cur[k] ? S.b1 : S.b0;
    const int i0 = s_i0[k];
    int *ix = reinterpret_cast<int *>(sm + at);
    float *f = sm + at + S.slots;
    for (int q = tid; q < s_used[k]; q += kRunThreads) {
      ix[q] = src.ix[i0 + q];
      f[q] = src.x[i0 + q];
      f[S.slots + q] = src.ux[i0 + q];
      f[2 * S.slots + q] = src.uy[i0 + q];
      f[3 * S.slots + q] = src.uz[i0 + q];
    }
    at += 5 * S.slots;
  }
  int fiter = R.fs->iter, fmove = R.fs->n_move;
  int errbits = 0;
  __syncthreads();
  for (int step = 0; step < R.steps; ++step) {
    const bool last = step == R.steps - 1;
    const int ph = (R.phase + step) % 3;
    float *J = R.Jrun + ((size_t)ph * kRunCopies + blockIdx.x % kRunCopies) * nf;
#pragma unroll 1
    for (int k = 0, at = 4 * nf; k < R.nsp; ++k) {
      const RunSpecies1 &S = R.sp[k];
      const Push1 &C = S.C;
      const int iter = s_iter[k] + step + 1, moved = s_move[k], used = s_used[k];
      const int shift = (C.mw && ((float)iter * C.dt) > (C.dx * (float)(moved + 1))) ? 1 : 0;
      int *six = reinterpret_cast<int *>(sm + at);
      float *f = sm + at + S.slots;
      float ks = 0.f, kc = 0.f;
#pragma unroll 1
      for (int b = 0; b < used; b += kRunThreads) {
        const int q = b + tid;
        int ix = q < used ? six[q] : -1;
        const bool valid = ix >= 0;
        const unsigned vm = __ballot_sync(0xffffffffu, valid);
        if (!vm) continue;  // a warp of holes
        if (lane == 0) atomicAdd(&s_pushed[k], (unsigned)__popc(vm));
        float x = 0.f, ux = 0.f, uy = 0.f, uz = 0.f;
        if (valid) {
          x = f[q];
          ux = f[S.slots + q];
          uy = f[2 * S.slots + q];
          uz = f[3 * S.slots + q];
          if (ix >= C.nx) {
            errbits |= ERR1_ESCAPE;
            ix = C.nx - 1;
          }
        } else {
          ix = 0;
        }
        const Move1 m = push_lane(sm + oe, sm + ob, ix, x, ux, uy, uz, C);
        if (valid) {
          const float y = m.kin - kc;
          const float t = ks + y;
          kc = (t - ks) - y;
          ks = t;
          if (!(fabsf(m.dx) < 1.0f)) errbits |= ERR1_ESCAPE;
          int nix = ix + m.di - shift;
          if (!C.open) nix += ((nix < 0) ? C.nx : 0) - ((nix >= C.nx) ? C.nx : 0);
          six[q] = (nix >= 0 && nix < C.nx) ? nix : -1;
          f[q] = m.x1;
          f[S.slots + q] = ux;
          f[2 * S.slots + q] = uy;
          f[3 * S.slots + q] = uz;
        }
        deposit_warp(J, valid, ix, x, m, C);
      }
      if (last) {
        const double e = zc::block_sum_double<kRunThreads>((double)ks - (double)kc, sred);
        if (tid == 0 && e != 0.0) atomicAdd(&S.st->ekin_acc, e);
      }
      __syncthreads();  // the species' slots and counters are read
      int n = 0;
      // the column that the move uncovered (spec_inject_particles)
      if (shift && blockIdx.x == (unsigned)iter % gridDim.x) {
        int first;
        n = lattice_range(S.I, S.lat, C.nx, moved + 1, &first);
        for (int q = tid; q < n; q += kRunThreads) {
          const int o = used + q;
          if (o >= S.slots) {  // (room is sized for every column: cannot happen)
            errbits |= ERR1_OVERFLOW;
            continue;
          }
          six[o] = C.nx - 1;
          f[o] = S.lat[first + q];
          f[S.slots + o] = S.I.ufl[0];
          f[2 * S.slots + o] = S.I.ufl[1];
          f[3 * S.slots + o] = S.I.ufl[2];
        }
      }
      if (tid == 0) {
        s_move[k] = moved + shift;
        s_used[k] = min(used + n, S.slots);
      }
      at += 5 * S.slots;
    }
    if (!grid_barrier(R.bar, R.bar0 + (unsigned)(step + 1) * gridDim.x)) {
      if (tid == 0) atomicOr(R.err, ERR1_TIMEOUT);
      return;
    }
    // the deposited current; the buffer read a step ago is cleared
    {
      const float *Jr = R.Jrun + (size_t)ph * kRunCopies * nf;
      for (int k = 4 * tid; k < nf; k += 4 * kRunThreads) {
        float4 v[kRunCopies];
#pragma unroll
        for (int c = 0; c < kRunCopies; ++c) v[c] = __ldcg(reinterpret_cast<const float4 *>(&Jr[c * nf + k]));
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int c = 0; c < kRunCopies; ++c) {
          sum.x += v[c].x;
          sum.y += v[c].y;
          sum.z += v[c].z;
          sum.w += v[c].w;
        }
        *reinterpret_cast<float4 *>(&sm[oj + k]) = sum;
      }
      float *Jz = R.Jrun + (size_t)((ph + 2) % 3) * kRunCopies * nf;
      for (int k = 4 * (blockIdx.x * kRunThreads + tid); k < kRunCopies * nf; k += 4 * gridDim.x * kRunThreads)
        *reinterpret_cast<float4 *>(&Jz[k]) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    // current fold, filter, field advance, window shift: as k1_fields
    if (M.cur_periodic) {
      float *Jc = sm + oj;
      if (tid < 9) Jc[(tid / 3 - 1 + GC0) * 3 + tid % 3] += Jc[(nx + tid / 3 - 1 + GC0) * 3 + tid % 3];
      __syncthreads();
      if (tid < 9) Jc[(nx + tid / 3 - 1 + GC0) * 3 + tid % 3] = Jc[(tid / 3 - 1 + GC0) * 3 + tid % 3];
      __syncthreads();
    }
    for (int p = 0; p < M.S.n; ++p) {
      const float sa = M.S.sa[p], sb = M.S.sb[p];
      const float *Ji = sm + oj;
      float *O = sm + oo;
      // four values a thread; the guard cells keep theirs
      for (int k = 4 * tid; k < nf; k += 4 * kRunThreads) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 A = k >= 4 ? *reinterpret_cast<const float4 *>(Ji + k - 4) : z;
        const float4 B = *reinterpret_cast<const float4 *>(Ji + k);
        const float4 C = k + 4 < nf ? *reinterpret_cast<const float4 *>(Ji + k + 4) : z;
        float4 r = make_float4(sa * A.y + sb * B.x + sa * B.w, sa * A.z + sb * B.y + sa * C.x,
                               sa * A.w + sb * B.z + sa * C.y, sa * B.x + sb * B.w + sa * C.z);
        if (k < GC0 * 3 || k + 4 > (nx + GC0) * 3) {
          const int lo = GC0 * 3 - k, hi = (nx + GC0) * 3 - k;  // filtered: lo <= e < hi
          r.x = (0 >= lo && 0 < hi) ? r.x : B.x;
          r.y = (1 >= lo && 1 < hi) ? r.y : B.y;
          r.z = (2 >= lo && 2 < hi) ? r.z : B.z;
          r.w = (3 >= lo && 3 < hi) ? r.w : B.w;
        }
        *reinterpret_cast<float4 *>(O + k) = r;
      }
      __syncthreads();
      if (M.cur_periodic) {  // copies of the filtered cells
        if (tid < 9) {
          const int g = tid / 3, c = tid % 3, gi = (g == 0) ? -1 : nx + g - 1, from = (g == 0) ? nx - 1 : g - 1;
          O[(gi + GC0) * 3 + c] = O[(from + GC0) * 3 + c];
        }
        __syncthreads();
      }
      const int t = oj;
      oj = oo;
      oo = t;
    }
    if (last && blockIdx.x == 0)
      for (int k = tid; k < nv; k += kRunThreads) R.Jout[k] = sm[oj + k];
    const float hdt = M.dt / 2.0f;
    yee_b1(sm + oe, sm + ob, nx, hdt / M.dx);
    __syncthreads();
    yee_e1(sm + oe, sm + ob, sm + oj, nx, M.dt, M.dt / M.dx);
    __syncthreads();
    if (M.bc == 2) {
      if (tid == 0) mur1(sm + oe, s_mur, nx, M.dt, M.dx);
      __syncthreads();
    }
    yee_b1(sm + oe, sm + ob, nx, hdt / M.dx);
    __syncthreads();
    if (M.bc == 1) {
      periodic_gc1(sm + oe, sm + ob, nx);
      __syncthreads();
    }
    fiter += 1;
    if (M.mw && ((float)fiter * M.dt) > (M.dx * (float)(fmove + 1))) {
      for (int k = tid; k < nf; k += kRunThreads) {
        sm[oj + k] = (k < nx * 3) ? sm[oe + k + 3] : 0.f;
        sm[oo + k] = (k < nx * 3) ? sm[ob + k + 3] : 0.f;
      }
      __syncthreads();
      int t = oe;
      oe = oj;
      oj = t;
      t = ob;
      ob = oo;
      oo = t;
      fmove += 1;
    }
  }
  // The particles back: to their places, or with open ends (or a window) the
  // survivors appended to the other buffer, one atomic a CTA.
  {
    for (int k = 0, at = 4 * nf; k < R.nsp; ++k) {
      const RunSpecies1 &S = R.sp[k];
      const bool open = S.C.open;
      const int cur = s_cur[k], used = s_used[k];
      const Parts dst = (cur != 0) != open ? S.b1 : S.b0;  // open: the other one
      const int *six = reinterpret_cast<const int *>(sm + at);
      const float *f = sm + at + S.slots;
      for (int b = 0; b < used; b += kRunThreads) {
        const int q = b + tid, ix = q < used ? six[q] : -1;
        int o = s_i0[k] + q;
        if (open) {
          const unsigned lm = __ballot_sync(0xffffffffu, ix >= 0);
          if (lane == 0) s_n[warp] = __popc(lm);
          __syncthreads();
          if (warp == 0) {
            const int v = s_n[lane];
            int inc = v;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
              const int y = __shfl_up_sync(0xffffffffu, inc, d);
              if (lane >= d) inc += y;
            }
            s_n[lane] = inc - v;
            if (lane == 31) s_at = inc ? atomicAdd(&S.st->np[1 - cur], inc) : 0;
          }
          __syncthreads();
          o = s_at + s_n[warp] + __popc(lm & ((1u << lane) - 1));
          __syncthreads();
        }
        if (ix >= 0) {
          if (o < S.C.cap) {
            dst.ix[o] = ix;
            dst.x[o] = f[q];
            dst.ux[o] = f[S.slots + q];
            dst.uy[o] = f[2 * S.slots + q];
            dst.uz[o] = f[3 * S.slots + q];
          } else {  // (the host makes room for every column: cannot happen)
            errbits |= ERR1_OVERFLOW;
          }
        }
      }
      if (tid == 0)
        atomicAdd(reinterpret_cast<unsigned long long *>(&S.st->pushed), (unsigned long long)s_pushed[k]);
      if (blockIdx.x == 0 && tid == 0) {
        // (the other CTAs read these before the first barrier)
        if (open) {
          S.st->np[cur] = 0;
          S.st->cur = 1 - cur;
        }
        S.st->ekin = __ldcg(&S.st->ekin_acc);
        S.st->ekin_acc = 0.0;
        S.st->iter = s_iter[k] + R.steps;
        S.st->n_move = s_move[k];
      }
      at += 5 * S.slots;
    }
  }
  if (errbits) atomicOr(R.err, errbits);
  if (blockIdx.x != 0) return;
  for (int k = tid; k < nv; k += kRunThreads) {
    R.E[k] = sm[oe + k];
    R.B[k] = sm[ob + k];
  }
  if (tid < 12) R.mur[tid] = s_mur[tid];
  if (tid == 0) {
    R.fs->iter = fiter;
    R.fs->n_move = fmove;
  }
}

// laser launch (emf_add_laser, em1d/emf.c:191-260): the plane-wave pulse
// added to Ey/Ez at the cell nodes and By/Bz half a cell ahead, with the
// reference's float/double mix; periodic runs then refresh the guard cells
__global__ void __launch_bounds__(1024) k1_laser(float *E, float *B, int nx, zc::LaserConst L, int periodic) {
  const float amp = L.omega0 * L.a0;
  const float cp = cos((double)L.polarization), sp = sin((double)L.polarization);
  const float k = L.omega0;
  for (int i = threadIdx.x; i < nx; i += blockDim.x) {
    const float z = i * L.dx, z2 = z + L.dx / 2;
    const float a = amp * zc::laser_env(L, z), a2 = amp * zc::laser_env(L, z2);
    const int o = (i + GC0) * 3;
    E[o + 1] += +a * cos((double)(k * z)) * cp;
    E[o + 2] += +a * cos((double)(k * z)) * sp;
    B[o + 1] += -a2 * cos((double)(k * z2)) * sp;
    B[o + 2] += +a2 * cos((double)(k * z2)) * cp;
  }
  __syncthreads();
  if (periodic) periodic_gc1(E, B, nx);
}

// field energy per component (emf.c:590-612): double sums of float squares, a
// block a component (24 us by one block, double precision being slow here; 6)
__global__ void __launch_bounds__(1024) k1_emf_energy(const float *E, const float *B, int nx, float dx, double *out) {
  __shared__ double sred[32];
  const int c = blockIdx.x;
  const float *F = (c < 3) ? E : B;
  double s = 0.0;
  for (int i = threadIdx.x; i < nx; i += blockDim.x) {
    const float v = F[(i + GC0) * 3 + c % 3];
    s += (double)(v * v);
  }
  const double t = zc::block_sum_double<1024>(s, sred);
  if (threadIdx.x == 0) out[c] = t * (0.5 * dx);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct Species1 {
  float m_q, q;
  Inject1 inj;
  int iter = 0, n_move = 0;  // mirrors of the device counters
  int cap = 0;
  long long np_bound = 0;    // upper bound of the device count
  Parts buf[2] = {};
  SpecState1 *d_st = nullptr;
  float *d_lat = nullptr;    // in-cell positions of an injected cell's particles (null: none injected)
};

}  // namespace zc1

using namespace zc1;

struct zc1_sim {
  int nx;
  float box, dx, dt;
  int device;
  int field_bc, current_periodic, part_open, mw, sort_every;
  int push_ctas = 0;         // cap of the push's CTAs (0: one wave)
  int iter = 0, n_move = 0;  // mirrors of the field's device counters
  Smooth1 smooth{};
  cudaStream_t st = nullptr;
  float *E = nullptr, *B = nullptr, *Jdep = nullptr, *Jout = nullptr, *mur = nullptr;
  FieldState1 *d_fs = nullptr;
  int *d_err = nullptr, *d_cnt = nullptr;
  double *d_emf = nullptr;
  // several steps in one launch (k1_run): its deposit buffers and barrier,
  // the barrier's count and the next deposit buffer
  float *Jrun = nullptr;
  unsigned *run_bar = nullptr;
  unsigned bar_count = 0;
  int run_phase = 0;
  size_t run_smem = 0;     // its shared memory at most (0: it cannot be used)
  int sms = 1;             // multiprocessors: its CTAs, which wait on one another, at most
  size_t fields_smem = 0;  // dynamic shared memory of the fields kernel (0: global variant)
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  float last_ms = 0.f;
  int timing = 0;          // steps enqueued since ev0, not yet waited for
  long long launches = 0;  // kernels launched by the steps so far
  // the captured block of sort_every steps (the last one sorts), and the
  // same block with an event pair around every kernel for profiling
  cudaGraphExec_t block = nullptr, block_prof = nullptr;
  int block_kernels = 0, block_prof_kernels = 0;
  size_t prof_graph_slots = 0;  // event pairs the profiling graph records
  int capturing = 0;
  // optional per-kernel timing: an event pair around every launch, summed
  // per kind after the steps (zc1_set_profile / zc1_get_profile)
  int profile = 0;
  std::vector<cudaEvent_t> prof_ev;
  std::vector<int> prof_kind;
  size_t prof_used = 0;
  double prof_ms[ZC1_NKIND] = {};
  long long prof_n[ZC1_NKIND] = {};
  std::vector<Species1> sp;
};

namespace {

zc_status fail1f(zc_status s, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  zc::set_error_message(buf);
  return s;
}

zc_status fail1(zc_status s, const char *what) { return fail1f(s, "%s", what); }

#define CK1(call)                                                                               \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess) return fail1f(ZC_ECUDA, "%s: %s", #call, cudaGetErrorString(e_));    \
  } while (0)
#define TRY1(call)                \
  do {                            \
    zc_status r_ = (call);        \
    if (r_ != ZC_OK) return r_;   \
  } while (0)

struct Guard1 {
  int old = 0;
  explicit Guard1(int d) {
    cudaGetDevice(&old);
    cudaSetDevice(d);
  }
  ~Guard1() { cudaSetDevice(old); }
};

// The calls that are waiting for steps on a device right now, over all threads
// (see run_steps).
std::atomic<int> g_waiting[64];
struct Waiting {
  std::atomic<int> &n;
  explicit Waiting(int device) : n(g_waiting[device & 63]) { n.fetch_add(1); }
  ~Waiting() { n.fetch_sub(1); }
};

constexpr int kPushThreads = 256;
constexpr int kMaxCtas = 152 * 4;  // the push CTAs resident together (4 per SM)

// CTAs of the push: one particle per thread, up to one wave, or up to the
// simulation's own cap (simulations that share the GPU leave each other room)
int push_blocks(const zc1_sim *s, int cap) {
  const int most = s->push_ctas > 0 ? std::min(s->push_ctas, kMaxCtas) : kMaxCtas;
  return std::max(1, std::min(most, (cap + kPushThreads - 1) / kPushThreads));
}

int sort_blocks(const zc1_sim *s) { return s->push_ctas > 0 ? std::min(s->push_ctas, kMaxCtas) : kMaxCtas; }

zc_status alloc_parts(Parts &p, int cap) {
  CK1(cudaMalloc(&p.ix, sizeof(int) * (size_t)std::max(cap, 1)));
  CK1(cudaMalloc(&p.x, sizeof(float) * (size_t)std::max(cap, 1)));
  CK1(cudaMalloc(&p.ux, sizeof(float) * (size_t)std::max(cap, 1)));
  CK1(cudaMalloc(&p.uy, sizeof(float) * (size_t)std::max(cap, 1)));
  CK1(cudaMalloc(&p.uz, sizeof(float) * (size_t)std::max(cap, 1)));
  return ZC_OK;
}

void free_parts(Parts &p) {
  cudaFree(p.ix);
  cudaFree(p.x);
  cudaFree(p.ux);
  cudaFree(p.uy);
  cudaFree(p.uz);
  p = Parts{};
}

zc_status copy_parts(const Parts &src, const Parts &dst, int n, cudaStream_t st) {
  if (n <= 0) return ZC_OK;
  CK1(cudaMemcpyAsync(dst.ix, src.ix, sizeof(int) * n, cudaMemcpyDeviceToDevice, st));
  CK1(cudaMemcpyAsync(dst.x, src.x, sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
  CK1(cudaMemcpyAsync(dst.ux, src.ux, sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
  CK1(cudaMemcpyAsync(dst.uy, src.uy, sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
  CK1(cudaMemcpyAsync(dst.uz, src.uz, sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
  return ZC_OK;
}

zc_status read_state(zc1_sim *s, const Species1 &p, SpecState1 &h) {
  CK1(cudaMemcpyAsync(&h, p.d_st, sizeof(SpecState1), cudaMemcpyDeviceToHost, s->st));
  CK1(cudaStreamSynchronize(s->st));
  return ZC_OK;
}

void drop_graph(zc1_sim *s) {
  if (s->block) cudaGraphExecDestroy(s->block);
  if (s->block_prof) cudaGraphExecDestroy(s->block_prof);
  s->block = s->block_prof = nullptr;
  s->block_kernels = s->block_prof_kernels = 0;
  s->prof_graph_slots = 0;
  s->prof_used = 0;
}

zc_status check_err(zc1_sim *s) {
  int e = 0;
  CK1(cudaMemcpyAsync(&e, s->d_err, sizeof(int), cudaMemcpyDeviceToHost, s->st));
  CK1(cudaStreamSynchronize(s->st));
  if (e & ERR1_TIMEOUT) return fail1(ZC_ETIMEOUT, "a wait for the other blocks of a 1-D step timed out");
  if (e & ERR1_OVERFLOW) return fail1(ZC_EOVERFLOW, "1-D particle buffer full at injection");
  if (e & ERR1_ESCAPE) return fail1(ZC_EPARTICLE_ESCAPE, "a particle moved a cell or more, or left the grid");
  return ZC_OK;
}

// room for `steps` more steps of injection in both buffers of every species, keeping
// the current ones; the device count is read (a sync) only when its upper
// bound no longer fits, and the buffers grow only when the true count does
// not (which also drops the captured graph: it holds the old buffers)
zc_status ensure_cap(zc1_sim *s, int steps) {
  for (auto &p : s->sp) {
    // at most one window move, hence one injected column, per step
    const long long extra = (s->mw && p.inj.type != 1) ? (long long)steps * p.inj.ppc : 0;
    if (p.np_bound + extra <= p.cap) continue;
    SpecState1 h;
    TRY1(read_state(s, p, h));
    TRY1(check_err(s));
    const int n = h.np[h.cur];
    p.np_bound = n;
    if (n + extra <= p.cap) continue;
    const long long want = std::max<long long>(n + extra, (long long)(1.25 * n) + 1024 + extra);
    if (want > (1LL << 30)) return fail1(ZC_EOVERFLOW, "1-D particle buffer above 2^30 particles");
    const int cap = (int)want;
    Parts nb[2];
    for (int b = 0; b < 2; ++b) TRY1(alloc_parts(nb[b], cap));
    TRY1(copy_parts(p.buf[h.cur], nb[0], n, s->st));
    h.np[0] = n;
    h.np[1] = 0;
    h.cur = 0;
    CK1(cudaMemcpyAsync(p.d_st, &h, sizeof(SpecState1), cudaMemcpyHostToDevice, s->st));
    CK1(cudaStreamSynchronize(s->st));
    free_parts(p.buf[0]);
    free_parts(p.buf[1]);
    p.buf[0] = nb[0];
    p.buf[1] = nb[1];
    p.cap = cap;
    drop_graph(s);
  }
  return ZC_OK;
}

// start of a profiled launch of `kind`: returns the slot of its event pair
// (-1 when profiling is off)
int prof_begin(zc1_sim *s, int kind) {
  if (!s->profile) return -1;
  const size_t slot = s->prof_used;
  if (2 * slot + 2 > s->prof_ev.size()) {
    cudaEvent_t a = nullptr, b = nullptr;
    if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) {
      if (a) cudaEventDestroy(a);
      return -1;
    }
    s->prof_ev.push_back(a);
    s->prof_ev.push_back(b);
    s->prof_kind.push_back(kind);
  }
  s->prof_kind[slot] = kind;
  // inside a capture the record becomes a graph node that records the event
  // each time the graph runs
  if (s->capturing)
    cudaEventRecordWithFlags(s->prof_ev[2 * slot], s->st, cudaEventRecordExternal);
  else
    cudaEventRecord(s->prof_ev[2 * slot], s->st);
  s->prof_used = slot + 1;
  return (int)slot;
}

void prof_end(zc1_sim *s, int slot) {
  if (slot < 0) return;
  if (s->capturing)
    cudaEventRecordWithFlags(s->prof_ev[2 * (size_t)slot + 1], s->st, cudaEventRecordExternal);
  else
    cudaEventRecord(s->prof_ev[2 * (size_t)slot + 1], s->st);
}

// adds the launches recorded in slots [from, to) to the per-kind sums (after
// a stream sync)
void prof_add(zc1_sim *s, size_t from, size_t to) {
  for (size_t i = from; i < to; ++i) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, s->prof_ev[2 * i], s->prof_ev[2 * i + 1]) == cudaSuccess) {
      s->prof_ms[s->prof_kind[i]] += ms;
      s->prof_n[s->prof_kind[i]] += 1;
    }
  }
}

// the eager launches recorded since the last collection (the profiling
// graph keeps the first prof_graph_slots slots)
void prof_collect(zc1_sim *s) {
  if (s->prof_used > s->prof_graph_slots) prof_add(s, s->prof_graph_slots, s->prof_used);
  s->prof_used = s->prof_graph_slots;
}

// enqueues the cell sort of species p (3 kernels); returns the kernel count
int enqueue_sort(zc1_sim *s, Species1 &p) {
  const int pf = prof_begin(s, ZC1_K_SORT);
  cudaMemsetAsync(s->d_cnt, 0, sizeof(int) * s->nx, s->st);
  k1_cell_count<<<sort_blocks(s), 256, 0, s->st>>>(p.buf[0], p.buf[1], p.d_st, s->d_cnt);
  k1_cell_scan<<<1, 1024, 0, s->st>>>(s->d_cnt, s->nx, p.d_st);
  k1_cell_scatter<<<sort_blocks(s), 256, 0, s->st>>>(p.buf[0], p.buf[1], p.d_st, s->d_cnt);
  prof_end(s, pf);
  return 3;
}

Push1 push_const(const zc1_sim *s, const Species1 &p) {
  Push1 C;
  C.tem = (float)(0.5 * s->dt / p.m_q);
  C.dt_dx = s->dt / s->dx;
  C.qnx = p.q * s->dx / s->dt;
  C.q = p.q;
  C.dt = s->dt;
  C.dx = s->dx;
  C.nx = s->nx;
  C.mw = s->mw;
  C.open = (s->mw || s->part_open) ? 1 : 0;
  C.cap = p.cap;
  C.jstride = 3 * (s->nx + GC0 + GC1);
  return C;
}

Fields1 field_const(const zc1_sim *s) {
  Fields1 M;
  M.nx = s->nx;
  M.dt = s->dt;
  M.dx = s->dx;
  M.bc = s->field_bc;
  M.cur_periodic = s->current_periodic;
  M.mw = s->mw;
  M.S = s->smooth;
  return M;
}

// enqueues one step (sim_iter): the push of every species (each followed by
// its cell sort when `sort`), then the fields kernel; nothing is decided on
// the host, so the same calls serve eager steps and graph capture.  Returns
// the kernel count.
int enqueue_step(zc1_sim *s, bool sort) {
  int k = 0;
  for (auto &p : s->sp) {
    const Push1 C = push_const(s, p);
    const int pf = prof_begin(s, ZC1_K_PUSH);
    k1_push<<<push_blocks(s, p.cap), kPushThreads, 0, s->st>>>(p.buf[0], p.buf[1], p.d_st, s->E, s->B, s->Jdep, C,
                                                            p.inj, s->d_err);
    prof_end(s, pf);
    k += 1;
    if (sort) k += enqueue_sort(s, p);
  }
  const Fields1 M = field_const(s);
  const int pf = prof_begin(s, ZC1_K_FIELDS);
  if (s->fields_smem)
    k1_fields<true><<<1, 1024, s->fields_smem, s->st>>>(s->E, s->B, s->Jdep, s->Jout, s->mur, s->d_fs, M);
  else
    k1_fields<false><<<1, 1024, 0, s->st>>>(s->E, s->B, s->Jdep, s->Jout, s->mur, s->d_fs, M);
  prof_end(s, pf);
  return k + 1;
}

// the host's mirror of one step's counters (the device takes the same
// decisions from the same float arithmetic)
void advance_mirror(zc1_sim *s) {
  for (auto &p : s->sp) {
    const int shift = (s->mw && ((float)(p.iter + 1) * s->dt) > (s->dx * (float)(p.n_move + 1))) ? 1 : 0;
    p.iter += 1;
    p.n_move += shift;
    if (shift && p.inj.type != 1) p.np_bound += p.inj.ppc;
  }
  s->iter += 1;
  if (s->mw && ((float)s->iter * s->dt) > (s->dx * (float)(s->n_move + 1))) s->n_move += 1;
}

// sort after this step's push: spec->iter (after the advance) a multiple of n_sort
bool sorts_next(const zc1_sim *s, const Species1 &p) {
  return s->sort_every > 0 && (p.iter + 1) % s->sort_every == 0;
}

// one step launched directly (species share their iteration count: they are
// added before the first advance)
zc_status step_eager(zc1_sim *s) {
  TRY1(ensure_cap(s, 1));
  s->launches += enqueue_step(s, !s->sp.empty() && sorts_next(s, s->sp[0]));
  CK1(cudaGetLastError());
  advance_mirror(s);
  return ZC_OK;
}

// a block of sort_every steps ending with the sort, as one graph
zc_status run_block(zc1_sim *s) {
  const int nb = s->sort_every;
  TRY1(ensure_cap(s, nb));
  cudaGraphExec_t &exec = s->profile ? s->block_prof : s->block;
  int &kernels = s->profile ? s->block_prof_kernels : s->block_kernels;
  if (!exec) {
    if (s->profile) {
      CK1(cudaStreamSynchronize(s->st));
      prof_collect(s);
      s->prof_graph_slots = 0;
      s->prof_used = 0;
    }
    cudaGraph_t g = nullptr;
    CK1(cudaStreamBeginCapture(s->st, cudaStreamCaptureModeThreadLocal));
    s->capturing = 1;
    int k = 0;
    for (int i = 0; i < nb; ++i) k += enqueue_step(s, i == nb - 1);
    s->capturing = 0;
    const cudaError_t e = cudaStreamEndCapture(s->st, &g);
    if (e != cudaSuccess) return fail1f(ZC_ECUDA, "1-D step capture: %s", cudaGetErrorString(e));
    const cudaError_t ei = cudaGraphInstantiate(&exec, g, 0);
    cudaGraphDestroy(g);
    if (ei != cudaSuccess) {
      exec = nullptr;
      return fail1f(ZC_ECUDA, "1-D step graph: %s", cudaGetErrorString(ei));
    }
    kernels = k;
    if (s->profile) s->prof_graph_slots = s->prof_used;
  }
  CK1(cudaGraphLaunch(exec, s->st));
  s->launches += kernels;
  if (s->profile) {
    // the graph records the same events at every replay: read them now
    CK1(cudaStreamSynchronize(s->st));
    prof_add(s, 0, s->prof_graph_slots);
  }
  for (int i = 0; i < nb; ++i) advance_mirror(s);
  return ZC_OK;
}

// Up to `most` steps in one launch (k1_run), to the next cell sort at the
// latest; *done: how many.  None when kernels are timed one by one, there are
// no species or too many, or the grids and every CTA's share of the particles
// do not fit its shared memory (then the two kernels a step, in graphs).
//
// The CTAs: one a multiprocessor when one caller waits for the steps.  One who
// does not wait may have other simulations' steps beside these, and launches
// that fill the GPU would run one after another: a quarter of the
// multiprocessors then (64 runs of the 1000-cell deck side by side: 21.7 G
// particles/s against 8.3 with the full grid and 12.9 with the two kernels; one
// run alone takes 15.2 us a step against 11.0 and 22).  Callers that wait in
// several threads share the GPU likewise, half each or a quarter (that deck
// with 64000 particles, us a step of one run with 1, 2, 4, 8, 32 threads: 11.9
// 7.0 4.3 3.7 3.7, with the full grid 11.9 10.4 9.6 9.2 8.8, with the two
// kernels 22 12.6 7.6 5.9 5.8).  A single step that nobody waits for is left to
// the two kernels: 25.0 us against 26.9.
zc_status run_steps(zc1_sim *s, int most, bool waits, int *done) {
  *done = 0;
  if (!s->run_smem || s->profile || s->sp.empty() || (int)s->sp.size() > kRunSpecies) return ZC_OK;
  const int to_sort = s->sort_every - s->sp[0].iter % s->sort_every;
  const int n = std::min(most, to_sort);
  if (n == 1 && !waits) return ZC_OK;
  TRY1(ensure_cap(s, n));
  long long np = 1;
  for (auto &p : s->sp) np = std::max(np, p.np_bound);
  // one CTA a multiprocessor, at least a warp of particles each (a
  // simulation's own cap counts CTAs of kPushThreads)
  const int sharers = waits ? std::min(4, std::max(1, g_waiting[s->device & 63].load())) : 4;
  const int room = std::max(1, s->sms / sharers);
  const int most_ctas =
      s->push_ctas > 0 ? std::max(1, std::min(s->sms, s->push_ctas * kPushThreads / kRunThreads)) : room;
  const int grid = (int)std::max<long long>(1, std::min<long long>(most_ctas, np / 256));
  Run1 R{};
  R.nsp = (int)s->sp.size();
  R.steps = n;
  R.phase = s->run_phase;
  R.bar0 = s->bar_count;
  R.bar = s->run_bar;
  R.Jrun = s->Jrun;
  R.E = s->E;
  R.B = s->B;
  R.Jout = s->Jout;
  R.mur = s->mur;
  R.fs = s->d_fs;
  R.err = s->d_err;
  R.M = field_const(s);
  size_t smem = 4 * sizeof(float) * grid_stride1(s->nx);
  for (int k = 0; k < R.nsp; ++k) {
    Species1 &p = s->sp[k];
    const long long share = (p.np_bound + grid - 1) / grid;
    // the columns of n window moves go round the CTAs
    const long long cols = (s->mw && p.inj.type != 1) ? (long long)((n + grid - 1) / grid) * p.inj.ppc : 0;
    const long long slots = (share + cols + kRunThreads - 1) / kRunThreads * kRunThreads;
    smem += 5 * sizeof(float) * (size_t)slots;
    if (smem > s->run_smem) return ZC_OK;
    R.sp[k] = RunSpecies1{p.buf[0], p.buf[1], p.d_st, p.d_lat, (int)slots, push_const(s, p), p.inj};
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kRunThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s->st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  CK1(cudaLaunchKernelEx(&cfg, k1_run, R));
  s->bar_count += (unsigned)n * (unsigned)grid;
  s->run_phase = (s->run_phase + n) % 3;
  s->launches += 1;
  if (n == to_sort)
    for (auto &p : s->sp) s->launches += enqueue_sort(s, p);
  CK1(cudaGetLastError());
  for (int i = 0; i < n; ++i) advance_mirror(s);
  *done = n;
  return ZC_OK;
}

zc_status enqueue_steps(zc1_sim *s, int nsteps, bool waits) {
  if (!s || nsteps < 0) return fail1(ZC_EINVAL, "invalid argument");
  Guard1 g(s->device);
  if (!s->timing) {
    CK1(cudaEventRecord(s->ev0, s->st));
    s->timing = 1;
  }
  int k = 0;
  while (k < nsteps) {
    int n = 0;
    TRY1(run_steps(s, nsteps - k, waits, &n));
    k += n;
    if (n) continue;
    const bool aligned = !s->sp.empty() && s->sort_every > 0 && s->sp[0].iter % s->sort_every == 0;
    if (aligned && nsteps - k >= s->sort_every) {
      TRY1(run_block(s));
      k += s->sort_every;
    } else {
      TRY1(step_eager(s));
      k += 1;
    }
    if (s->profile && s->prof_used >= s->prof_graph_slots + 4096) {
      CK1(cudaStreamSynchronize(s->st));
      prof_collect(s);
    }
  }
  return ZC_OK;
}

}  // namespace

extern "C" {

zc_status zc1_create(const zc1_desc *d, zc1_sim **out) {
  if (!d || !out) return fail1(ZC_EINVAL, "null argument");
  *out = nullptr;
  if (d->nx < 4) return fail1(ZC_EINVAL, "1-D grid needs at least 4 cells");
  if (!(d->box > 0) || !(d->dt > 0)) return fail1(ZC_EINVAL, "box and dt must be positive");
  const float dx = d->box / d->nx;
  if (d->dt >= dx) return fail1f(ZC_EINVAL, "Invalid timestep, courant condition violation, dtmax = %f", dx);
  zc1_sim *s = new (std::nothrow) zc1_sim;
  if (!s) return fail1(ZC_ENOMEM, "out of host memory");
  s->nx = d->nx;
  s->box = d->box;
  s->dx = dx;
  s->dt = d->dt;
  s->device = d->device;
  s->mw = d->moving_window ? 1 : 0;
  s->field_bc = s->mw ? 0 : (d->open_fields ? 2 : 1);
  s->current_periodic = s->mw ? 0 : 1;
  s->part_open = d->open_particles ? 1 : 0;
  s->sort_every = d->sort_every > 0 ? d->sort_every : 16;
  s->push_ctas = d->push_ctas > 0 ? d->push_ctas : 0;
  Guard1 g(s->device);
  const size_t gbytes = sizeof(float) * 3 * (s->nx + GC0 + GC1);
  const size_t rbytes = sizeof(float) * 3 * kRunCopies * grid_stride1(s->nx);
  cudaError_t e = cudaStreamCreateWithFlags(&s->st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&s->E, gbytes);
  if (e == cudaSuccess) e = cudaMalloc(&s->B, gbytes);
  if (e == cudaSuccess) e = cudaMalloc(&s->Jdep, gbytes * kJCopies);
  if (e == cudaSuccess) e = cudaMalloc(&s->Jout, gbytes);
  if (e == cudaSuccess) e = cudaMalloc(&s->Jrun, rbytes);
  if (e == cudaSuccess) e = cudaMemset(s->Jrun, 0, rbytes);
  if (e == cudaSuccess) e = cudaMalloc(&s->run_bar, sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMemset(s->run_bar, 0, sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMalloc(&s->mur, sizeof(float) * 12);
  if (e == cudaSuccess) e = cudaMalloc(&s->d_fs, sizeof(FieldState1));
  if (e == cudaSuccess) e = cudaMalloc(&s->d_err, sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&s->d_cnt, sizeof(int) * s->nx);
  if (e == cudaSuccess) e = cudaMalloc(&s->d_emf, sizeof(double) * 6);
  if (e == cudaSuccess) e = cudaEventCreate(&s->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&s->ev1);
  if (e == cudaSuccess) e = cudaMemset(s->E, 0, gbytes);
  if (e == cudaSuccess) e = cudaMemset(s->B, 0, gbytes);
  if (e == cudaSuccess) e = cudaMemset(s->Jdep, 0, gbytes * kJCopies);
  if (e == cudaSuccess) e = cudaMemset(s->Jout, 0, gbytes);
  if (e == cudaSuccess) e = cudaMemset(s->mur, 0, sizeof(float) * 12);
  if (e == cudaSuccess) e = cudaMemset(s->d_fs, 0, sizeof(FieldState1));
  if (e == cudaSuccess) e = cudaMemset(s->d_err, 0, sizeof(int));
  // the fields kernel keeps its four grids in shared memory when they fit.
  // Its dynamic shared-memory ceiling is a property of the kernel for the
  // whole process, so it is raised to the device's maximum (a ceiling, not an
  // allocation) rather than to this grid's size, which could lower it below
  // what another simulation launches with.
  int optin = 0;
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, s->device);
  const size_t smem = 4 * gbytes;
  if (e == cudaSuccess && smem <= (size_t)optin) {
    e = cudaFuncSetAttribute(k1_fields<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    if (e == cudaSuccess) s->fields_smem = smem;
  }
  // k1_run: what its static arrays (under 4 KB) leave
  if (e == cudaSuccess) {
    e = cudaFuncSetAttribute(k1_run, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 4096);
    if (e == cudaSuccess) s->run_smem = optin - 4096;
  }
  if (e != cudaSuccess) {
    zc1_destroy(s);
    return fail1f(ZC_ECUDA, "1-D simulation setup: %s", cudaGetErrorString(e));
  }
  *out = s;
  return ZC_OK;
}

void zc1_destroy(zc1_sim *s) {
  if (!s) return;
  Guard1 g(s->device);
  if (s->st) cudaStreamSynchronize(s->st);
  drop_graph(s);
  for (auto &p : s->sp) {
    free_parts(p.buf[0]);
    free_parts(p.buf[1]);
    cudaFree(p.d_st);
    cudaFree(p.d_lat);
  }
  cudaFree(s->E);
  cudaFree(s->B);
  cudaFree(s->Jdep);
  cudaFree(s->Jrun);
  cudaFree(s->run_bar);
  cudaFree(s->Jout);
  cudaFree(s->mur);
  cudaFree(s->d_fs);
  cudaFree(s->d_err);
  cudaFree(s->d_cnt);
  cudaFree(s->d_emf);
  if (s->ev0) cudaEventDestroy(s->ev0);
  if (s->ev1) cudaEventDestroy(s->ev1);
  for (cudaEvent_t e : s->prof_ev) cudaEventDestroy(e);
  if (s->st) cudaStreamDestroy(s->st);
  delete s;
}

zc_status zc1_add_species(zc1_sim *s, const zc1_species_desc *d, const zc1_part *parts, int np, int *id) {
  if (!s || !d || (np > 0 && !parts) || np < 0) return fail1(ZC_EINVAL, "invalid argument");
  if (s->mw && (d->uth[0] != 0 || d->uth[1] != 0 || d->uth[2] != 0))
    return fail1(ZC_EINVAL, "moving-window injection on the 1-D step supports cold species only");
  if (d->ppc <= 0) return fail1(ZC_EINVAL, "ppc must be positive");
  if (!s->sp.empty() && s->sp[0].iter != 0)
    return fail1(ZC_EINVAL, "species are added to the 1-D step before its first advance");
  for (int i = 0; i < np; ++i)
    if (parts[i].ix < 0 || parts[i].ix >= s->nx) return fail1(ZC_EINVAL, "particle cell outside the grid");
  Guard1 g(s->device);
  Species1 p;
  p.m_q = d->m_q;
  p.q = d->q;
  p.inj.ppc = d->ppc;
  p.inj.type = d->density;
  p.inj.start = d->start;
  p.inj.end = d->end;
  p.inj.dx = s->dx;
  for (int c = 0; c < 3; ++c) p.inj.ufl[c] = d->ufl[c];
  // a window that injects fills up to about nx * ppc particles: room for
  // that from the start keeps the host from reading the count back (a wait
  // on the stream) while the window fills
  long long want = std::max(np + np / 4 + 1024, 1024);
  if (s->mw && d->density != 1) want = std::max(want, (long long)(1.25 * s->nx * d->ppc) + 1024);
  if (want > (1LL << 30)) return fail1(ZC_EOVERFLOW, "1-D particle buffer above 2^30 particles");
  p.cap = (int)want;
  for (int b = 0; b < 2; ++b) TRY1(alloc_parts(p.buf[b], p.cap));
  CK1(cudaMalloc(&p.d_st, sizeof(SpecState1)));
  // reference records (AoS) -> SoA
  std::vector<int> ix(np);
  std::vector<float> x(np), ux(np), uy(np), uz(np);
  for (int i = 0; i < np; ++i) {
    ix[i] = parts[i].ix;
    x[i] = parts[i].x;
    ux[i] = parts[i].ux;
    uy[i] = parts[i].uy;
    uz[i] = parts[i].uz;
  }
  if (np) {
    CK1(cudaMemcpy(p.buf[0].ix, ix.data(), sizeof(int) * np, cudaMemcpyHostToDevice));
    CK1(cudaMemcpy(p.buf[0].x, x.data(), sizeof(float) * np, cudaMemcpyHostToDevice));
    CK1(cudaMemcpy(p.buf[0].ux, ux.data(), sizeof(float) * np, cudaMemcpyHostToDevice));
    CK1(cudaMemcpy(p.buf[0].uy, uy.data(), sizeof(float) * np, cudaMemcpyHostToDevice));
    CK1(cudaMemcpy(p.buf[0].uz, uz.data(), sizeof(float) * np, cudaMemcpyHostToDevice));
  }
  if (s->mw && p.inj.type != 1) {  // only a window that injects reads them
    std::vector<float> lat(p.inj.ppc);
    for (int i = 0; i < p.inj.ppc; ++i) lat[i] = (float)((i + 0.5) / p.inj.ppc);
    CK1(cudaMalloc(&p.d_lat, sizeof(float) * lat.size()));
    CK1(cudaMemcpy(p.d_lat, lat.data(), sizeof(float) * lat.size(), cudaMemcpyHostToDevice));
  }
  SpecState1 h{};
  h.np[0] = np;
  CK1(cudaMemcpy(p.d_st, &h, sizeof(SpecState1), cudaMemcpyHostToDevice));
  p.np_bound = np;
  s->sp.push_back(p);
  drop_graph(s);
  if (id) *id = (int)s->sp.size() - 1;
  // cell order for the warp reduction of the first steps
  s->launches += enqueue_sort(s, s->sp.back());
  CK1(cudaGetLastError());
  CK1(cudaStreamSynchronize(s->st));
  return ZC_OK;
}

zc_status zc1_set_smooth(zc1_sim *s, int type, int level) {
  if (!s) return fail1(ZC_EINVAL, "null simulation handle");
  if (type < 0 || type > 2) return fail1(ZC_EINVAL, "invalid smoothing type");
  if (type != 0 && level <= 0) return fail1(ZC_EINVAL, "Invalid smooth level along x direction");
  if (type != 0 && level > 15) return fail1(ZC_EINVAL, "smoothing level above 15 is not supported");
  Smooth1 S{};
  if (type != 0) {
    for (int i = 0; i < level; ++i) S.sa[S.n] = 0.25f, S.sb[S.n++] = 0.5f;
    if (type == 2) {
      // compensator [a, b, a] for n binomial passes (get_smooth_comp, current.c:244-253)
      const float a = -1;
      const float b = (4.0 + 2.0 * level) / level;
      const float total = 2 * a + b;
      S.sa[S.n] = a / total, S.sb[S.n++] = b / total;
    }
  }
  s->smooth = S;
  drop_graph(s);
  return ZC_OK;
}

zc_status zc1_set_fields(zc1_sim *s, const float *E, const float *B) {
  if (!s) return fail1(ZC_EINVAL, "null simulation handle");
  Guard1 g(s->device);
  const size_t gbytes = sizeof(float) * 3 * (s->nx + GC0 + GC1);
  CK1(cudaStreamSynchronize(s->st));
  if (E) CK1(cudaMemcpy(s->E, E, gbytes, cudaMemcpyHostToDevice));
  if (B) CK1(cudaMemcpy(s->B, B, gbytes, cudaMemcpyHostToDevice));
  return ZC_OK;
}

zc_status zc1_add_laser(zc1_sim *s, const zc_laser *in) {
  if (!s || !in) return fail1(ZC_EINVAL, "null argument");
  zc_laser L = *in;
  // parameter checks, em1d/emf.c:193-219
  if (L.fwhm != 0) {
    if (L.fwhm <= 0) return fail1(ZC_EINVAL, "Invalid laser FWHM, must be > 0");
    L.rise = L.fwhm;
    L.fall = L.fwhm;
    L.flat = 0.;
  }
  if (L.rise <= 0) return fail1(ZC_EINVAL, "Invalid laser RISE, must be > 0");
  if (L.flat < 0) return fail1(ZC_EINVAL, "Invalid laser FLAT, must be >= 0");
  if (L.fall <= 0) return fail1(ZC_EINVAL, "Invalid laser FALL, must be > 0");
  Guard1 g(s->device);
  zc::LaserConst c{};
  c.type = 0;
  c.start = L.start;
  c.rise = L.rise;
  c.flat = L.flat;
  c.fall = L.fall;
  c.a0 = L.a0;
  c.omega0 = L.omega0;
  c.polarization = L.polarization;
  c.dx = s->dx;
  k1_laser<<<1, 1024, 0, s->st>>>(s->E, s->B, s->nx, c, s->field_bc == 1 ? 1 : 0);
  CK1(cudaGetLastError());
  CK1(cudaStreamSynchronize(s->st));
  return ZC_OK;
}

zc_status zc1_get_fields(zc1_sim *s, float *E, float *B) {
  if (!s) return fail1(ZC_EINVAL, "null simulation handle");
  Guard1 g(s->device);
  const size_t gbytes = sizeof(float) * 3 * (s->nx + GC0 + GC1);
  CK1(cudaStreamSynchronize(s->st));
  if (E) CK1(cudaMemcpy(E, s->E, gbytes, cudaMemcpyDeviceToHost));
  if (B) CK1(cudaMemcpy(B, s->B, gbytes, cudaMemcpyDeviceToHost));
  return ZC_OK;
}

zc_status zc1_get_current(zc1_sim *s, float *J) {
  if (!s || !J) return fail1(ZC_EINVAL, "null argument");
  Guard1 g(s->device);
  CK1(cudaStreamSynchronize(s->st));
  CK1(cudaMemcpy(J, s->Jout, sizeof(float) * 3 * (s->nx + GC0 + GC1), cudaMemcpyDeviceToHost));
  return ZC_OK;
}

zc_status zc1_step_async(zc1_sim *s, int nsteps) { return enqueue_steps(s, nsteps, false); }

zc_status zc1_step(zc1_sim *s, int nsteps) {
  if (!s) return fail1(ZC_EINVAL, "null simulation handle");
  Waiting here(s->device);
  TRY1(enqueue_steps(s, nsteps, true));
  return zc1_synchronize(s);
}

zc_status zc1_set_profile(zc1_sim *s, int on) {
  if (!s) return fail1(ZC_EINVAL, "null simulation handle");
  s->profile = on ? 1 : 0;
  for (int k = 0; k < ZC1_NKIND; ++k) {
    s->prof_ms[k] = 0.0;
    s->prof_n[k] = 0;
  }
  return ZC_OK;
}

zc_status zc1_get_profile(zc1_sim *s, double ms[ZC1_NKIND], long long launches[ZC1_NKIND]) {
  if (!s) return fail1(ZC_EINVAL, "null simulation handle");
  for (int k = 0; k < ZC1_NKIND; ++k) {
    if (ms) ms[k] = s->prof_ms[k];
    if (launches) launches[k] = s->prof_n[k];
  }
  return ZC_OK;
}

zc_status zc1_get_launches(zc1_sim *s, long long *n) {
  if (!s || !n) return fail1(ZC_EINVAL, "null argument");
  *n = s->launches;
  return ZC_OK;
}

zc_status zc1_last_step_ms(zc1_sim *s, float *ms) {
  if (!s || !ms) return fail1(ZC_EINVAL, "null argument");
  *ms = s->last_ms;
  return ZC_OK;
}

zc_status zc1_energy(zc1_sim *s, double emf[6], double *kin) {
  if (!s) return fail1(ZC_EINVAL, "null simulation handle");
  Guard1 g(s->device);
  if (emf) {
    k1_emf_energy<<<6, 1024, 0, s->st>>>(s->E, s->B, s->nx, s->dx, s->d_emf);
    CK1(cudaGetLastError());
    CK1(cudaMemcpyAsync(emf, s->d_emf, sizeof(double) * 6, cudaMemcpyDeviceToHost, s->st));
  }
  std::vector<SpecState1> h(s->sp.size());
  for (size_t i = 0; i < s->sp.size(); ++i)
    CK1(cudaMemcpyAsync(&h[i], s->sp[i].d_st, sizeof(SpecState1), cudaMemcpyDeviceToHost, s->st));
  CK1(cudaStreamSynchronize(s->st));
  if (kin)
    for (size_t i = 0; i < s->sp.size(); ++i) {
      // spec->energy = q m_q sum dx (particles.c:1038)
      const Species1 &p = s->sp[i];
      kin[i] = (double)(p.q * p.m_q) * h[i].ekin * (double)s->dx;
    }
  return ZC_OK;
}

zc_status zc1_species_count(zc1_sim *s, int k, int *np) {
  if (!s || !np || k < 0 || k >= (int)s->sp.size()) return fail1(ZC_EINVAL, "invalid argument");
  Guard1 g(s->device);
  SpecState1 h;
  TRY1(read_state(s, s->sp[k], h));
  *np = h.np[h.cur];
  s->sp[k].np_bound = *np;
  return ZC_OK;
}

zc_status zc1_get_particles(zc1_sim *s, int k, zc1_part *out, int cap, int *np) {
  if (!s || !np || k < 0 || k >= (int)s->sp.size()) return fail1(ZC_EINVAL, "invalid argument");
  Guard1 g(s->device);
  Species1 &p = s->sp[k];
  SpecState1 h;
  TRY1(read_state(s, p, h));
  const int n = h.np[h.cur];
  const Parts &b = p.buf[h.cur];
  *np = n;
  if (n > cap || (n > 0 && !out)) return fail1(ZC_EINVAL, "output buffer too small");
  std::vector<int> ix(n);
  std::vector<float> x(n), ux(n), uy(n), uz(n);
  if (n) {
    CK1(cudaMemcpy(ix.data(), b.ix, sizeof(int) * n, cudaMemcpyDeviceToHost));
    CK1(cudaMemcpy(x.data(), b.x, sizeof(float) * n, cudaMemcpyDeviceToHost));
    CK1(cudaMemcpy(ux.data(), b.ux, sizeof(float) * n, cudaMemcpyDeviceToHost));
    CK1(cudaMemcpy(uy.data(), b.uy, sizeof(float) * n, cudaMemcpyDeviceToHost));
    CK1(cudaMemcpy(uz.data(), b.uz, sizeof(float) * n, cudaMemcpyDeviceToHost));
  }
  for (int i = 0; i < n; ++i) out[i] = zc1_part{ix[i], x[i], ux[i], uy[i], uz[i]};
  return ZC_OK;
}

zc_status zc1_get_info(zc1_sim *s, int *iter, int *n_move) {
  if (!s) return fail1(ZC_EINVAL, "null simulation handle");
  if (iter) *iter = s->iter;
  if (n_move) *n_move = s->n_move;
  return ZC_OK;
}

zc_status zc1_synchronize(zc1_sim *s) {
  if (!s) return fail1(ZC_EINVAL, "null simulation handle");
  Guard1 g(s->device);
  if (s->timing) {
    CK1(cudaEventRecord(s->ev1, s->st));
    CK1(cudaEventSynchronize(s->ev1));
    cudaEventElapsedTime(&s->last_ms, s->ev0, s->ev1);
    s->timing = 0;
  }
  CK1(cudaStreamSynchronize(s->st));
  prof_collect(s);
  return check_err(s);
}

zc_status zc1_species_pushed(zc1_sim *s, int k, long long *pushed) {
  if (!s || !pushed || k < 0 || k >= (int)s->sp.size()) return fail1(ZC_EINVAL, "invalid argument");
  Guard1 g(s->device);
  SpecState1 h;
  TRY1(read_state(s, s->sp[k], h));
  *pushed = h.pushed;
  return ZC_OK;
}

}  // extern "C"
