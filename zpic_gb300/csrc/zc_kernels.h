// zc_kernels.h -- launch interface between the host runtime (zc_api.cu) and
// the kernels (zc_particles.cu, zc_fields.cu).
#pragma once

#include <algorithm>

#include "zc_internal.cuh"

namespace zc {

struct PushConst {
  float tem, dt_dx, dt_dy, qnx, qny, q;   // particles.c:1111-1117
  int nx, ny, ntx, nty;
  int shift;                              // moving-window shift applied this step (0/1)
  int mw;                                 // absorbing boundaries along x
  // tile current as integers (see jsplit): a contribution v counts as
  // rint(v js) = h 2^2L + m 2^L + l; js_invl = 2^-L, js_twol = 2^L,
  // js_inv2l = 2^-2L, js_two2l = 2^2L; deterministic global
  // sums in units of 2^-40 take each integer times js_det (2^40 / js)
  float js, js_invl, js_twol, js_inv2l, js_two2l;
  int js_l;
  int js_run;                             // |v| js < 2^43: a lane's sums of two parts hold it (RunSums)
  long long js_det;
};

struct TileSet {
  const int *off, *cap;
  int *np;
  int ntiles;
};

struct Outbox {                           // particles leaving a tile, per tile `cap` slots
  Particles p;
  int *dst, *cnt;
  int cap;
};

struct Spill {                            // particles without room in a tile
  Particles p;
  int *cnt;
  int cap;
};

struct LayoutConst {
  int TX, TY, ntx, nty, nx, ny;
};

// Deterministic mode: the current is accumulated as 64-bit fixed point,
// every contribution rounded once to a multiple of 2^-40.  Integer sums are
// exact, so the result does not depend on the order of the additions (warp
// order, atomics, tiles, spill list): runs are bit-reproducible.  Range:
// |J| < 2^23 per cell and component.  Kinetic-energy terms are split into a
// multiple of 2^-30 and a remainder counted in units of 2^-62, each summed
// as a 64-bit integer (range 2^33, resolution 2^-62).
struct FixedJ {
  unsigned long long *p;  // 3 planes laid out as the float J planes
  int pitch;
  size_t plane;
  float *f;               // the float J planes (the push's direct deposits)
};
constexpr double kJFixScale = 1099511627776.0;         // 2^40
constexpr double kEFixHi = 1073741824.0;                 // 2^30
constexpr double kEFixLo = 4611686018427387904.0;        // 2^62

// a float kinetic-energy term as two integers: hi = rint(v 2^30) and lo =
// rint((v - hi 2^-30) 2^62), without double arithmetic: t = v 2^30 is exact,
// so are its nearest integer hf and the remainder t - hf (|.| <= 1/2), and
// the remainder times 2^32 is lo (exact for v >= 2^-39, rounded below)
__device__ __forceinline__ void efix_split(float v, long long &hi, long long &lo) {
  const float t = __fmul_rn(v, 1073741824.0f);  // 2^30
  const float hf = rintf(t);
  hi = __float2ll_rn(hf);
  lo = __float2ll_rn(__fmul_rn(__fsub_rn(t, hf), 4294967296.0f));  // 2^32
}
// Sums of such pairs, exact: a counts 2^2, c 2^-30, d 2^-62.  What value() makes
// of them depends on the sum alone, not on how it was put together.
struct EfixSum {
  long long a = 0, c = 0, d = 0;
  __device__ __forceinline__ void add(long long hi, long long lo) {
    a += hi >> 32;
    c += (hi & 0xffffffffLL) + (lo >> 32);
    d += lo & 0xffffffffLL;
  }
  __device__ __forceinline__ double value() const {
    const long long c1 = c + (d >> 32);
    return (double)(a + (c1 >> 32)) * 4.0 +
           ((double)(c1 & 0xffffffffLL) * (1.0 / kEFixHi) + (double)(d & 0xffffffffLL) * (1.0 / kEFixLo));
  }
};

// one species' push
struct PushSpecies {
  Particles pin, pout;
  TileSet T;
  Outbox Oin, O;                          // pending incoming (previous step), leavers (this step)
  Spill Sin, S;                           // spilled particles: to push, and those of this step
  double *ekin;                           // kinetic energy of every tile part
  double *ekin_spill;                     // and of every block of the spill push
  long long *ekin_words;                  // deterministic mode: every tile's two fixed-point words instead,
  unsigned long long *ekin_fix;           // and the spill push's
  PushConst C;
};

// all species of a small grid in one launch: tiles by clusters of `parts`
// CTAs, then kSpillParts blocks for the spilled particles of each species
constexpr int kMaxTogether = 8, kMaxParts = 8, kSpillParts = 8;
constexpr int kPushWarps = 4;             // warps of a push CTA (float builds)
// CTAs of that launch that a multiprocessor holds: 4 of the float builds (up to
// 128 registers, 128 threads); of the deterministic ones 3 of 256 threads (80
// registers), or 2 with the 91 KB of a 32x32 tile's current and fields, and 6
// of 128 threads (tiles of less than 256 cells)
__host__ __device__ constexpr int push_all_ctas(int TX, int TY, bool det) {
  return !det ? 4 : (TX * TY >= 1024 ? 2 : (TX * TY >= 256 ? 3 : 6));
}
struct PushAll {
  int nsp, ntiles, parts;
  PushSpecies sp[kMaxTogether];
};

struct PushLaunch {
  const CUtensorMap *tm_eb;
  const PushSpecies *one;                 // one species (or null),
  const PushAll *all;                     // or all of them
  const float *EB;                        // the fields the particles see (spill push)
  Grid G;
  int *err;
  int ntiles, TX, TY;
  int fast;                               // 1: FMA build of the push kernels
  int det;                                // 1: fixed-point currents into fj
  FixedJ fj;
};

#ifdef __CUDACC__
// appends a particle to a spill list; flags the host (re-layout due) and
// records an overflow when the list is full
__device__ __forceinline__ void spill_particle(const Spill &S, int *errbits, int ix, int iy, float x, float y,
                                               float ux, float uy, float uz) {
  const int q = atomicAdd(S.cnt, 1);
  *errbits |= ERR_SPILLED;
  if (q < S.cap) store_particle(S.p, q, ix, iy, x, y, ux, uy, uz);
  else *errbits |= ERR_OVERFLOW;
}

__device__ __forceinline__ void spill_particle(const Spill &S, int *errbits, const PRec &r) {
  spill_particle(S, errbits, r.ix, r.iy, r.x, r.y, r.ux, r.uy, r.uz);
}
#endif

// columns of a tile's staged E/B box: the tile, one column before it and two
// after, up to a multiple of 4 and to a pitch that suits the gather.  A warp
// reads the nodes of some 16 cells of a row, in two rows.  The fast builds
// read 8-byte pairs, half a warp (8 cells, 9 nodes) at a time: with a pitch
// of 8 modulo 16 pairs the two rows lie 16 banks apart.  The exact builds
// read 4-byte values, 17 nodes at a time: 12 modulo 32 keeps most apart.
// (36 columns, the least for a 32-column tile, put the two rows 4 banks
// apart: 18 conflicts a unit of 32 particles at 2048^2, 14 with 40 and pairs.)
__host__ __device__ constexpr int push_box_w(int TX, bool fast) {
  return TX == 32 ? (fast ? 40 : 44) : (TX == 16 ? (fast ? 24 : 20) : 12);
}

// particles
bool tile_supported(int TX, int TY);
cudaError_t launch_push_tiles(const PushLaunch &a, cudaStream_t st);
cudaError_t launch_push_tiles_exact(const PushLaunch &a, cudaStream_t st);
cudaError_t launch_push_tiles_fast(const PushLaunch &a, cudaStream_t st);
cudaError_t launch_push_tiles_exact_det(const PushLaunch &a, cudaStream_t st);
cudaError_t launch_push_tiles_fast_det(const PushLaunch &a, cudaStream_t st);
// spill push of a.one, nblocks blocks (at most kSpillBlocks)
constexpr int kSpillBlocks = 152;
cudaError_t launch_push_spill(const PushLaunch &a, int nblocks, cudaStream_t st);
cudaError_t launch_push_spill_exact(const PushLaunch &a, int nblocks, cudaStream_t st);
cudaError_t launch_push_spill_fast(const PushLaunch &a, int nblocks, cudaStream_t st);
cudaError_t launch_push_spill_exact_det(const PushLaunch &a, int nblocks, cudaStream_t st);
cudaError_t launch_push_spill_fast_det(const PushLaunch &a, int nblocks, cudaStream_t st);
// fixed-point current planes <-> float planes (n values)
cudaError_t launch_fixed_to_float(const unsigned long long *src, float *dst, size_t n, cudaStream_t st);
cudaError_t launch_float_to_fixed(const float *src, unsigned long long *dst, size_t n, cudaStream_t st);
// counting sort of every tile by cell (src -> dst, same offsets): holes
// dropped, np set to the particle count, cell order through tile_slot;
// max_n: the particles a tile stages in shared memory (a tile with more
// takes the rest from global memory; 0: no staging, the sort for runs that
// share the GPU); a timed-out wait on the staging copies sets ERR_TIMEOUT
// in err
cudaError_t launch_cellsort(const Particles &src, const Particles &dst, const int *off, int *np,
                            const LayoutConst &L, int ntiles, int max_n, int *err, cudaStream_t st);
// particles (slots that are not holes) of every tile into cnt
cudaError_t launch_count_valid(const Particles &buf, const int *off, const int *np, int *cnt, int ntiles,
                               cudaStream_t st);
// moves the particles pending in an outbox into their tiles (appended)
cudaError_t launch_settle(const Particles &buf, const TileSet &T, const Outbox &O, const Spill &S, int *err,
                          int ntx, int nty, int mw, cudaStream_t st);
// AoS records (device memory or mapped host memory) -> SoA list; cell_cnt
// (nx * ny counters, or null) receives the particles of every cell
cudaError_t launch_stage_to_list(const void *aos, int n, const Particles &list, int *cell_cnt,
                                 const LayoutConst &L, int *err, cudaStream_t st);
// per tile: cell counts -> first positions of the cells (in place), tile counts
cudaError_t launch_cell_starts(int *cell, int *cnt, const LayoutConst &L, int ntiles, cudaStream_t st);
// list -> tiles in the sorted (lane-run) layout, from the cell starts
cudaError_t launch_scatter_sorted(const Particles &list, int n, const Particles &dst, const int *off,
                                  const int *cnt, int *cell_pos, const LayoutConst &L, cudaStream_t st);
cudaError_t launch_count_list(const Particles &list, const int *n_ptr, int n_cap, int *cnt, const LayoutConst &L,
                              cudaStream_t st);
cudaError_t launch_copy_tiles(const Particles &src, const int *off_old, const int *np_old, const Particles &dst,
                              const int *off_new, int *fill, int ntiles, cudaStream_t st);
cudaError_t launch_scatter_list(const Particles &list, const int *n_ptr, int n_cap, const Particles &dst,
                                const int *off, const int *cap, int *fill, const LayoutConst &L, int *err,
                                cudaStream_t st);
cudaError_t launch_append_list(const Particles &list, int n, const Particles &buf, const TileSet &T,
                               const Spill &S, const LayoutConst &L, int *err, cudaStream_t st);
// a column of cold particles injected after a window move: per row of the
// column, the ppc lattice positions that pass the density test, in the order
// of spec_set_x (em2d/particles.c:159-211, 335-349)
struct ColumnInject {
  int ix, ny, cnt;  // column, rows, particles per cell
  float ux, uy, uz;
  float px[64], py[64];
};
cudaError_t launch_inject_column(const Particles &list, const ColumnInject &C, cudaStream_t st);
cudaError_t launch_gather_aos(const Particles &buf, const int *off, const int *np, const long long *dst_off,
                              int *aos, int ntiles, cudaStream_t st);
cudaError_t launch_list_to_aos(const Particles &list, const int *n_ptr, int n_cap, int *aos, long long d0,
                               cudaStream_t st);
// device-side loading: lattice spacing, per-column inclusion masks (bit a
// of colmask[i]: lattice point a of column i is inside the profile),
// thermal spread and drift, generator key
struct InitConst {
  int ppcx, ppcy;
  float hx, hy;
  float uth[3], ufl[3];
  unsigned seed_lo, seed_hi;
};
cudaError_t launch_init_tiles(const Particles &buf, const int *off, const int *colpts, const unsigned *colmask,
                              const InitConst &I, const LayoutConst &L, int ntiles, cudaStream_t st);
// phase-space density of one species (quantity codes 1 x1, 2 x2, 4 u1,
// 5 u2, 6 u3), added to pha[n1 * n2]
struct PhaConst {
  int q1, q2, n1, n2;
  float x1min, x2min, rdx1, rdx2, dx, dy, q;
};
cudaError_t launch_phasespace(const Particles &buf, const int *off, const int *np, int ntiles, const Particles &spill,
                              const int *spill_cnt, int spill_cap, float *pha, const PhaConst &P,
                              const LayoutConst &L, int per_tile, cudaStream_t st);  // per_tile: particles of a full tile
cudaError_t launch_charge(const Particles &buf, const int *off, const int *np, int ntiles, const Particles &spill,
                          const int *spill_cnt, int spill_cap, float *rho, int nx, int ny, float q, int mw,
                          cudaStream_t st);
// the kinetic-energy sum of one species into *out: n partials of tile parts
// and spill blocks (part); deterministic mode: n tiles' fixed-point words, two
// each (words), and the spill push's two (fix)
struct KinSum {
  const double *part;
  const long long *words;
  const unsigned long long *fix;
  double *out;
  int n;
  float q_mq;
};
#ifdef __CUDACC__
// the sum of K's partials, by a block of NT threads; in thread 0.  Partials in
// a fixed order; words as integers, rounded once, so that neither the tiles nor
// the particles that spilled have a part in the bits.
template <int NT>
__device__ __forceinline__ double kin_total(const KinSum &K) {
  __shared__ double sred[NT / 32];
  __shared__ EfixSum swords[NT / 32];
  if (!K.words) {
    double s = 0;
    for (int i = threadIdx.x; i < K.n; i += NT) s += K.part[i];
    return block_sum_double<NT>(s, sred);
  }
  EfixSum e;
  for (int i = threadIdx.x; i < K.n; i += NT) e.add(K.words[2 * (size_t)i], K.words[2 * (size_t)i + 1]);
  if (threadIdx.x == 0) e.add((long long)K.fix[0], (long long)K.fix[1]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    e.a += __shfl_down_sync(0xffffffffu, e.a, o);
    e.c += __shfl_down_sync(0xffffffffu, e.c, o);
    e.d += __shfl_down_sync(0xffffffffu, e.d, o);
  }
  if ((threadIdx.x & 31) == 0) swords[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < NT / 32; ++w) {
      e.a += swords[w].a;
      e.c += swords[w].c;
      e.d += swords[w].d;
    }
  __syncthreads();
  return e.value();
}
#endif
// one block a species
struct KinSums {
  KinSum k[kMaxTogether];
};
cudaError_t launch_kin_sums(const KinSums &K, int nsp, float dx, float dy, cudaStream_t st);

// fields
struct YeeConst {
  float cxb, cyb;                         // (dt/2)/dx, (dt/2)/dy  (emf.c:507-508)
  float cxe, cye, dt;                     // dt/dx, dt/dy, dt      (emf.c:540-541)
  int mw;                                 // moving window: x guard cells are not periodic
  int shift;                              // the window moves after this step: fields stored one cell left
};

cudaError_t launch_aos_to_planes(const float *aos, float *planes, const Grid &G, int ncomp, cudaStream_t st);
cudaError_t launch_planes_to_aos(const float *planes, float *aos, const Grid &G, int ncomp, cudaStream_t st);
cudaError_t launch_fold(float *J, const Grid &G, int mw, cudaStream_t st);
// all filter passes along one axis in one launch
constexpr int kMaxSmoothPasses = 16;
struct SmoothPasses {
  int n;
  float sa[kMaxSmoothPasses], sb[kMaxSmoothPasses];
};
// every x filter pass, then every y pass, out of place (Jin -> Jout)
cudaError_t launch_smooth(const float *Jin, float *Jout, const Grid &G, const SmoothPasses &PX,
                          const SmoothPasses &PY, int mw, cudaStream_t st);
// epart (or null): per-block field-energy partials of the new fields, 6
// doubles a block, yee_blocks(G) blocks.  jzero (or null): a current buffer
// the kernel clears (3 planes).  gc: the guard cells are written as the
// guard-cell update leaves them (k_emf_gc then not needed; nx, ny >= 3)
// zero: words the kernel clears (spill counts)
struct ZeroWords {
  int n;
  int *p[kMaxTogether];
};
cudaError_t launch_yee(const CUtensorMap *tm_eb, const CUtensorMap *tm_j, float *EBout, const Grid &G,
                       const YeeConst &Y, int *err, double *epart, float *jzero, bool gc, const ZeroWords &zero,
                       cudaStream_t st);
// external fields added to what the particles see: types (0 none, 1 uniform,
// 2 a grid), values per component; out null: none
struct ExtField {
  float *out = nullptr;
  const float *E = nullptr, *B = nullptr;
  int Et = 0, Bt = 0;
  float v0[6] = {};
};
// fold of the raw deposits Jraw, filter into Jout, Yee advance, external
// fields and clearing of the next raw buffer, in one launch (periodic guard
// cells included); tm_j: a box of kFieldBW x kFieldBH x 3 over Jraw
inline bool fields_together(const Grid &G, const SmoothPasses &PX, const SmoothPasses &PY) {
  return G.nx >= 6 && G.ny >= 6 && PX.n <= 4 && PY.n <= 4;  // a 4-cell halo, disjoint folds
}
cudaError_t launch_fields(const CUtensorMap *tm_eb, const CUtensorMap *tm_j, const float *Jraw, float *Jout,
                          float *Jnext, float *EBout, const ExtField &ext, const Grid &G, const YeeConst &Y,
                          const SmoothPasses &PX, const SmoothPasses &PY, int *err, double *epart,
                          const ZeroWords &zero, cudaStream_t st);
int yee_blocks(const Grid &G);
cudaError_t launch_emf_gc(float *EB, const Grid &G, int mw, cudaStream_t st);
cudaError_t launch_ext_add(const float *EB, float *EBp, const float *extE, const float *extB, int Etype, int Btype,
                           float3 E0, float3 B0, const Grid &G, cudaStream_t st);
cudaError_t launch_window_shift(const float *EBin, float *EBout, const Grid &G, cudaStream_t st);
// the kinetic-energy words of up to kEkinRefs species, by value
constexpr int kEkinRefs = 32;
struct EkinRefs {
  const double *p[kEkinRefs];
};
// field energy (emf, 6 values) and the species' kinetic energies (kin) written
// by the device into the given arrays (device or mapped host memory); either
// may be null
cudaError_t launch_energy_direct(const float *EB, const Grid &G, double *partial, int nblocks, float dx, float dy,
                                 const EkinRefs &K, int nsp, double *emf, double *kin, cudaStream_t st);
cudaError_t launch_emf_energy(const float *EB, const Grid &G, double *partial, int nblocks, double *out, float dx,
                              float dy, cudaStream_t st);
// appends one row (6 field-energy components, then each species' kinetic
// energy) at hist[*hist_n] and increments *hist_n, unless cap rows exist.
// EB null: the partials are already there (the Yee kernel's).  The kinetic
// sums ks (device memory) are made here first
cudaError_t launch_energy_history(const float *EB, const Grid &G, double *partial, int nblocks, double *hist,
                                  int *hist_n, int cap, int cols, const KinSum *ks, int nsp, float dx, float dy,
                                  cudaStream_t st);
// dst[k] = *src[k] for k < n (error words of a batch)
cudaError_t launch_gather_words(int *const *src, int n, int *dst, cudaStream_t st);
struct LaserConst {
  int type;
  float start, rise, flat, fall, a0, omega0, polarization, W0, focus, axis;
  float dx, dy;
};
cudaError_t launch_laser(float *EB, const Grid &G, const LaserConst &L, cudaStream_t st);

#ifdef __CUDACC__
// longitudinal envelope of a laser pulse (lon_env, em2d/emf.c:158-186 and
// em1d/emf.c:157-180): sin^2 rise and fall around a flat top, evaluated with
// the double-precision sin on float arguments as the reference does
__device__ inline float laser_env(const LaserConst &L, float z) {
  const double half_pi = 1.57079632679489661923132169163975144;
  if (z > L.start) return 0.0f;
  if (z > L.start - L.rise) {
    float u = z - L.start;
    float e = sin(half_pi * u / L.rise);
    return e * e;
  }
  if (z > L.start - (L.rise + L.flat)) return 1.0f;
  if (z > L.start - (L.rise + L.flat + L.fall)) {
    float u = z - (L.start - L.rise - L.flat - L.fall);
    float e = sin(half_pi * u / L.fall);
    return e * e;
  }
  return 0.0f;
}
#endif

// sets the message returned by zc_last_error() on this thread
void set_error_message(const char *msg);

constexpr int kYeeOX = 32, kYeeOY = 16;   // Yee output tile (buffer cells)
constexpr int kYeeBW = kYeeOX + 8;        // TMA box: 4 columns of halo each side
constexpr int kYeeBH = kYeeOY + 3;
constexpr int kFieldBW = kYeeOX + 12;     // raw current of a tile: 4 cells before, 8 and 5 after
constexpr int kFieldBH = kYeeOY + 9;

}  // namespace zc
