// zc_push_impl.cuh -- particle push + current deposit kernels.
//
// Included twice, inside namespaces zc::exact and zc::fast, by
// zc_push_exact.cu (compiled with --fmad=false and IEEE division / square
// root: every float32 operation rounds as in the reference C, particles
// advanced from the same fields land on the same bits) and zc_push_fast.cu
// (FMA contraction and the hardware's approximate float32 division and
// square root: same algorithm, results within a few float32 ulps per
// operation of the exact build).
//
//   k_push_tiles  one CTA per particle tile (TX x TY cells).  The tile's E/B
//                 with a 1-lower / 2-upper cell halo arrive in shared memory
//                 by one 3-D TMA box; every particle of the tile is pushed
//                 (staggered bilinear gather, relativistic Boris, move) and
//                 its current deposited with the zigzag scheme.  Tiles are
//                 kept sorted by cell, so the lanes of a warp mostly share a
//                 cell: their gathers are broadcasts, and the current of the
//                 segment of a particle that stays in its cell is summed in
//                 the lane's registers (deterministic builds: as integers)
//                 before it is deposited.  The fast and exact builds deposit with
//                 float reductions on the global J planes, which L2 performs
//                 natively; the deterministic builds accumulate a shared
//                 integer J tile (exact, order-independent sums) and add it
//                 to the global fixed-point planes.  Cell-crossing particles
//                 (a few per cent) wait in a per-warp shared-memory queue and
//                 are finished (motion split and deposited, new cell, leaving
//                 or staying) a warp's worth at a time, so that code runs with
//                 (nearly) full warps.  Particles that leave go to the
//                 tile's outbox, from which the destination tile pulls them
//                 at the start of the next step's push.
//   k_push_spill  the same physics for particles that did not fit a tile,
//                 from global memory (normally empty).
//
// Requires zc_internal.cuh and zc_kernels.h to be included first.

// ---------------------------------------------------------------------------
// field / current accessors: shared-memory tile (1-cell lower halo) or the
// global padded planes
// ---------------------------------------------------------------------------
template <int BW, int PL>
struct TileFields {
  const float *s;
  __device__ __forceinline__ float operator()(int c, int i, int j) const {
    return s[c * PL + (j + 1) * BW + (i + 1)];
  }
};
// The tile current is kept as three planes of 32-bit integers: a
// contribution v counts as the integer rint(v js) = h 2^2L + m 2^L + l (js a
// power of two, |m|, |l| <= 2^(L-1)), each part added to its plane with a
// 32-bit integer atomic (float atomic adds on shared memory run as
// compare-and-swap loops, integer ones are single instructions).  The host
// picks L so that no plane can overflow with the most contributions a tile
// can take, and js = 2^40 (the unit of the deterministic mode) unless the
// largest contribution needs a smaller one.  The parts are rounded with the
// 1.5 2^23 shifter (exact for |t| < 2^22) instead of conversion instructions.
constexpr float kShifter = 12582912.0f;  // 1.5 * 2^23
constexpr int kShifterBits = 0x4B400000;

__device__ __forceinline__ void jsplit(float v, const PushConst &C, int &h, int &m, int &l) {
  const float x = __fmul_rn(v, C.js);                  // exact: js is a power of two
  const float th = __fmaf_rn(x, C.js_inv2l, kShifter);  // rint(x 2^-2L) + shifter
  h = __float_as_int(th) - kShifterBits;
  const float r1 = __fmaf_rn(-__fsub_rn(th, kShifter), C.js_two2l, x);  // exact remainder
  const float tm = __fmaf_rn(r1, C.js_invl, kShifter);
  m = __float_as_int(tm) - kShifterBits;
  const float r2 = __fmaf_rn(-__fsub_rn(tm, kShifter), C.js_twol, r1);  // exact remainder
  l = __float_as_int(__fadd_rn(r2, kShifter)) - kShifterBits;
}

// node offsets of the integer J tile, per component: Jx takes columns
// -1..TX, Jy rows -1..TY, Jz both one more (the halo each can receive)
template <int TX, int TY>
struct JTileLayout {
  static constexpr int WX = TX + 2, HX = TY + 3;
  static constexpr int WY = TX + 3, HY = TY + 2;
  static constexpr int WZ = TX + 3, HZ = TY + 3;
  static constexpr int OX = 0, OY = WX * HX, OZ = OY + WY * HY;
  static constexpr int N = OZ + WZ * HZ;  // nodes per plane
  // component, row and column (halo included) of node k
  __device__ __forceinline__ static void where(int k, int &c, int &r, int &col) {
    if (k < OY) {
      c = 0, r = k / WX, col = k % WX;
    } else if (k < OZ) {
      c = 1, r = (k - OY) / WY, col = (k - OY) % WY;
    } else {
      c = 2, r = (k - OZ) / WZ, col = (k - OZ) % WZ;
    }
  }
  __device__ __forceinline__ static int node(int c, int i, int j) {
    return c == 0 ? OX + (j + 1) * WX + (i + 1) : (c == 1 ? OY + (j + 1) * WY + (i + 1) : OZ + (j + 1) * WZ + (i + 1));
  }
};

// fast and exact builds: every deposit goes straight to the global J
// planes as a float reduction, which L2 performs (no compare-and-swap loop);
// g points at the tile's first cell, (i, j) run over -1 .. TX, -1 .. TY
struct TileCurrentGlobal {
  float *g;
  int pitch;
  size_t plane;
  __device__ __forceinline__ void add(int c, int i, int j, float v) const {
    atomicAdd(g + c * plane + (long long)j * pitch + i, v);
  }
};

// the integer a node of the tile holds: h 2^2L + m 2^L + l
__device__ __forceinline__ long long tile_node_sum(const int *p, int n, int k, int L) {
  return (long long)p[k] * (1LL << (2 * L)) + (long long)p[n + k] * (1LL << L) + p[2 * n + k];
}

template <class LAY>
struct TileCurrentSplit {
  int *p;  // planes h, m, l of LAY::N nodes each
  const PushConst *C;
  __device__ __forceinline__ static int column(unsigned cell) { return (int)(cell & (LAY::WX - 3)); }
  __device__ __forceinline__ static int row(unsigned cell) { return (int)((cell >> 16) & (LAY::HY - 3)); }
  __device__ __forceinline__ void add(int c, int i, int j, float v) const {
    int h, m, l;
    jsplit(v, *C, h, m, l);
    addi(c, i, j, h, m, l);
  }
  __device__ __forceinline__ void addi(int c, int i, int j, int h, int m, int l) const {
    const int k = LAY::node(c, i, j);
    atomicAdd(&p[k], h);
    atomicAdd(&p[LAY::N + k], m);
    atomicAdd(&p[2 * LAY::N + k], l);
  }
};

struct GlobalFields {
  const float *g;
  int pitch;
  size_t plane;
  __device__ __forceinline__ float operator()(int c, int i, int j) const {
    return __ldg(&g[c * plane + (size_t)(j + 1) * pitch + (i + 1)]);
  }
};
struct GlobalCurrent {
  float *g;
  int pitch;
  size_t plane;
  __device__ __forceinline__ void add(int c, int i, int j, float v) const {
    atomicAdd(&g[c * plane + (size_t)(j + 1) * pitch + (i + 1)], v);
  }
};

// deterministic mode: every contribution rounded once to the integer
// rint(v js) (as the tile current rounds it) and summed in units of 2^-40
__device__ __forceinline__ long long to_fixed(float v, const PushConst &C) {
  return __float2ll_rn(v * C.js) * C.js_det;
}

struct GlobalCurrentFixed {
  unsigned long long *g;
  int pitch;
  size_t plane;
  const PushConst *C;
  __device__ __forceinline__ void add(int c, int i, int j, float v) const {
    atomicAdd(&g[c * plane + (size_t)(j + 1) * pitch + (i + 1)], (unsigned long long)to_fixed(v, *C));
  }
};

// ---------------------------------------------------------------------------
// per-particle physics (restates em2d/particles.c:773-924, 1029-1226)
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ float lerp2(const F &f, int c, int a, int b, float wa, float wb) {
  return (f(c, a, b) * (1.0f - wa) + f(c, a + 1, b) * wa) * (1.0f - wb) +
         (f(c, a, b + 1) * (1.0f - wa) + f(c, a + 1, b + 1) * wa) * wb;
}

// staggered bilinear interpolation at (x, y) of cell (i, j) of the accessor
// frame (interpolate_fld, particles.c:1029-1071)
template <class F>
__device__ __forceinline__ void gather(const F &fld, int i, int j, float x, float y, float &ex, float &ey, float &ez,
                                       float &bx, float &by, float &bz) {
  const int ih = i + ((x < 0.5f) ? -1 : 0);
  const int jh = j + ((y < 0.5f) ? -1 : 0);
  const float w1h = x + ((x < 0.5f) ? 0.5f : -0.5f);
  const float w2h = y + ((y < 0.5f) ? 0.5f : -0.5f);
  ex = lerp2(fld, 0, ih, j, w1h, y);
  ey = lerp2(fld, 1, i, jh, x, w2h);
  ez = lerp2(fld, 2, i, j, x, y);
  bx = lerp2(fld, 3, i, jh, x, w2h);
  by = lerp2(fld, 4, ih, j, w1h, y);
  bz = lerp2(fld, 5, ih, jh, w1h, w2h);
}

#ifdef ZC_FAST
// Fast builds: Ex and By are interpolated at the same nodes with the same
// weights, and so are Ey and Bx.  The tile keeps each of the two as pairs
// (one 8-byte load instead of two of 4), and all six components are
// interpolated two at a time with packed float pairs: 16 loads and 18 packed
// operations a particle instead of 24 and 36.
template <int BW, int PL>
struct TilePairs {
  const float2 *xb, *yb;  // (Ex, By), (Ey, Bx)
  const float *ez, *bz;
};

__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 lerp2p(float2 a, float2 b, float2 c, float2 d, float2 wx, float2 wy) {
  const float2 lo = __ffma2_rn(wx, sub2(b, a), a), hi = __ffma2_rn(wx, sub2(d, c), c);
  return __ffma2_rn(wy, sub2(hi, lo), lo);
}

template <int BW, int PL>
__device__ __forceinline__ void gather(const TilePairs<BW, PL> &f, int i, int j, float x, float y, float &ex,
                                       float &ey, float &ez, float &bx, float &by, float &bz) {
  const bool lx = x < 0.5f, ly = y < 0.5f;
  const float xh = x + (lx ? 0.5f : -0.5f), yh = y + (ly ? 0.5f : -0.5f);
  const int s = (j + 1) * BW + (i + 1);
  const int sx = s - (lx ? 1 : 0), sy = s - (ly ? BW : 0), sc = sx - (ly ? BW : 0);
  const float2 *a = f.xb + sx, *b = f.yb + sy;
  const float2 r0 = lerp2p(a[0], a[1], a[BW], a[BW + 1], make_float2(xh, xh), make_float2(y, y));
  const float2 r1 = lerp2p(b[0], b[1], b[BW], b[BW + 1], make_float2(x, x), make_float2(yh, yh));
  const float *e = f.ez + s, *g = f.bz + sc;
  const float2 r2 = lerp2p(make_float2(e[0], g[0]), make_float2(e[1], g[1]), make_float2(e[BW], g[BW]),
                           make_float2(e[BW + 1], g[BW + 1]), make_float2(x, xh), make_float2(y, yh));
  ex = r0.x;
  by = r0.y;
  ey = r1.x;
  bx = r1.y;
  ez = r2.x;
  bz = r2.y;
}

// the arguments here are sums of 1 and squares: never denormal
__device__ __forceinline__ float rsqrt_ftz(float v) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float rcp_ftz(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
#endif

struct Seg {
  float x0, x1, y0, y1, dx, dy, qvz;
  int ix, iy;
};

// the 8 current contributions of one straight segment inside one cell
// (particles.c:886-922): Jx at (ix,iy),(ix,iy+1); Jy at (ix,iy),(ix+1,iy);
// Jz at the four corners (ix,iy),(ix+1,iy),(ix,iy+1),(ix+1,iy+1)
struct SegCurrent {
  float v[8];
};

__device__ __forceinline__ SegCurrent segment_current(const Seg &s, float qnx, float qny) {
#ifdef ZC_FAST
  // the same weights, re-associated (fast builds), two at a time: Jx, Jy
  // from the segment's mid-point; with p, m = c + d/2, d - c/2 of the start /
  // end y weights c, d of a row, the Jz corners of that row are
  // q (a p + b m), a, b the start / end x weights, which add up to q (p + m)
  SegCurrent r;
  const float jx = qnx * s.dx, jy = qny * s.dy;
  const float ym = 0.5f * (s.y0 + s.y1), xm = 0.5f * (s.x0 + s.x1);
  const float2 j1 = __fmul2_rn(make_float2(jx, jy), make_float2(ym, xm));
  const float2 j0 = sub2(make_float2(jx, jy), j1);
  const float p1 = s.y0 + 0.5f * s.y1, m1 = s.y1 - 0.5f * s.y0;
  const float2 q = make_float2(s.qvz, s.qvz);
  const float2 qp = __fmul2_rn(q, make_float2(1.5f - p1, p1)), qm = __fmul2_rn(q, make_float2(0.5f - m1, m1));
  const float2 z1 = __ffma2_rn(make_float2(s.x1, s.x1), qm, __fmul2_rn(make_float2(s.x0, s.x0), qp));
  const float2 z0 = sub2(__fadd2_rn(qp, qm), z1);
  r.v[0] = j0.x;
  r.v[1] = j1.x;
  r.v[2] = j0.y;
  r.v[3] = j1.y;
  r.v[4] = z0.x;
  r.v[5] = z1.x;
  r.v[6] = z0.y;
  r.v[7] = z1.y;
  return r;
#else
  const float s0x0 = 1.0f - s.x0, s0x1 = s.x0;
  const float s1x0 = 1.0f - s.x1, s1x1 = s.x1;
  const float s0y0 = 1.0f - s.y0, s0y1 = s.y0;
  const float s1y0 = 1.0f - s.y1, s1y1 = s.y1;
  const float jx = qnx * s.dx;
  const float jy = qny * s.dy;
  const float ay0 = 0.5f * (s0y0 + s1y0), ay1 = 0.5f * (s0y1 + s1y1);
  const float ax0 = 0.5f * (s0x0 + s1x0), ax1 = 0.5f * (s0x1 + s1x1);
  const float q = s.qvz;
  SegCurrent r;
  r.v[0] = jx * ay0;
  r.v[1] = jx * ay1;
  r.v[2] = jy * ax0;
  r.v[3] = jy * ax1;
  r.v[4] = q * (s0x0 * s0y0 + s1x0 * s1y0 + (s0x0 * s1y0 - s1x0 * s0y0) / 2.0f);
  r.v[5] = q * (s0x1 * s0y0 + s1x1 * s1y0 + (s0x1 * s1y0 - s1x1 * s0y0) / 2.0f);
  r.v[6] = q * (s0x0 * s0y1 + s1x0 * s1y1 + (s0x0 * s1y1 - s1x0 * s0y1) / 2.0f);
  r.v[7] = q * (s0x1 * s0y1 + s1x1 * s1y1 + (s0x1 * s1y1 - s1x1 * s0y1) / 2.0f);
  return r;
#endif
}

template <class D>
__device__ __forceinline__ void add_current(const D &dep, int ix, int iy, const SegCurrent &c) {
  dep.add(0, ix, iy, c.v[0]);
  dep.add(0, ix, iy + 1, c.v[1]);
  dep.add(1, ix, iy, c.v[2]);
  dep.add(1, ix + 1, iy, c.v[3]);
  dep.add(2, ix, iy, c.v[4]);
  dep.add(2, ix + 1, iy, c.v[5]);
  dep.add(2, ix, iy + 1, c.v[6]);
  dep.add(2, ix + 1, iy + 1, c.v[7]);
}

// A lane's running sums of the deterministic builds: each contribution counts
// as rint(v js) = h 2^22 + l, |l| <= 2^21, and |h| <= 2^21 where |v| js < 2^43
// (PushConst::js_run); 512 of them fit 32 bits.  Two parts are enough for sums
// that short; the tile's sums take the three of jsplit.
struct RunSums {
  int h[8], l[8];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int q = 0; q < 8; ++q) h[q] = l[q] = 0;
  }
  __device__ __forceinline__ void add(const SegCurrent &cur, float js) {
    constexpr int pa[4] = {0, 1, 4, 5};  // pairs (0, 2), (1, 3), (4, 6), (5, 7), as they were computed
    const float2 sh = make_float2(kShifter, kShifter);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int q = pa[k];
      const float2 x = __fmul2_rn(make_float2(cur.v[q], cur.v[q + 2]), make_float2(js, js));  // exact
      const float2 th = __ffma2_rn(x, make_float2(0x1p-22f, 0x1p-22f), sh);
      const float2 r =  // exact remainder
          __ffma2_rn(__ffma2_rn(th, make_float2(-1.f, -1.f), sh), make_float2(0x1p22f, 0x1p22f), x);
      const float2 tl = __fadd2_rn(r, sh);
      h[q] += __float_as_int(th.x) - kShifterBits;
      h[q + 2] += __float_as_int(th.y) - kShifterBits;
      l[q] += __float_as_int(tl.x) - kShifterBits;
      l[q + 2] += __float_as_int(tl.y) - kShifterBits;
    }
  }
  // to the tile's three planes, as jsplit cuts an integer; the sums start again
  template <class DEP>
  __device__ __forceinline__ void flush(const DEP &dep, unsigned cell) {
    const int i = DEP::column(cell), j = DEP::row(cell), L = dep.C->js_l, s = 22 - L;
    constexpr int c[8] = {0, 0, 1, 1, 2, 2, 2, 2}, di[8] = {0, 0, 0, 1, 0, 1, 0, 1}, dj[8] = {0, 1, 0, 0, 0, 0, 1, 1};
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      // (h 2^22 + l = vh 2^2L + vm 2^L + vl: the low L bits of l, then those of
      // r + h 2^s, which makes r - vm a multiple of 2^min(s, L); no 64-bit shifts)
      const int vl = (int)((unsigned)l[q] << (32 - L)) >> (32 - L), r = (l[q] - vl) >> L;
      const int vm = (int)((((unsigned)h[q] << s) + (unsigned)r) << (32 - L)) >> (32 - L);
      const int vh = L >= s ? (h[q] + ((r - vm) >> s)) >> (L - s) : (h[q] << (s - L)) + ((r - vm) >> L);
      dep.addi(c[q], i + di[q], j + dj[q], vh, vm, vl);
      h[q] = l[q] = 0;
    }
  }
};

// splits segment `a` at the y cell edge: `a` keeps the part before the edge,
// the returned segment holds the rest (particles.c:842-871)
__device__ __forceinline__ Seg split_y(Seg &a, int dj) {
  const int yb = (dj == 1);
  const float f = (a.y1 - yb) / a.dy;
  const float xc = a.x0 + a.dx * (1.0f - f);
  Seg n;
  n.y0 = 1 - yb;
  n.y1 = a.y1 - dj;
  n.dy = a.dy * f;
  n.iy = a.iy + dj;
  n.x0 = xc;
  n.x1 = a.x1;
  n.dx = a.dx * f;
  n.ix = a.ix;
  n.qvz = a.qvz * f;
  a.y1 = yb;
  a.dy *= (1.0f - f);
  a.dx *= (1.0f - f);
  a.x1 = xc;
  a.qvz *= (1.0f - f);
  return n;
}

// Zigzag trajectory split (particles.c:773-879): returns the first segment,
// which always starts in the particle's own cell; the (at most two) further
// segments of a cell-crossing motion are deposited right away.
template <class D>
__device__ __forceinline__ Seg zigzag_first(const D &dep, int ix, int iy, int di, int dj, float x0, float y0,
                                            float dx, float dy, float qnx, float qny, float qvz) {
  Seg a;
  a.x0 = x0;
  a.y0 = y0;
  a.dx = dx;
  a.dy = dy;
  a.x1 = x0 + dx;
  a.y1 = y0 + dy;
  a.qvz = qvz * 0.5f;  // qvz/2.0 in the reference: exact halving either way
  a.ix = ix;
  a.iy = iy;
  if (di != 0) {
    const int xb = (di == 1);
    const float f = (x0 + dx - xb) / dx;
    const float yc = y0 + dy * (1.0f - f);
    Seg b;
    b.x0 = 1 - xb;
    b.x1 = (x0 + dx) - di;
    b.dx = dx * f;
    b.ix = ix + di;
    b.y0 = yc;
    b.y1 = a.y1;
    b.dy = dy * f;
    b.iy = iy;
    b.qvz = a.qvz * f;
    a.x1 = xb;
    a.dx *= (1.0f - f);
    a.dy *= (1.0f - f);
    a.y1 = yc;
    a.qvz *= (1.0f - f);
    if (dj != 0) {
      if (a.y1 < 0.0f || a.y1 >= 1.0f) {
        // the first piece crosses the y edge; the x tail lies past it
        const Seg c = split_y(a, dj);
        b.y0 -= dj;
        b.y1 -= dj;
        b.iy += dj;
        add_current(dep, c.ix, c.iy, segment_current(c, qnx, qny));
      } else {
        const Seg c = split_y(b, dj);
        add_current(dep, c.ix, c.iy, segment_current(c, qnx, qny));
      }
    }
    add_current(dep, b.ix, b.iy, segment_current(b, qnx, qny));
  } else if (dj != 0) {
    const Seg c = split_y(a, dj);
    add_current(dep, c.ix, c.iy, segment_current(c, qnx, qny));
  }
  return a;
}

// displacement (cells) and q v_z of a particle with the new momentum
__device__ __forceinline__ void displacement(float ux, float uy, float uz, float &mx, float &my, float &qvz,
                                             const PushConst &C) {
#ifdef ZC_FAST
  const float rg = rsqrt_ftz(1.0f + ux * ux + uy * uy + uz * uz);
#else
  const float rg = 1.0f / sqrtf(1.0f + ux * ux + uy * uy + uz * uz);
#endif
  mx = C.dt_dx * rg * ux;
  my = C.dt_dy * rg * uy;
  qvz = C.q * uz * rg;
}

// gather + Boris for one particle at cell (i, j) of the accessor frame
// (particles.c:1029-1207); leaves the displacement in (mx, my), returns the
// kinetic-energy term utsq/(gamma+1).  A motion of one cell or more (or NaN)
// is not supported by the deposit: the callers flag it.  A trimmed position
// of exactly 1.0f (x + mx = -tiny, +1 rounds up) is legal, as in the
// reference.
template <class F>
__device__ __forceinline__ float push_particle(const F &fld, int i, int j, float x, float y, float &ux,
                                               float &uy, float &uz, float &mx, float &my, float &qvz,
                                               const PushConst &C) {
  float ex, ey, ez, bx, by, bz;
  gather(fld, i, j, x, y, ex, ey, ez, bx, by, bz);

  const float tem = C.tem;
  ex *= tem;
  ey *= tem;
  ez *= tem;
  float tx = ux + ex, ty = uy + ey, tz = uz + ez;
  const float u2 = tx * tx + ty * ty + tz * tz;
#ifdef ZC_FAST
  const float g2 = 1.0f + u2, ig = rsqrt_ftz(g2);
  const float kin = u2 * rcp_ftz(g2 * ig + 1.0f);
  const float tg = tem * ig;
#else
  const float g = sqrtf(1.0f + u2);
  const float kin = u2 / (g + 1);
  const float tg = tem / g;
#endif
  bx *= tg;
  by *= tg;
  bz *= tg;
#ifdef ZC_FAST
  const float s2 = 2.0f * rcp_ftz(1.0f + bx * bx + by * by + bz * bz);
#else
  const float s2 = 2.0f / (1.0f + bx * bx + by * by + bz * bz);
#endif
  float vx = tx + ty * bz - tz * by;
  float vy = ty + tz * bx - tx * bz;
  float vz = tz + tx * by - ty * bx;
  bx *= s2;
  by *= s2;
  bz *= s2;
  tx += vy * bz - vz * by;
  ty += vz * bx - vx * bz;
  tz += vx * by - vy * bx;
  ux = tx + ex;
  uy = ty + ey;
  uz = tz + ez;

  displacement(ux, uy, uz, mx, my, qvz, C);
  return kin;
}

// new cell after the move, window shift and boundary; false when the
// particle left through an absorbing x boundary (particles.c:1234-1259)
__device__ __forceinline__ bool apply_boundary(int &ix, int &iy, int di, int dj, const PushConst &C) {
  ix += di - C.shift;
  iy += dj;
  iy += ((iy < 0) ? C.ny : 0) - ((iy >= C.ny) ? C.ny : 0);
  if (C.mw) return ix >= 0 && ix < C.nx;
  ix += ((ix < 0) ? C.nx : 0) - ((ix >= C.nx) ? C.nx : 0);
  return true;
}

__device__ __forceinline__ void kahan_add(float &s, float &c, float v) {
  const float y = v - c;
  const float t = s + y;
  c = (t - s) - y;
  s = t;
}

// ---------------------------------------------------------------------------
// K1: push + deposit, one CTA per tile.  The input of tile t is its own
// slots plus the particles that the previous step posted for it in the
// outboxes of its (up to 8) neighbouring tiles (`Oin`); leavers of this step
// go to this tile's slot of `O`.
//
// Own particles keep their slots: each is written back to the slot it was
// read from (a particle that leaves writes a hole there), so the cell order
// the sort gave the tile survives until the next sort except for the few
// particles that change cell.  The particles bound for the tile are listed
// from the neighbours' outboxes (one warp per neighbour), pushed in full
// warps after the own ones and appended after slot np.  The main loop has
// no block-wide barrier.
//
// Every warp takes an equal, contiguous share of the tile's slots, 32 slots
// (a unit) at a time.  Lane l meets the particles l kLaneRun ...
// l kLaneRun + kLaneRun - 1 of a chunk of the sorted order one after another,
// and sums their single-segment currents in registers while they stay in one
// cell; a lane adds its sums to J when its cell changes.  The deterministic
// builds do that with integers (RunSums): 115 us for 4.2 M particles on 512^2
// cells, where the sums over the lanes of a cell, with 24 words a shuffle
// step, took 188 to 213; 332 against 683 us for 16.8 M.
//
// What bounds it (fast build, 2048^2 cells, 67 M particles): no single unit.
// A launch takes 0.940 ms against 0.49 ms for its 48 bytes a particle at the
// measured HBM rate, with 57 % of the issue slots, 60 % of the L1 data passes,
// 62 % of the SM's request port (the reductions on J) and 43 % of DRAM in
// use, and a third of a warp's time spent waiting for its next particles.
// It took 0.993 ms and 446 instructions a unit (307 now) before the work of
// cell-crossing particles moved out of the main loop, the float pairs, the
// contiguous shares and the particle prefetch in registers; writing the tile
// back in cell order from here (in place of the sort pass) was slower
// (1.13 ms): scattered 16-byte stores make L2 fetch what they do not cover.
// ---------------------------------------------------------------------------
// resident CTAs per SM the float builds are compiled for: 6 (up to 80
// registers a thread) measured faster than 7 (72, spilling in the main loop;
// the shared memory of 7 tiles leaves little L1 to catch the spills: 1.058
// against 0.942 ms a 2048^2 launch) and 5 (0.931 there, but 8 % slower on
// grids of about a thousand tiles, which then take two rounds)
#ifndef ZC_PUSH_MIN_CTAS
#define ZC_PUSH_MIN_CTAS 6
#endif
// the deterministic builds: 768 threads per SM (80 registers each; 512^2, 32 x
// 16 tiles, measured before a lane's sums were cut in 32 bits: 118 us; 512
// threads, no spills: 120; 1024, 64 registers: 199)
constexpr int kDetThreads = 768;
//
// SPLIT: a tile is worked on by a cluster of `parts` CTAs (this one is
// `rank`), for grids with too few tiles to fill the GPU.  Each stages the
// tile's fields, pushes its share of the slots and pulls from its share of
// the neighbours; the counters of leavers and appended arrivals are rank 0's
// (distributed shared memory).
template <int TX, int TY, int NT, bool DET, bool SPLIT>
__device__ __forceinline__ void push_tile(const CUtensorMap &tm_eb, const PushSpecies &A, int *err, const FixedJ &fj,
                                          int t, int rank, int parts) {
  const Particles &pin = A.pin, &pout = A.pout;
  const TileSet &T = A.T;
  const Outbox &Oin = A.Oin, &O = A.O;
  const Spill &S = A.S;
  const PushConst &C = A.C;
#ifdef ZC_FAST
  constexpr int BW = push_box_w(TX, true);
#else
  constexpr int BW = push_box_w(TX, false);
#endif
  constexpr int BH = TY + 3;
  constexpr int PL = BW * BH;
  constexpr int NW = NT / 32;
  using LAY = JTileLayout<TX, TY>;
  __shared__ __align__(128) float sEB[6 * PL];  // E/B tile with its halo
  // deterministic builds: J tile, integer parts h, m, l (jsplit)
  __shared__ __align__(16) int sJi[DET ? 3 * LAY::N : 1];
  __shared__ unsigned long long s_ekin[2];                // fixed-point kinetic energy (DET)
  __shared__ __align__(8) uint64_t bar;
  __shared__ double sred[NW];
  // per-warp queue of the particles that need more than the common case (see
  // `finish`): x, y before and ux, uy, uz after the push, the cell word and
  // the own slot; finished 32 at a time, so at most 31 wait when the next
  // unit's 32 lanes queue theirs.  The exact builds keep mx, my and q v_z too
  // (a square root and a division that the fast builds make again in a few
  // instructions), unless the tile's own memory leaves no room (32x32: a CTA
  // less a multiprocessor).
#ifdef ZC_FAST
  constexpr bool KEEP = false;
#else
  constexpr bool KEEP = TX * TY <= 512;
#endif
  constexpr int QCAP = 63;
  __shared__ float qf[NW][KEEP ? 8 : 5][QCAP];
  __shared__ unsigned qc[NW][QCAP];
  __shared__ int qs[NW][QCAP];
  __shared__ int nb[8], s_nnb;        // distinct neighbour tiles
  // incoming particles bound for this tile, listed as (outbox slot << 4 |
  // neighbour) so that they are pushed in full warps
  constexpr int INCAP = 64;
  __shared__ int s_in[INCAP];
  __shared__ int s_nin;
  __shared__ int s_app, s_leave;      // appended arrivals, leavers (warp-aggregated atomics)

  const int tx = t % C.ntx, ty = t / C.ntx;
  const int cx0 = tx * TX, cy0 = ty * TY;  // first cell of the tile = buffer coords of its halo
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1;
  int errbits = 0;
  int qcount = 0;  // warp-uniform

  const unsigned base = (unsigned)T.off[t];  // (tile offsets are below 2^31)
  const int n_own = T.np[t];
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    mbar_expect_tx(&bar, 6 * PL * 4);
    tma_load_3d(sEB, &tm_eb, cx0, cy0, 0, &bar);
    s_nin = 0;
    s_app = 0;
    s_leave = 0;
    s_ekin[0] = 0;
    s_ekin[1] = 0;
  }
  if (warp == NW - 1) {
    // the distinct neighbour tiles, one a lane
    const int m = lane + (lane >= 4);  // 3 x 3 without the middle
    int x = tx + m % 3 - 1, y = ty + m / 3 - 1;
    y += (y < 0) ? C.nty : 0;
    y -= (y >= C.nty) ? C.nty : 0;
    const bool out = x < 0 || x >= C.ntx;
    x += (x < 0) ? C.ntx : 0;
    x -= (x >= C.ntx) ? C.ntx : 0;
    const int id = x + y * C.ntx;
    const bool is = lane < 8 && !(out && C.mw) && id != t;
    const unsigned same = __match_any_sync(0xffffffffu, is ? id : -1 - lane);
    const bool first = is && __ffs(same) - 1 == lane;
    const unsigned fm = __ballot_sync(0xffffffffu, first);
    if (first) nb[__popc(fm & below)] = id;
    if (lane == 0) s_nnb = __popc(fm);
  }
  // This warp's slots: an equal share of the tile's units of 32 slots, one
  // contiguous run (equal to a unit, so that no warp waits a chunk's time for
  // another at the end).  Its first unit is on its way before the fields are.
  const int gwarp = SPLIT ? rank * NW + warp : warp, nwarps = SPLIT ? parts * NW : NW;
  const int units = (n_own + 31) / 32;
  const int share = units / nwarps, extra = units % nwarps;
  const int c_begin = 32 * (gwarp * share + min(gwarp, extra));
  const int c_end = min(n_own, c_begin + 32 * (share + (gwarp < extra ? 1 : 0)));
  // this lane's slot in the unit that starts at slot c
  const auto slot_of = [&](int c) {
    return c + lane;
  };
  // a lane without a particle carries the last unit's particle, a hole's
  // momenta (zero at first, then pushed along at its cell's centre), or these
  // zeros: finite values whose results `valid` masks;
  // its position is set to the cell centre (a hole's is stale)
  float4 nu = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 nxy = make_float2(0.f, 0.f);
  int ns = slot_of(c_begin);
  if (c_begin < c_end && ns < n_own) {
    nu = __ldcs(&pin.u[base + ns]);
    nxy = __ldcs(&pin.xy[base + ns]);
  }
  if constexpr (DET)
    for (int k = threadIdx.x; k < 3 * LAY::N; k += NT) sJi[k] = 0;
  __syncthreads();
  if constexpr (SPLIT) cluster_arrive();  // np is read, the counters are zero
  // the outboxes of this warp's neighbours: counts and first entries
  constexpr int NBW = (8 + NW - 1) / NW;
  const int nnb = s_nnb;
  int in_n[NBW], in_dst[NBW];
#pragma unroll
  for (int q = 0; q < NBW; ++q) {
    const int m = gwarp + q * nwarps;
    in_n[q] = m < nnb ? Oin.cnt[nb[m]] : 0;
    in_dst[q] = (m < nnb && lane < Oin.cap) ? Oin.dst[(long long)nb[m] * Oin.cap + lane] : -1;
  }
  const bool loaded = mbar_wait_bounded(&bar, 0);
  if (!loaded) errbits |= ERR_TIMEOUT;
  if constexpr (SPLIT) cluster_wait();

#ifdef ZC_FAST
  // in place: planes Ex Ey Ez Bx By Bz -> Ez, Bz, pairs (Ex, By), (Ey, Bx)
  {
    constexpr int NK = (PL + NT - 1) / NT;
    float v[NK][6];
#pragma unroll
    for (int n = 0; n < NK; ++n) {
      const int k = min((int)threadIdx.x + n * NT, PL - 1);
#pragma unroll
      for (int c = 0; c < 6; ++c) v[n][c] = sEB[c * PL + k];
    }
    __syncthreads();
    float2 *xb = reinterpret_cast<float2 *>(sEB + 2 * PL), *yb = xb + PL;
#pragma unroll
    for (int n = 0; n < NK; ++n) {
      const int k = min((int)threadIdx.x + n * NT, PL - 1);
      sEB[k] = v[n][2];
      sEB[PL + k] = v[n][5];
      xb[k] = make_float2(v[n][0], v[n][4]);
      yb[k] = make_float2(v[n][1], v[n][3]);
    }
    __syncthreads();
  }
  const TilePairs<BW, PL> fld{reinterpret_cast<const float2 *>(sEB + 2 * PL),
                              reinterpret_cast<const float2 *>(sEB + 4 * PL), sEB, sEB + PL};
#else
  const TileFields<BW, PL> fld{sEB};
#endif
  const PushConst Cl = C;
  const auto dep = [&] {
    if constexpr (DET)
      return TileCurrentSplit<LAY>{sJi, &Cl};
    else
      return TileCurrentGlobal{fj.f + (size_t)(cy0 + 1) * fj.pitch + (cx0 + 1), fj.pitch, fj.plane};
  }();
  float ks = 0.f, kc = 0.f;
  long long khi = 0, klo = 0;  // DET: fixed-point kinetic energy of this thread's particles
  // this lane's running single-segment current and its cell word (kHole: none)
  SegCurrent acc;
#pragma unroll
  for (int q = 0; q < 8; ++q) acc.v[q] = 0.f;
  RunSums run;  // DET: the same as integers
  run.clear();
  unsigned acc_cell = kHole, nadd = 0;
  // the bits of a cell word that all cells of this tile share
  const unsigned tile_mask = ~((unsigned)(TX - 1) | (unsigned)(TY - 1) << 16);
  const unsigned tile_word = (unsigned)cx0 | (unsigned)cy0 << 16;

  // Finishes the last (at most 32) queued particles of this warp: the
  // current of all segments of the motion, the new cell, and the particle to
  // its slot, to the end of the tile or to the outbox.  Cell crossings (a few
  // per cent of the particles), the columns a window shift moves out of the
  // tile and arrivals come here; everything that only they need (the split,
  // the boundary, the destination tile, the slot counters) stays out of the
  // main loop and runs with nearly full warps.
  auto finish = [&]() {
    const int nq = min(qcount, 32);
    qcount -= nq;
    const bool act = lane < nq;
    const int e = qcount + (act ? lane : 0);
    const unsigned cw = qc[warp][e];
    const int oslot = qs[warp][e];
    float x = qf[warp][0][e], y = qf[warp][1][e];
    const float ux = qf[warp][2][e], uy = qf[warp][3][e], uz = qf[warp][4][e];
    int ix = (int)(cw & 0xffffu), iy = (int)(cw >> 16);
    int di = 0, dj = 0, code = 0, dest = 0;  // code: 0 gone, 1 stays, 2 leaves
    if (act) {
      float mx, my, qvz;
      if constexpr (KEEP) {
        mx = qf[warp][5][e];
        my = qf[warp][6][e];
        qvz = qf[warp][7][e];
      } else {
        displacement(ux, uy, uz, mx, my, qvz, Cl);  // as the push had it
      }
      errbits |= !(fabsf(mx) < 1.0f && fabsf(my) < 1.0f) ? ERR_ESCAPE : 0;
      float x1 = x + mx, y1 = y + my;
      di = (x1 >= 1.0f) - (x1 < 0.0f);
      dj = (y1 >= 1.0f) - (y1 < 0.0f);
      x1 -= di;
      y1 -= dj;
      const Seg a = zigzag_first(dep, ix & (TX - 1), iy & (TY - 1), di, dj, x, y, mx, my, Cl.qnx, Cl.qny, qvz);
      add_current(dep, a.ix, a.iy, segment_current(a, Cl.qnx, Cl.qny));
      x = x1;
      y = y1;
      const bool keep = apply_boundary(ix, iy, di, dj, Cl);
      // (the cell is inside the grid when the particle is kept; dest is unused otherwise)
      dest = (int)((unsigned)ix / TX) + (int)((unsigned)iy / TY) * Cl.ntx;
      code = keep ? ((dest == t) ? 1 : 2) : 0;
      if (oslot >= 0) {
        if (code == 1) store_particle(pout, base + oslot, ix, iy, x, y, ux, uy, uz);
        else store_hole(pout, base + oslot);
      }
    }
    __syncwarp();
    // leavers to the outbox, arrivals that stay appended after slot np: one
    // shared-memory atomic per warp and kind
    const bool app = code == 1 && oslot < 0;
    const unsigned mleave = __ballot_sync(0xffffffffu, code == 2);
    const unsigned mapp = __ballot_sync(0xffffffffu, app);
    if (mleave | mapp) {
      int lb = 0, ab = 0;
      if (lane == 0) {
        if constexpr (SPLIT) {
          if (mleave) lb = rank0_add(&s_leave, __popc(mleave));
          if (mapp) ab = rank0_add(&s_app, __popc(mapp));
        } else {
          if (mleave) lb = atomicAdd(&s_leave, __popc(mleave));
          if (mapp) ab = atomicAdd(&s_app, __popc(mapp));
        }
      }
      lb = __shfl_sync(0xffffffffu, lb, 0);
      ab = __shfl_sync(0xffffffffu, ab, 0);
      if (code == 2) {
        const int s = lb + __popc(mleave & below);
        const long long obase = (long long)t * O.cap;
        if (s < O.cap) {
          store_particle(O.p, obase + s, ix, iy, x, y, ux, uy, uz);
          O.dst[obase + s] = dest;
        } else {
          spill_particle(S, &errbits, ix, iy, x, y, ux, uy, uz);
        }
      } else if (app) {
        const int s = n_own + ab + __popc(mapp & below);
        if (s < T.cap[t]) store_particle(pout, base + s, ix, iy, x, y, ux, uy, uz);
        else spill_particle(S, &errbits, ix, iy, x, y, ux, uy, uz);
      }
    }
    __syncwarp();  // the queue is read before it is filled again
  };

  // One particle per lane: push, and in the common case (it stays in its
  // cell) current and output right here: the cell word is written back as it
  // was read.  The other particles are queued for `finish`.  The 32 lanes of
  // a warp call it together (warp-level collectives only).  `oslot` is the
  // lane's own slot (>= 0) or negative (none); `incoming` marks arriving
  // particles, which have no slot yet and all go through the queue.  A lane
  // without a particle (`valid` false) runs the same instructions on finite
  // values; its slot, a hole, is written as the hole it is.
  auto process = [&](bool valid, int oslot, bool incoming, unsigned cw, float x, float y, float ux, float uy,
                     float uz) {
    // the cell in the tile (sizes are powers of two, the tile starts at a
    // multiple of them): always inside the staged halo
    errbits |= (valid && ((cw ^ tile_word) & tile_mask)) ? ERR_ESCAPE : 0;
    const int li = (int)(cw & (TX - 1)), lj = (int)((cw >> 16) & (TY - 1));
    float mx, my, qvz;
    const float x0 = x, y0 = y;
    const float kin = push_particle(fld, li, lj, x, y, ux, uy, uz, mx, my, qvz, Cl);
    if constexpr (DET) {
      long long h, l;
      efix_split(valid ? kin : 0.0f, h, l);
      khi += h;
      klo += l;
    } else {
      kahan_add(ks, kc, valid ? kin : 0.f);
    }
    const float x1 = x0 + mx, y1 = y0 + my;
    // inside [0, 1) on both axes, as unsigned bit patterns (negative values,
    // -0 and NaN compare above); `finish` tells the cases apart
    const unsigned top = max((unsigned)__float_as_int(x1), (unsigned)__float_as_int(y1));
    const bool queue = valid && (incoming || top >= 0x3f800000u || li < Cl.shift);
    const bool single = valid && !queue;
    // the output, before the current sums so that the particle's registers
    // are free while they run
    if (oslot >= 0 && !queue) {
      pout.u[base + oslot] = make_float4(ux, uy, uz, __int_as_float((int)(valid ? cw - (unsigned)Cl.shift : kHole)));
      pout.xy[base + oslot] = make_float2(x1, y1);
    }
    {
      const unsigned qm = __ballot_sync(0xffffffffu, queue);
      if (qm) {
        if (queue) {
          const int e = qcount + __popc(qm & below);
          qf[warp][0][e] = x0;
          qf[warp][1][e] = y0;
          qf[warp][2][e] = ux;
          qf[warp][3][e] = uy;
          qf[warp][4][e] = uz;
          if constexpr (KEEP) {
            qf[warp][5][e] = mx;
            qf[warp][6][e] = my;
            qf[warp][7][e] = qvz;
          }
          qc[warp][e] = cw;
          qs[warp][e] = oslot;
        }
        qcount += __popc(qm);
        __syncwarp();
      }
    }
    // the whole motion inside the cell: one segment (particles.c:781-797);
    // the other lanes contribute nothing here: every contribution is
    // proportional to dx, dy or qvz, so zeroing those three zeroes all eight
    Seg a;
    a.x0 = x0;
    a.y0 = y0;
    a.dx = single ? mx : 0.f;
    a.dy = single ? my : 0.f;
    a.x1 = x1;
    a.y1 = y1;
    a.qvz = single ? qvz * 0.5f : 0.f;
    a.ix = li;
    a.iy = lj;
    SegCurrent cur = segment_current(a, Cl.qnx, Cl.qny);

    if constexpr (DET) {
      // every contribution rounded to fixed point first, then summed as
      // integers: the same total whatever lanes hold which particles
      if (Cl.js_run) {
        // the lane's running sums: to the J tile when its cell changes, and
        // before they can overflow
        const bool full = (++nadd & 511) == 0;
        const bool change = (single && cw != acc_cell) || full;
        if (change && acc_cell != kHole) run.flush(dep, acc_cell);
        run.add(cur, Cl.js);
        acc_cell = single ? cw : (full ? kHole : acc_cell);
      } else if (single) {  // charges that the sums' two parts are too short for
        add_current(dep, li, lj, cur);
      }
    } else {
      // the lane's running sum: added to J when the lane's cell changes
      // (the sum is over this lane's particles of one cell, in order)
      const bool change = single && cw != acc_cell;
      if (change && acc_cell != kHole) add_current(dep, acc_cell & (TX - 1), (acc_cell >> 16) & (TY - 1), acc);
      const float carry = change ? 0.0f : 1.0f;  // acc + cur, or cur
#ifdef ZC_FAST
      constexpr int pa[4] = {0, 1, 4, 5};  // pairs (0, 2), (1, 3), (4, 6), (5, 7), as they were computed
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int q = pa[k];
        const float2 v = __ffma2_rn(make_float2(acc.v[q], acc.v[q + 2]), make_float2(carry, carry),
                                    make_float2(cur.v[q], cur.v[q + 2]));
        acc.v[q] = v.x;
        acc.v[q + 2] = v.y;
      }
#else
#pragma unroll
      for (int q = 0; q < 8; ++q) acc.v[q] = __fmaf_rn(acc.v[q], carry, cur.v[q]);
#endif
      acc_cell = change ? cw : acc_cell;
    }
  };

  // incoming particles: warp w scans the outboxes of neighbours w, w + NW,
  // ... for the slots bound for this tile and lists them; a full list
  // leaves the rest to be pushed right here
#pragma unroll
  for (int q = 0; q < NBW; ++q) {
    const int m = gwarp + q * nwarps;
    if (m >= nnb) break;
    const int n = in_n[q];
    const long long ob = (long long)nb[m] * Oin.cap;
    for (int e0 = 0; e0 < n; e0 += 32) {
      const int e = e0 + lane;
      const bool bound = e < n && (e0 == 0 ? in_dst[q] : Oin.dst[ob + e]) == t;
      const unsigned bm = __ballot_sync(0xffffffffu, bound);
      if (!bm) continue;
      int slot = 0;
      if (lane == 0) slot = atomicAdd(&s_nin, __popc(bm));
      slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(bm & below);
      if (bound && slot < INCAP) s_in[slot] = (e << 4) | m;
      const bool over = bound && slot >= INCAP;
      if (__any_sync(0xffffffffu, over)) {
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 r = make_float2(0.5f, 0.5f);
        if (over) u = Oin.p.u[ob + e], r = Oin.p.xy[ob + e];
        process(over, -1, true, (unsigned)__float_as_int(u.w), r.x, r.y, u.x, u.y, u.z);
        if (qcount >= 32) finish();
      }
    }
  }
  __syncthreads();

  // own slots, 32 at a time (a unit), the next unit loaded into registers
  // while one is pushed (staging it in shared memory costs as many
  // shared-memory passes as half the field gather).  In a full chunk lane l
  // takes slot 32 k + l at step k, which holds the chunk's particle
  // l kLaneRun + k in cell order.  Every particle goes back to the slot it came
  // from.
  for (int c = c_begin; c < c_end;) {
    const float4 uu = nu;
    const unsigned cw = (unsigned)__float_as_int(uu.w);
    const int s = ns;
    const bool inr = s < n_own, valid = inr && cw != kHole;
    const float x = valid ? nxy.x : 0.5f, y = valid ? nxy.y : 0.5f;
    c += 32;
    ns = slot_of(c);
    if (c < c_end && ns < n_own) {
      nu = __ldcs(&pin.u[base + ns]);
      nxy = __ldcs(&pin.xy[base + ns]);
    }
    process(valid, inr ? s : -1, false, cw, x, y, uu.x, uu.y, uu.z);
    if (qcount >= 32) finish();
  }

  // the listed incoming particles, in units of 32 spread over the warps
  {
    const int nin = min(s_nin, INCAP);
    for (int i = warp; i * 32 < nin; i += NW) {
      const int k = i * 32 + lane;
      const bool valid = k < nin;
      float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
      float2 r = make_float2(0.5f, 0.5f);
      if (valid) {
        const int v = s_in[k];
        const long long q = (long long)nb[v & 15] * Oin.cap + (v >> 4);
        u = Oin.p.u[q];
        r = Oin.p.xy[q];
      }
      process(valid, -1, true, (unsigned)__float_as_int(u.w), r.x, r.y, u.x, u.y, u.z);
      if (qcount >= 32) finish();
    }
  }

  finish();  // what is left in the queue
  if (acc_cell != kHole) {  // the lanes' last sums
    if constexpr (DET) run.flush(dep, acc_cell);
    else add_current(dep, acc_cell & (TX - 1), (acc_cell >> 16) & (TY - 1), acc);
  }

  if constexpr (DET) {
    // kinetic energy: integer sums, exact in any order, of the whole tile
    // (its parts' too)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      khi += __shfl_down_sync(0xffffffffu, khi, off);
      klo += __shfl_down_sync(0xffffffffu, klo, off);
    }
    if (lane == 0) {
      if constexpr (SPLIT) {
        if (khi) rank0_add(&s_ekin[0], (unsigned long long)khi);
        if (klo) rank0_add(&s_ekin[1], (unsigned long long)klo);
      } else {
        if (khi) atomicAdd(&s_ekin[0], (unsigned long long)khi);
        if (klo) atomicAdd(&s_ekin[1], (unsigned long long)klo);
      }
    }
  }
  if constexpr (SPLIT) {
    cluster_arrive();  // every part's leavers, arrivals and energies are counted
    cluster_wait();
  } else {
    __syncthreads();
  }
  if (threadIdx.x == 0 && (!SPLIT || rank == 0)) {
    T.np[t] = n_own + min(s_app, T.cap[t] - n_own);
    O.cnt[t] = min(s_leave, O.cap);
    if constexpr (DET) {
      A.ekin_words[2 * (size_t)t] = (long long)s_ekin[0];
      A.ekin_words[2 * (size_t)t + 1] = (long long)s_ekin[1];
    }
  }
  if constexpr (DET) {
    // the integer J tile goes to the global fixed-point planes (units of
    // 2^-40) with 64-bit integer atomics (cells outside the buffer hold no
    // deposits)
    for (int k = threadIdx.x; k < LAY::N; k += NT) {
      const long long v = tile_node_sum(sJi, LAY::N, k, Cl.js_l);
      if (!v) continue;
      int c, r, col;
      LAY::where(k, c, r, col);
      const int gy = cy0 + r, gx = cx0 + col;
      if (gx < fj.pitch && (size_t)gy * fj.pitch < fj.plane)
        atomicAdd(&fj.p[c * fj.plane + (size_t)gy * fj.pitch + gx], (unsigned long long)(v * Cl.js_det));
    }
    if (threadIdx.x == 0 && !loaded && !mbar_wait_bounded(&bar, 0))
      errbits |= ERR_TIMEOUT;  // second bounded wait for the load still in flight
  } else {
    const double e = block_sum_double<NT>((double)ks - (double)kc, sred);
    if (threadIdx.x == 0) A.ekin[t * parts + rank] = e;

    if (threadIdx.x == 0 && !loaded && !mbar_wait_bounded(&bar, 0))
      errbits |= ERR_TIMEOUT;  // second bounded wait for the load still in flight
  }
  if (errbits) atomicOr(err, errbits);
}

// ---------------------------------------------------------------------------
// spill push: same physics from global memory (rarely non-empty), by block
// `block` of `nblocks`; leaves the block's kinetic energy in A.ekin_spill
// (deterministic builds: adds it to the two words of A.ekin_fix)
// ---------------------------------------------------------------------------
template <int NT, bool DET>
__device__ __forceinline__ void push_spill(const float *EB, const FixedJ &fj, const Grid &G, const PushSpecies &A,
                                           int *err, int block, int nblocks) {
  __shared__ double sred[NT / 32];
  const PushConst &C = A.C;
  const Particles &sin = A.Sin.p;
  const Spill &S = A.S;
  const int n = min(*A.Sin.cnt, A.Sin.cap);
  if (n == 0) {  // the usual case: nothing spilled (uniform across the blocks)
    if (!DET && threadIdx.x == 0) A.ekin_spill[block] = 0.0;
    return;
  }
  const GlobalFields fld{EB, G.pitch, G.plane};
  const auto dep = [&] {
    if constexpr (DET)
      return GlobalCurrentFixed{fj.p, fj.pitch, fj.plane, &C};
    else
      return GlobalCurrent{fj.f, G.pitch, G.plane};
  }();
  int errbits = 0;
  float ks = 0.f, kc = 0.f;
  long long khi = 0, klo = 0;
  for (int k = block * NT + threadIdx.x; k < n; k += nblocks * NT) {
    const PRec r = load_particle(sin, k);
    int ix = r.ix, iy = r.iy;
    float x = r.x, y = r.y, ux = r.ux, uy = r.uy, uz = r.uz;
    if (ix < 0 || ix >= C.nx || iy < 0 || iy >= C.ny) {
      errbits |= ERR_ESCAPE;
      ix = min(max(ix, 0), C.nx - 1);
      iy = min(max(iy, 0), C.ny - 1);
    }
    float mx, my, qvz;
    const float kin = push_particle(fld, ix, iy, x, y, ux, uy, uz, mx, my, qvz, C);
    if (!(fabsf(mx) < 1.0f && fabsf(my) < 1.0f)) errbits |= ERR_ESCAPE;
    float x1 = x + mx, y1 = y + my;
    const int di = (x1 >= 1.0f) - (x1 < 0.0f), dj = (y1 >= 1.0f) - (y1 < 0.0f);
    x1 -= di;
    y1 -= dj;
    if constexpr (DET) {
      long long h, l;
      efix_split(kin, h, l);
      khi += h;
      klo += l;
    } else {
      kahan_add(ks, kc, kin);
    }
    const Seg a = zigzag_first(dep, ix, iy, di, dj, x, y, mx, my, C.qnx, C.qny, qvz);
    add_current(dep, ix, iy, segment_current(a, C.qnx, C.qny));
    x = x1;
    y = y1;
    if (apply_boundary(ix, iy, di, dj, C)) spill_particle(S, &errbits, ix, iy, x, y, ux, uy, uz);
  }
  if constexpr (DET) {
    if (khi) atomicAdd(A.ekin_fix, (unsigned long long)khi);
    if (klo) atomicAdd(A.ekin_fix + 1, (unsigned long long)klo);
  } else {
    const double e = block_sum_double<NT>((double)ks - (double)kc, sred);
    if (threadIdx.x == 0) A.ekin_spill[block] = e;
  }
  if (errbits) atomicOr(err, errbits);
}

// ---------------------------------------------------------------------------
// kernels: one species' tiles; its spilled particles; and, for small grids,
// every species' tiles (each by a cluster of `parts` CTAs) and spilled
// particles in one launch
// ---------------------------------------------------------------------------
template <int TX, int TY, int NT, bool DET>
__global__ void __launch_bounds__(NT, DET ? kDetThreads / NT : ZC_PUSH_MIN_CTAS)
    k_push_tiles(const __grid_constant__ CUtensorMap tm_eb, const __grid_constant__ PushSpecies A, int *err,
                 FixedJ fj) {
  push_tile<TX, TY, NT, DET, false>(tm_eb, A, err, fj, blockIdx.x, 0, 1);
}

template <int NT, bool DET>
__global__ void __launch_bounds__(NT) k_push_spill(const float *EB, FixedJ fj, Grid G,
                                                   const __grid_constant__ PushSpecies A, int *err) {
  push_spill<NT, DET>(EB, fj, G, A, err, blockIdx.x, gridDim.x);
}

template <int TX, int TY, int NT, bool DET>
__global__ void __launch_bounds__(NT, DET ? kDetThreads / NT : 4)
    k_push_all(const __grid_constant__ CUtensorMap tm_eb, const __grid_constant__ PushAll P, const float *EB, Grid G,
               int *err, FixedJ fj) {
  // (the rule that splits tiles counts on these places)
  static_assert(push_all_ctas(TX, TY, DET) <= (DET ? kDetThreads / NT : 4), "more places than the launch bounds give");
  const int b = blockIdx.x, ntile = P.nsp * P.ntiles * P.parts;
  if (b < ntile) {
    const int q = b / P.parts, k = q / P.ntiles;
    push_tile<TX, TY, NT, DET, true>(tm_eb, P.sp[k], err, fj, q - k * P.ntiles, b - q * P.parts, P.parts);
  } else {
    const int k = (b - ntile) / kSpillParts;
    push_spill<NT, DET>(EB, fj, G, P.sp[k], err, (b - ntile) % kSpillParts, kSpillParts);
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <int TX, int TY, bool DET>
static cudaError_t launch_push_t(const PushLaunch &a, cudaStream_t st) {
  // 4 warps per CTA (shorter barriers, CTAs in more phases); the
  // deterministic build's integer J tile keeps 8 warps per CTA
  constexpr int NT = (DET && TX * TY >= 256) ? 256 : 32 * kPushWarps;
  if (a.all) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(a.all->nsp * (a.all->ntiles * a.all->parts + kSpillParts));
    cfg.blockDim = dim3(NT);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = a.all->parts;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_push_all<TX, TY, NT, DET>, *a.tm_eb, *a.all, a.EB, a.G, a.err, a.fj);
  }
  k_push_tiles<TX, TY, NT, DET><<<a.ntiles, NT, 0, st>>>(*a.tm_eb, *a.one, a.err, a.fj);
  return cudaGetLastError();
}

template <bool DET>
static cudaError_t launch_push_tiles_variant(const PushLaunch &a, cudaStream_t st) {
  const int TX = a.TX, TY = a.TY;
#define ZC_TILE(X, Y) \
  if (TX == X && TY == Y) return launch_push_t<X, Y, DET>(a, st);
  ZC_TILE(16, 16)
  ZC_TILE(8, 8)
  ZC_TILE(16, 8)
  ZC_TILE(32, 16)
  ZC_TILE(32, 32)
  ZC_TILE(8, 16)
  ZC_TILE(16, 32)
#undef ZC_TILE
  return cudaErrorInvalidValue;
}

template <bool DET>
static cudaError_t launch_push_spill_variant(const PushLaunch &a, int nblocks, cudaStream_t st) {
  k_push_spill<256, DET><<<nblocks, 256, 0, st>>>(a.EB, a.fj, a.G, *a.one, a.err);
  return cudaGetLastError();
}
