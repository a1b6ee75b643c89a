// forward_quad.cuh -- row-quad forward projector (device code; instantiated and
// launched by forward_quad.cu).
//
// A thread marches four vertically adjacent rays of one detector column.  Rays
// that leave the volume through its side faces have the column's in-plane clip,
// so their k-th samples share the in-plane position (e_k, d_k) and differ only in
// z, by the row distance p (texels), which is the same between all rows and
// nearly constant over a slab.  For p in one of the intervals (0, 1/3), (1/3, 1/2),
// (1/2, 2/3), (2/3, 1), (1, 4/3) row i's plane is one of two known planes above
// the lowest row's, so the 3 to 6 planes of the quad are interpolated in e and d
// once, at fixed offsets from one address, and each row takes one of two z lerps.
// Every value is the slab kernel's for that ray (same texels, operations and
// order): results are bitwise equal to it.
//
// What bounds it.  Not HBM: the volume is staged box by box from L2 (about 9 bytes
// per ray and voxel of depth), and not issue slots: measured on B200, next to
// other work, an FFMA with three register operands takes 1.5 cycles of an SM
// quarter, one with two 1.1, any ALU operation (compare, select, integer) 2, a
// shared load 2, and a packed FFMA2 2.1 to 2.9 for its two results.  So the inner
// loop has no select (the second candidate of a row is a predicated multiply-add),
// no index clamp (a slab's samples are checked at their two ends, coordinates being
// monotone along a ray) and packs the plane interpolations by pairs of planes.
// 36 views of 512x384 into 256^3 (p = 0.44 to 0.63), the forward kernel alone: 3.46
// ms with the previous row-quad kernel (planes selected per row, 16-column warps), 3.11
// once silhouette rays were taken by whole warps, 2.57 now (1060 GSamples/s), with
// 103 instead of 125 warp instructions per four samples and 29.7 instead of 25.8 of
// 32 lanes busy.
//  * Warps hold 8 columns x 4 row groups: columns enter and leave the volume some
//    voxels apart, so 16-column warps keep 27.7 lanes busy and 32-column warps 20.
//    The box strides (36 x 9, 28 x 7, 28 x 5, 36 x 5 words) put the four groups, a few planes
//    apart, on different banks.
//  * Rays clipped by the top or bottom face have samples of their own.  A warp deals
//    them out over its lanes (own rays); marched by the thread of their row group they
//    kept the warp waiting for four rays in a row (180 views of 256x192 into 128^3:
//    3.13 ms instead of 2.44).
#pragma once

#include "forward_host.h"

namespace cbct {

namespace {

// Tile and pipeline shape: TU columns x G groups of four rows per CTA, a warp
// holding WC columns x 32 / WC groups, slabs of TS voxels, NS TMA stages.  SKEW: a
// warp's upper two groups sit eight columns beside its lower two.  With rows a texel
// apart the groups are four planes apart, which any dense box puts 16 banks apart, so
// the first and third fall on the same banks; eight columns to the side they fall
// between (180 views of 256x192 into 128^3: bank conflicts 249 to 133 million
// wavefronts, 2.42 to 2.31 ms, although 18 instead of 21 lanes are busy).
template <int TU_, int G_, int WC_, int TS_, int NS_, bool SKEW_ = false>
struct QuadCfg {
  static constexpr int R = 4, TU = TU_, G = G_, WC = WC_, TS = TS_, NS = NS_;
  static constexpr bool SKEW = SKEW_;
  static_assert(!SKEW_ || (WC_ == 8 && TU_ == 16), "a skewed warp has two halves of 8 columns");
  static constexpr int TV = 4 * G_, threads = TU_ * G_, BY = TS_ + 1;
  static_assert(TU_ % WC_ == 0 && G_ % (32 / WC_) == 0, "a tile holds whole warps");
  // Column and row group of a thread in the tile.
  static __device__ __forceinline__ int col(int tid) {
    const int warp = SKEW ? (tid >> 5) ^ ((tid & 31) / (2 * WC)) : tid >> 5;
    return (warp % (TU / WC)) * WC + (tid & 31) % WC;
  }
  static __device__ __forceinline__ int group(int tid) {
    return ((tid >> 5) / (TU / WC)) * (32 / WC) + (tid & 31) / WC;
  }
};

template <int NS>
struct QuadShared {
  uint64_t bars[NS];
  int mlo, mhi, abort_flag;
  double red[8];
};

// One plane at q: the same operations, the first two interpolations packed.
template <class V, int BX, int FORM>
__device__ __forceinline__ float plane1(const V* __restrict__ q, float2 te, float2 nte, float2 td, float2 ntd) {
  const float2 a = make_float2(sm_f(q[0]), sm_f(q[BX])), b = make_float2(sm_f(q[1]), sm_f(q[BX + 1]));
  if (FORM == kLerpXisE) {
    const float2 x = lerp2_gather(a, b, te);
    return fmaf(td.x, x.y - x.x, x.x);
  }
  if (FORM == kLerpXisD) {
    const float2 x = lerp2_gather(make_float2(a.x, b.x), make_float2(a.y, b.y), td);
    return fmaf(te.x, x.y - x.x, x.x);
  }
  const float2 e = __ffma2_rn(te, b, __ffma2_rn(nte, a, a));
  return fmaf(td.x, e.y, fmaf(ntd.x, e.x, e.x));
}

// Samples k .. ke-1 of four rows at any distance: two planes per row.
template <class V, int BX, int BY, int FORM>
__device__ __forceinline__ void quad_march_any(const V* __restrict__ s, float k, float ke, float2 c0, float2 dc,
                                               const float2 (&z0)[2], const float2 (&dz)[2], float cmo,
                                               float2 (&acc)[2]) {
  constexpr int BXY = BX * BY;
  for (; k < ke; k += 1.f) {
    const float2 kk = make_float2(k, k);
    const float2 pq = __ffma2_rn(kk, dc, c0);
    const float2 f = floor2_small(pq);
    const float2 t = sub2(pq, f);
    const float cb = fmaf(f.y, float(BX), f.x) + cmo;
    const float2 te = make_float2(t.x, t.x), nte = make_float2(-t.x, -t.x);
    const float2 td = make_float2(t.y, t.y), ntd = make_float2(-t.y, -t.y);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float2 cz = __ffma2_rn(kk, dz[j], z0[j]);
      const float2 fz = floor2_small(cz);
      const float2 ix = __ffma2_rn(fz, make_float2(float(BXY), float(BXY)), make_float2(cb, cb));
      const V* q0 = s + (unsigned)int_of_biased(ix.x);
      const V* q1 = s + (unsigned)int_of_biased(ix.y);
      const float2 lo = planes2<V, BX, FORM>(q0, q1, te, nte, td, ntd);
      const float2 hi = planes2<V, BX, FORM>(q0 + BXY, q1 + BXY, te, nte, td, ntd);
      acc[j] = __fadd2_rn(acc[j], __ffma2_rn(sub2(cz, fz), sub2(hi, lo), lo));
    }
  }
}

// Samples k .. ke-1 of one ray.
template <class V, int BX, int BY, int FORM>
__device__ __forceinline__ void ray_march(const V* __restrict__ s, float k, float ke, float2 c0, float2 dc, float z0,
                                          float dz, float cmo, float& acc) {
  constexpr int BXY = BX * BY;
  auto eval = [&](float q) {
    const float ce = fmaf(q, dc.x, c0.x), cd = fmaf(q, dc.y, c0.y), cz = fmaf(q, dz, z0);
    const float fe = floor_small(ce), fd = floor_small(cd), fz = floor_small(cz);
    const float te = ce - fe, td = cd - fd;
    const V* b = s + (unsigned)int_of_biased(fmaf(fz, float(BXY), fmaf(fd, float(BX), fe)) + cmo);
    const float2 l = planes2<V, BX, FORM>(b, b + BXY, make_float2(te, te), make_float2(-te, -te), make_float2(td, td),
                                    make_float2(-td, -td));
    return fmaf(cz - fz, l.y - l.x, l.x);
  };
  for (; k + 1.f < ke; k += 2.f) {
    const float v0 = eval(k), v1 = eval(k + 1.f);
    acc += v0;
    acc += v1;
  }
  if (k < ke) acc += eval(k);
}

// Samples k .. ke-1 of four rows whose planes are known up to one step: relative
// to the lowest row's plane f0, row i's lower plane is Ci or Ci + 1 at every
// sample (the caller checked the row distance at both ends, and z >= 0).  s is the
// box's address minus its origin's element index.
template <class V, int BX, int BY, int FORM, int C1, int C2, int C3>
__device__ __forceinline__ void quad_march(const V* __restrict__ s, float k, float ke, float2 c0, float2 dc,
                                           const float2 (&z0)[2], const float2 (&dz)[2], float2 (&acc)[2]) {
  constexpr int BXY = BX * BY, NP = C3 + 3;
  // a = z - lower candidate plane (exact for planes >= 0); the upper candidate
  // where a >= 1.
  auto row = [](float a, float g0, float l0, float g1, float l1) {
    float v;
    asm("{\n\t.reg .pred p;\n\t.reg .f32 b;\n\t"
        "setp.ge.f32 p, %1, 0f3F800000;\n\t"
        "fma.rn.f32 %0, %1, %2, %3;\n\t"
        "@p add.rn.f32 b, %1, 0fBF800000;\n\t"
        "@p fma.rn.f32 %0, b, %4, %5;\n\t}"
        : "=&f"(v)
        : "f"(a), "f"(g0), "f"(l0), "f"(g1), "f"(l1));
    return v;
  };
  const float2 round2 = make_float2(kRoundC, kRoundC);
  for (; k < ke; k += 1.f) {
    const float2 kk = make_float2(k, k);
    const float2 zz0 = __ffma2_rn(kk, dz[0], z0[0]), zz1 = __ffma2_rn(kk, dz[1], z0[1]);
    const float2 pq = __ffma2_rn(kk, dc, c0);
    const float2 bp = __fadd2_rd(pq, round2);
    const float2 nf = __ffma2_rn(bp, make_float2(-1.f, -1.f), round2);   // -floor, exact
    const float2 t = __fadd2_rn(pq, nf);
    const float te = t.x, td = t.y, be = bp.x, nfd = nf.y;
    const float nf0 = kRoundC - __fadd_rd(zz0.x, kRoundC);
    // the biased sum's mantissa holds the element index (plus the box origin, taken off s):
    // less than 2^22, see box_index_bound
    const V* q = s + int_of_biased(fmaf(nf0, -float(BXY), fmaf(nfd, -float(BX), be)));
    float L[NP], g[NP];
    const float2 te2 = make_float2(te, te), nte2 = make_float2(-te, -te), td2 = make_float2(td, td), ntd2 = make_float2(-td, -td);
#pragma unroll
    for (int j = 0; j + 1 < NP; j += 2) {
      const float2 l = planes2<V, BX, FORM>(q + j * BXY, q + (j + 1) * BXY, te2, nte2, td2, ntd2);
      L[j] = l.x;
      L[j + 1] = l.y;
    }
    if (NP & 1) L[NP - 1] = plane1<V, BX, FORM>(q + (NP - 1) * BXY, te2, nte2, td2, ntd2);
#pragma unroll
    for (int j = 0; j + 1 < NP; ++j) g[j] = L[j + 1] - L[j];
    const float2 a0 = __fadd2_rn(zz0, make_float2(nf0, nf0 - float(C1)));
    const float2 a1 = __fadd2_rn(zz1, make_float2(nf0 - float(C2), nf0 - float(C3)));
    const float v0 = fmaf(a0.x, g[0], L[0]), v1 = row(a0.y, g[C1], L[C1], g[C1 + 1], L[C1 + 1]);
    const float v2 = row(a1.x, g[C2], L[C2], g[C2 + 1], L[C2 + 1]), v3 = row(a1.y, g[C3], L[C3], g[C3 + 1], L[C3 + 1]);
    acc[0] = __fadd2_rn(acc[0], make_float2(v0, v1));
    acc[1] = __fadd2_rn(acc[1], make_float2(v2, v3));
  }
}

// Class of four rows from the least and largest distance of the outer two over
// a range of samples (rows are equally spaced): the interval of row distances
// (0, 1/3), (1/3, 1/2), (1/2, 2/3), (2/3, 1), (1, 4/3), or -1.  The margin
// covers the rounding of the coordinates.
__device__ __forceinline__ int quad_class(float smin, float smax) {
  constexpr float m = 6e-3f;
  if (smin >= m && smax <= 1.f - m) return 0;
  if (smin >= 1.f + m && smax <= 1.5f - m) return 1;
  if (smin >= 1.5f + m && smax <= 2.f - m) return 2;
  if (smin >= 2.f + m && smax <= 3.f - m) return 3;
  if (smin >= 3.f + m && smax <= 4.f - m) return 4;
  return -1;
}

// A ray marched by itself: pixel, next sample, sum, frame coordinates.
struct OwnRay {
  int u, v;
  float k, acc;
  float2 c, d;
  float z0, dz;
};

// One CTA: ray tile `tile` of the call.  GATHER: the gather kernel's
// interpolation (see LerpForm).
template <class V, int BX, class C, bool GATHER>
__device__ __forceinline__ void fwd_quad_body(const CUtensorMap* map_v, const CUtensorMap* map_t,
                                              const V* __restrict__ vol, const ViewParams* __restrict__ views,
                                              const GridConst& gc, int BZ, int nsl_max, bool check, const FwdOut& o,
                                              int* flags, const TileId& tile, unsigned char* smem_raw,
                                              QuadShared<C::NS>& sh) {
  constexpr int R = 4, TS = C::TS, NS = C::NS, BY = C::BY, BXY = BX * BY;
  const ViewParams vp = views[tile.z];
  const int dom = vp.dom;
  const bool up = vp.dsgn > 0;
  const CUtensorMap* map = dom ? map_v : map_t;
  const int tid = threadIdx.x;
  const int p = tile.z;
  const int u0 = tile.x * C::TU, v0 = tile.y * C::TV;
  const int u = u0 + C::col(tid), vb = v0 + R * C::group(tid);
  const float Nf = float(gc.N);

  if (tid == 0) {
    sh.mlo = INT_MAX;
    sh.mhi = INT_MIN;
    sh.abort_flag = 0;
    for (int i = 0; i < NS; ++i) mbar_init(&sh.bars[i], 1);
    fence_mbar_init();
  }
  __syncthreads();

  // Rays in the view's frame (e = cross axis, d = slab axis): start and step.
  // Four rows that leave through the volume's side faces have one clip, hence
  // one in-plane path (a quad); the rays of other rows (`own`) are marched one by
  // one and dealt out over the warp's lanes, so that a row group cut by the top or
  // bottom face does not keep the whole warp waiting for four rays in a row.
  const int lane = tid & 31;
  float2 c0, dc, z0[R / 2], dz[R / 2], acc[R / 2];
  float kf = 0.f;
  unsigned hit = 0;
  bool quad = true;
  {
    const int uc = min(u, gc.W - 1);
    float a1 = 0.f, a2 = 0.f, zs[R], zd[R];
    int mn = INT_MAX, mx = INT_MIN;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const Ray r = make_ray(vp, gc, uc, min(vb + i, gc.H - 1));
      const float2 c = dom ? make_float2(r.c0x, r.c0y) : make_float2(r.c0y, r.c0x);
      const float2 d = dom ? make_float2(r.dcx, r.dcy) : make_float2(r.dcy, r.dcx);
      zs[i] = r.c0z;
      zd[i] = r.dcz;
      if (i == 0) { a1 = r.a1; a2 = r.a2; c0 = c; dc = d; }
      quad = quad && r.a1 == a1 && r.a2 == a2;
      if (u < gc.W && vb + i < gc.H && r.a2 > r.a1) {
        hit |= 1u << i;
        const int m0 = (max(int(floorf(c.y)), kSlabBase) - kSlabBase) / TS;
        const int m1 = (max(int(floorf(fmaf(Nf - 1.f, d.y, c.y))), kSlabBase) - kSlabBase) / TS;
        mn = min(mn, min(m0, m1));
        mx = max(mx, max(m0, m1));
      }
    }
    if (mn <= mx) {
      atomicMin(&sh.mlo, mn);
      atomicMax(&sh.mhi, mx);
    }
#pragma unroll
    for (int j = 0; j < R / 2; ++j) {
      z0[j] = make_float2(zs[2 * j], zs[2 * j + 1]);
      dz[j] = make_float2(zd[2 * j], zd[2 * j + 1]);
      acc[j] = make_float2(0.f, 0.f);
    }
  }
  quad = quad && hit == 15u;
  // Own rays of the warp in row order; this lane marches the lane-th, the
  // (lane + 32)-th and so on (their state lives in local memory).
  OwnRay own[R];
  int n_own = 0;
  {
    unsigned b[R];
#pragma unroll
    for (int j = 0; j < R; ++j) b[j] = __ballot_sync(0xffffffffu, !quad && (hit >> j & 1u));
    const int n1 = __popc(b[0]), n2 = n1 + __popc(b[1]), n3 = n2 + __popc(b[2]), n4 = n3 + __popc(b[3]);
#pragma unroll 1
    for (int q = 0; 32 * q < n4; ++q) {
      const int t = 32 * q + lane;
      const int j = t < n1 ? 0 : t < n2 ? 1 : t < n3 ? 2 : 3;
      const int first = j == 0 ? 0 : j == 1 ? n1 : j == 2 ? n2 : n3;
      const unsigned bits = j == 0 ? b[0] : j == 1 ? b[1] : j == 2 ? b[2] : b[3];
      const int src = t < n4 ? int(__fns(bits, 0, t - first + 1)) : 0;
      const int ou = __shfl_sync(0xffffffffu, u, src), ov = __shfl_sync(0xffffffffu, vb, src) + j;
      if (t < n4) {
        const Ray r = make_ray(vp, gc, ou, ov);
        own[q] = OwnRay{ou, ov, 0.f, 0.f, dom ? make_float2(r.c0x, r.c0y) : make_float2(r.c0y, r.c0x),
                        dom ? make_float2(r.dcx, r.dcy) : make_float2(r.dcy, r.dcx), r.c0z, r.dcz};
        n_own = q + 1;
      }
    }
  }
  __syncthreads();
  const int mlo = sh.mlo, mhi = sh.mhi;
  int nslab = (mhi >= mlo) ? (mhi - mlo + 1) : 0;
  if (nslab > nsl_max) {
    if (tid == 0) atomicAdd(&flags[0], 1);
    nslab = 0;
  }

  // Box origin (e, z) of every slab in marching order: the tile's four corner
  // rays at the slab's two bounding planes, clamped to the volume's texels.
  const uint32_t box_bytes = uint32_t(BXY * BZ * sizeof(V));
  const uint32_t stage_stride = (box_bytes + 127u) & ~127u;
  int2* const org = reinterpret_cast<int2*>(smem_raw + NS * stage_stride);
  {
    const float ke_ = dom ? gc.kx : gc.ky, be = dom ? gc.bx : gc.by;
    const float kd = dom ? gc.ky : gc.kx, bd = dom ? gc.by : gc.bx;
    const float Se = dom ? vp.Sx : vp.Sy, Sd = dom ? vp.Sy : vp.Sx;
    const int ue = min(u0 + C::TU, gc.W) - 1, ve = min(v0 + C::TV, gc.H) - 1;
    const int ne = dom ? gc.nx : gc.ny;
    const unsigned lanes = 0xffu << (tid & 24);
    for (int q = tid; q < nslab * 8; q += C::threads) {
      const int i = q >> 3, c = q & 7;
      const int m = up ? mlo + i : mhi - i;
      const float plane = float(kSlabBase + m * TS + ((c & 4) ? TS : 0));
      const int ucc = (c & 1) ? ue : u0, vcc = (c & 2) ? ve : v0;
      const float ex = fmaf(float(ucc), vp.Eux, vp.D0x), ey = fmaf(float(ucc), vp.Euy, vp.D0y);
      const float ez = fmaf(float(vcc), vp.Evz, vp.D0z);
      const float de = dom ? ex : ey, dd = dom ? ey : ex;
      const float t = ((plane - bd) / kd - Sd) / dd;
      const float ce = fmaf(fmaf(t, de, Se), ke_, be);
      const float cz = fmaf(t * ez, gc.kz, gc.bz);
      int e0 = min(max(int(floorf(fminf(fmaxf(ce, -1.0e5f), 1.0e5f))), -1), ne - 1), e1 = e0;
      int f0 = min(max(int(floorf(fminf(fmaxf(cz, -1.0e5f), 1.0e5f))), -1), gc.nz - 1), f1 = f0;
#pragma unroll
      for (int x = 1; x < 8; x <<= 1) {
        e0 = min(e0, __shfl_xor_sync(lanes, e0, x));
        e1 = max(e1, __shfl_xor_sync(lanes, e1, x));
        f0 = min(f0, __shfl_xor_sync(lanes, f0, x));
        f1 = max(f1, __shfl_xor_sync(lanes, f1, x));
      }
      if (c == 0) {
        const int oe = (e0 - 1) & ~(int(16 / sizeof(V)) - 1), oz = f0 - 1;
        org[i] = make_int2(oe, oz);
        if (check && (e1 + 2 - oe >= BX || f1 + 2 - oz >= BZ)) atomicAdd(&flags[0], 1);
      }
    }
  }
  __syncthreads();

  auto slab_d = [&](int i) { return kSlabBase + (up ? mlo + i : mhi - i) * TS; };
  auto issue = [&](int i) {
    uint64_t* bar = &sh.bars[i % NS];
    mbar_arrive_expect_tx(bar, box_bytes);
    tma_load_3d(smem_raw + (i % NS) * stage_stride, map, org[i].x, slab_d(i), org[i].y, bar);
  };
  if (tid == 0) {
    for (int i = 0; i < min(NS, nslab); ++i) issue(i);
  }

  int bad = 0, done = 0;
  for (int i = 0; i < nslab; ++i) {
    const int slot = i % NS;
    const bool ok = mbar_wait_bounded(&sh.bars[slot], (i / NS) & 1, gc.wait_limit);
    const V* s = reinterpret_cast<const V*>(smem_raw + slot * stage_stride);
    const int oe = org[i].x, oz = org[i].y, od = slab_d(i);
    const float lo = float(od), hi = lo + float(TS);
    const int org_idx = oe + od * BX + oz * BXY;
    const float cmo = kRoundC - float(org_idx);
    const V* const so = s - org_idx;
    // Samples between two that lie in the box lie in it (coordinates are monotone
    // along a ray; d is inside by the choice of ke): e and z at both ends.  The z
    // margin covers the rounding of the rows between a quad's outer two.
    const float e_lo = float(oe), e_hi = float(oe + BX - 1), z_lo = float(oz) + 0.01f, z_hi = float(oz + BZ - 1) - 0.01f;
    auto inside = [&](float ea, float eb, float zmin, float zmax) {
      return fminf(ea, eb) >= e_lo && fmaxf(ea, eb) < e_hi && zmin >= z_lo && zmax < z_hi;
    };
    if (quad) {
      const float k = kf, ke = slab_end(k, Nf, c0.y, dc.y, up, lo, hi);
      if (ke > k) {
        const float kl = ke - 1.f;
        // rows are equally spaced
        const float za = fmaf(k, dz[0].x, z0[0].x), zb = fmaf(kl, dz[0].x, z0[0].x);
        const float ya = fmaf(k, dz[1].y, z0[1].y), yb = fmaf(kl, dz[1].y, z0[1].y);
        const float sa = ya - za, sb = yb - zb, smin = fminf(sa, sb), smax = fmaxf(sa, sb);
        // (the quad's planes end one above the highest row's)
        const float zmin = fminf(fminf(za, zb), fminf(ya, yb)), zmax = fmaxf(fmaxf(za, zb), fmaxf(ya, yb));
        if (!inside(fmaf(k, dc.x, c0.x), fmaf(kl, dc.x, c0.x), zmin, zmax + 1.f)) {
          bad = 1;
        } else {
          const int cls = zmin >= 0.f ? quad_class(smin, smax) : -1;
          with_form<GATHER>(dom, [&](auto form) {
            constexpr int F = decltype(form)::value;
            switch (cls) {
              case 0: quad_march<V, BX, BY, F, 0, 0, 0>(so, k, ke, c0, dc, z0, dz, acc); break;
              case 1: quad_march<V, BX, BY, F, 0, 0, 1>(so, k, ke, c0, dc, z0, dz, acc); break;
              case 2: quad_march<V, BX, BY, F, 0, 1, 1>(so, k, ke, c0, dc, z0, dz, acc); break;
              case 3: quad_march<V, BX, BY, F, 0, 1, 2>(so, k, ke, c0, dc, z0, dz, acc); break;
              case 4: quad_march<V, BX, BY, F, 1, 2, 3>(so, k, ke, c0, dc, z0, dz, acc); break;
              default: quad_march_any<V, BX, BY, F>(s, k, ke, c0, dc, z0, dz, cmo, acc); break;
            }
          });
        }
      }
      kf = ke;
    }
#pragma unroll 1
    for (int q = 0; q < n_own; ++q) {
      OwnRay& r = own[q];
      const float k = r.k, ke = slab_end(k, Nf, r.c.y, r.d.y, up, lo, hi);
      if (ke > k) {
        const float kl = ke - 1.f, za = fmaf(k, r.dz, r.z0), zb = fmaf(kl, r.dz, r.z0);
        if (!inside(fmaf(k, r.d.x, r.c.x), fmaf(kl, r.d.x, r.c.x), fminf(za, zb), fmaxf(za, zb)))
          bad = 1;
        else
          with_form<GATHER>(dom, [&](auto form) {
            ray_march<V, BX, BY, decltype(form)::value>(s, k, ke, r.c, r.d, r.z0, r.dz, cmo, r.acc);
          });
        r.k = ke;
      }
    }
    // One barrier per slab: every thread is done with the stage before it is
    // refilled, and a wait that gave up anywhere ends the march (samples taken
    // after it stayed inside the box; the status reports them).
    if (__syncthreads_or(!ok)) {
      if (tid == 0) { atomicAdd(&flags[1], 1); sh.abort_flag = 1; }
      break;
    }
    done = i + 1;
    if (tid == 0 && i + NS < nslab) {
      fence_proxy_async();
      issue(i + NS);
    }
  }
  if (sh.abort_flag && tid == 0) {
    // Drain loads still in flight (bounded) before the CTA exits.
    for (int i = done; i < min(done + NS, nslab); ++i)
      if (!mbar_wait_bounded(&sh.bars[i % NS], (i / NS) & 1, kWaitLimit)) sh.abort_flag = 2;
  }
  if (check) {
    // every sample of a hit ray must be consumed
    if (quad && kf != Nf) bad = 1;
    for (int q = 0; q < n_own; ++q)
      if (own[q].k != Nf) bad = 1;
  }
  if (bad) atomicAdd(&flags[0], 1);

  double sq = 0.0;
  const float sum[R] = {acc[0].x, acc[0].y, acc[1].x, acc[1].y};
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int v = vb + j;
    const bool active = u < gc.W && v < gc.H, miss = active && !(hit >> j & 1u);
    const float val = grown_rays(vol, vp, gc, u, v, miss);
    if (quad) sq += fwd_store(o, gc, vp, p, u, v, sum[j] * make_ray(vp, gc, u, v).delta);
    else if (miss) sq += fwd_store(o, gc, vp, p, u, v, val);
  }
#pragma unroll 1
  for (int q = 0; q < n_own; ++q) {
    const OwnRay& r = own[q];
    sq += fwd_store(o, gc, vp, p, r.u, r.v, r.acc * make_ray(vp, gc, r.u, r.v).delta);
  }
  fwd_block_partial(o, sq, sh.red, tid, tile.bid);
}

template <class V, int BX, class C, int MINB, bool GATHER>
__global__ void __launch_bounds__(C::threads, MINB)
    fwd_quad_kernel(const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_t,
                    const V* __restrict__ vol, const ViewParams* __restrict__ views, GridConst gc, int BZ,
                    int nsl_max, int check, FwdOut o, int* flags) {
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 127) & ~uintptr_t(127));
  __shared__ QuadShared<C::NS> sh;
  fwd_quad_body<V, BX, C, GATHER>(&map_v, &map_t, vol, views, gc, BZ, nsl_max, check != 0, o, flags, launch_tile(), smem_raw,
                          sh);
}

// ------------------------------------------------------------------ shapes
template <class V>
using QuadKernel = void (*)(const CUtensorMap, const CUtensorMap, const V*, const ViewParams*, GridConst, int, int, int,
                            FwdOut, int*);

// Shapes, in the order of QuadShape.  The minimum CTAs per SM set the register
// budget (80, 128, 96 and 96 registers).
//  wide : 16 x 32 tiles of 128 threads, slabs of 8 voxels.  Fewest instructions per
//         sample; its boxes fit six CTAs per SM where rows are under 2/3 texel apart.
//  warp : one warp per CTA (8 x 16 rays), slabs of 6.  Twice the box bytes per ray,
//         but no warp waits for another and the last wave is short.
//  thin : 8 x 32 tiles of 64 threads, slabs of 4, for boxes that are large because
//         a detector pixel is about a voxel.
//  skew : 16 x 16 tiles of 64 threads, slabs of 4, for rows a texel or more apart
//         (see QuadCfg).
template <int SHAPE> struct ShapeOf;
template <> struct ShapeOf<kQuadWide> { using C = QuadCfg<16, 8, 8, 8, 1>; static constexpr int minb = 6; };
template <> struct ShapeOf<kQuadWarp> { using C = QuadCfg<8, 4, 8, 6, 1>; static constexpr int minb = 16; };
template <> struct ShapeOf<kQuadThin> { using C = QuadCfg<8, 8, 8, 4, 1>; static constexpr int minb = 10; };
template <> struct ShapeOf<kQuadSkew> { using C = QuadCfg<16, 4, 8, 4, 1, true>; static constexpr int minb = 10; };

// Box widths (elements) per shape and storage size.  fp32: BX * BY is 4, 12, 20 or
// 28 words mod 32, so that the four row groups of a warp, 4p planes apart, fall on
// different banks for most row distances p.
constexpr int kQuadWidths32[kQuadShapes][2] = {{36, 52}, {28, 36}, {28, 36}, {36, 44}};
constexpr int kQuadWidths16[kQuadShapes][2] = {{40, 56}, {40, 56}, {40, 56}, {40, 56}};

template <class V, int BX, int SHAPE, bool GATHER>
QuadKernel<V> quad_kernel_of() {
  return fwd_quad_kernel<V, BX, typename ShapeOf<SHAPE>::C, ShapeOf<SHAPE>::minb, GATHER>;
}

// Calls f(std::integral_constant<int, BX>, std::integral_constant<int, SHAPE>) for
// the compiled shape and width.
template <class V, int SHAPE, class F>
bool with_quad_width(int bx, F&& f) {
  constexpr const int(&w)[2] = sizeof(V) == 4 ? kQuadWidths32[SHAPE] : kQuadWidths16[SHAPE];
  if (bx == w[0]) f(std::integral_constant<int, w[0]>{}, std::integral_constant<int, SHAPE>{});
  else if (bx == w[1]) f(std::integral_constant<int, w[1]>{}, std::integral_constant<int, SHAPE>{});
  else return false;
  return true;
}

// Calls f(std::integral_constant<int, BX>, std::integral_constant<int, SHAPE>) for
// the plan's shape and box width.
template <class V, class F>
void with_quad(const cbct_plan* p, F&& f) {
  const int bx = sizeof(V) == 4 ? p->quad.bx : p->quad16.bx;
  const bool ok = p->quad_shape == kQuadWide   ? with_quad_width<V, kQuadWide>(bx, f)
                  : p->quad_shape == kQuadWarp ? with_quad_width<V, kQuadWarp>(bx, f)
                  : p->quad_shape == kQuadThin ? with_quad_width<V, kQuadThin>(bx, f)
                                               : with_quad_width<V, kQuadSkew>(bx, f);
  if (!ok) throw Error(CBCT_ERR_INTERNAL, "unsupported quad box width");
}

}  // namespace

// The plan's kernel in the gather form (forward_quad_gather.cu, a file of its own to
// compile beside this one).
template <class V>
QuadKernel<V> quad_kernel_gather(const cbct_plan* p);

}  // namespace cbct
