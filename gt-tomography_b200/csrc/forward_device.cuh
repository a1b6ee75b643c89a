// forward_device.cuh -- device code shared by the forward projectors: outputs
// and epilogues, bounds-checked marching, packed lerps and the per-ray samples
// of one slab box.
#pragma once

#include <climits>
#include <type_traits>

#include "device_common.cuh"

namespace cbct {

enum { kModeStore = 0, kModeResidual = 1, kModeRecip = 2 };

struct FwdOut {
  float* out;            // projections of the subset (W,H,P_s)
  const void* b;         // measured projections (residual mode; NULL reads as 0)
  int b_dtype;           // storage type of b (cbct_dtype)
  const float* pw;       // per-pixel weight (residual mode; nullable)
  float scale;           // residual scale
  int mode;
  int apply_offset;      // residual mode: multiply by the sin^2 Wang weight
  int accumulate;        // store mode: out += result
  double* partials;      // residual mode: per-block sum of squares (nullable)
  const float* wproj;    // projection weights of the subset (CBSubsetWeightOperator; nullable)
};

// Tile of one CTA: detector tile (x, y) of view z of the call, and its index
// among the call's tiles in launch order (its partial-sum slot).
struct TileId {
  int x, y, z;
  size_t bid;
};

namespace {

// Sample range of a ray restricted to the box grown by half a voxel: samples
// outside it touch only border texels and add exactly 0.  Returns false when
// no sample can contribute.
__device__ __forceinline__ bool grown_range(const ViewParams& vp, const GridConst& gc, int u, int v,
                                            const Ray& r, int& k0, int& k1) {
  const float dx = fmaf(float(u), vp.Eux, vp.D0x);
  const float dy = fmaf(float(u), vp.Euy, vp.D0y);
  const float dz = fmaf(float(v), vp.Evz, vp.D0z);
  const float gx = gc.hx + 0.5005f * gc.vx, gy = gc.hy + 0.5005f * gc.vy, gz = gc.hz + 0.5005f * gc.vz;
  const float tx1 = __fdiv_rn(gx - vp.Sx, dx), tx2 = __fdiv_rn(-gx - vp.Sx, dx);
  const float ty1 = __fdiv_rn(gy - vp.Sy, dy), ty2 = __fdiv_rn(-gy - vp.Sy, dy);
  const float tz1 = __fdiv_rn(gz, dz), tz2 = __fdiv_rn(-gz, dz);
  const float tl = fmaxf(fmaxf(fminf(tx1, tx2), fminf(ty1, ty2)), fminf(tz1, tz2));
  const float th = fminf(fminf(fmaxf(tx1, tx2), fmaxf(ty1, ty2)), fmaxf(tz1, tz2));
  const float ta = fminf(r.a1, r.a2), tb = fmaxf(r.a1, r.a2);
  if (!(tl <= th) || th < ta || tl > tb) return false;
  const float f = (r.a2 - r.a1) * gc.invN;
  if (f == 0.f) { k0 = 0; k1 = gc.N - 1; return true; }
  const float q1 = (tl - r.a1) / f, q2 = (th - r.a1) / f;
  const float lo = fmaxf(fminf(q1, q2) - 1.f, 0.f);
  const float hi = fminf(fmaxf(q1, q2) + 1.f, float(gc.N - 1));
  k0 = int(floorf(lo));
  k1 = int(ceilf(hi));
  return k0 <= k1;
}

template <class V>
__device__ __forceinline__ float march_global(const V* __restrict__ vol, const GridConst& gc,
                                              const Ray& r, int k0, int k1) {
  float acc = 0.f;
  for (int k = k0; k <= k1; ++k) {
    const float kf = float(k);
    acc += fetch3_global(vol, gc.nx, gc.ny, gc.nz, fmaf(kf, r.dcx, r.c0x), fmaf(kf, r.dcy, r.c0y),
                         fmaf(kf, r.dcz, r.c0z));
  }
  return acc;
}

// Sums of a warp's rays that miss the volume but pass within half a voxel of
// it (their samples read border texels): zero for the other lanes.  All lanes of
// the warp call it; `miss` marks the lanes whose ray (u, v) misses.  The warp
// takes these rays one after another, lane l sampling k0 + l, k0 + l + 32, ...:
// one ray per lane leaves a silhouette tile with one or two busy lanes for N
// samples of dependent global loads (most of the time of a one-view call).
// The sum does not depend on which kernel or tile the ray belongs to.  (Four rays at a
// time, as the slab kernel takes them, cost the pair and quad kernels registers: 180 views
// of 256x192 into 128^3 2.42 to 2.56 ms.)
template <class V>
__device__ __forceinline__ float grown_rays(const V* __restrict__ vol, const ViewParams& vp, const GridConst& gc,
                                            int u, int v, bool miss) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = (threadIdx.x + threadIdx.y * blockDim.x) & 31;
  bool need = false;
  if (miss) {
    int k0, k1;
    need = grown_range(vp, gc, u, v, make_ray(vp, gc, u, v), k0, k1);
  }
  float val = 0.f;
  for (unsigned m = __ballot_sync(FULL, need); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    const int uu = __shfl_sync(FULL, u, src), vv = __shfl_sync(FULL, v, src);
    const Ray r = make_ray(vp, gc, uu, vv);
    int k0 = 0, k1 = -1;
    grown_range(vp, gc, uu, vv, r, k0, k1);
    float acc = 0.f;
    for (int k = k0 + lane; k <= k1; k += 32) {
      const float kf = float(k);
      acc += fetch3_global(vol, gc.nx, gc.ny, gc.nz, fmaf(kf, r.dcx, r.c0x), fmaf(kf, r.dcy, r.c0y),
                           fmaf(kf, r.dcz, r.c0z));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
    if (lane == src) val = acc * r.delta;
  }
  return val;
}

// Output of one ray (store, reciprocal or weighted residual); returns the
// squared residual (residual mode) for the block's partial sum.
__device__ __forceinline__ double fwd_store(const FwdOut& o, const GridConst& gc, const ViewParams& vp, int p,
                                            int u, int v, float val) {
  double sq = 0.0;
  const size_t idx = ((size_t)p * gc.H + v) * gc.W + u;
  // CBSubsetWeightOperator: mult_M multiplies the projection by w, and mult_MH
  // of the residual weights its input by w again (CBSubsetWeightOperator.h:32-49).
  const float wp = o.wproj ? o.wproj[idx] : 1.f;
  val *= wp;
  if (o.mode == kModeStore) {
    o.out[idx] = o.accumulate ? o.out[idx] + val : val;
  } else if (o.mode == kModeRecip) {
    o.out[idx] = 1.f / fmaxf(val, 1e-6f);
  } else {
    const float d = o.b ? val - ld_any(o.b, idx, o.b_dtype) : val;
    sq = double(d) * double(d);
    float w = o.scale * wp;
    if (o.pw) w *= o.pw[idx];
    if (o.apply_offset) w *= offset_weight_full(gc.fov_u, gc.W, u, vp.ox);
    o.out[idx] = d * w;
  }
  return sq;
}

// Index of a CTA of a one-scan launch in launch order (x fastest).
__device__ __forceinline__ size_t launch_block_id() {
  return ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
}

__device__ __forceinline__ TileId launch_tile() {
  return TileId{int(blockIdx.x), int(blockIdx.y), int(blockIdx.z), launch_block_id()};
}

// Deterministic block sum of sq; one partial per block in launch order.
__device__ __forceinline__ void fwd_block_partial(const FwdOut& o, double sq, double* sh_red, int tid,
                                                  size_t bid) {
  if (o.partials != nullptr) {
    double t = warp_sum(sq);
    const int w = tid >> 5, l = tid & 31;
    if (l == 0) sh_red[w] = t;
    __syncthreads();
    if (tid < 32) {
      double q = (l < (int)(blockDim.x * blockDim.y) / 32) ? sh_red[l] : 0.0;
      q = warp_sum(q);
      if (tid == 0) o.partials[bid] = q;
    }
  }
}

// Epilogue shared by the per-ray variants.  All threads of the block must call it.
__device__ __forceinline__ void fwd_epilogue(const FwdOut& o, const GridConst& gc, const ViewParams& vp,
                                             int p, int u, int v, bool active, float val,
                                             double* sh_red, int tid, size_t bid) {
  const double sq = active ? fwd_store(o, gc, vp, p, u, v, val) : 0.0;
  fwd_block_partial(o, sq, sh_red, tid, bid);
}

// Packed lerp of two pairs: a + t (b - a) as (a - t a) + t b.
__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float2 t) {
  const float2 nt = make_float2(-t.x, -t.y);
  return __ffma2_rn(t, b, __ffma2_rn(nt, a, a));
}

// Samples of one ray inside one slab.  (ce, cd, cz) are frame texel
// coordinates; the box origin is (oe, od, oz); BX and BY are the box
// strides.  Consumes samples while floor(cd) stays inside the slab.
template <class V, int BX, int BY = kBoxY>
struct SlabSample {
  static constexpr int BXY = BX * BY;
  // Trilinear value of one sample whose frame coordinates are (ced.x, ced.y, cz)
  // and whose floors are (fe, fd, fz).  cmo = 1.5 * 2^23 - (box origin index):
  // the element index comes out of the mantissa of an exact sum.
  static __device__ __forceinline__ float eval(const V* __restrict__ s, float2 ced, float cz, float fe, float fd,
                                               float fz, float cmo, unsigned maxidx, int& bad, bool check) {
    const float2 aed = __fadd2_rn(ced, make_float2(-fe, -fd));
    const float az = cz - fz;
    const int idx0 = int_of_biased(fmaf(fz, float(BXY), fmaf(fd, float(BX), fe)) + cmo);
    if (check) bad |= (unsigned)idx0 > maxidx;
    const unsigned idx = min((unsigned)idx0, maxidx);
    const V* q = s + idx;
    const float2 a0 = make_float2(sm_f(q[0]), sm_f(q[BX]));              // (e0,d0,z0) (e0,d1,z0)
    const float2 b0 = make_float2(sm_f(q[1]), sm_f(q[BX + 1]));          // (e1,d0,z0) (e1,d1,z0)
    const float2 a1 = make_float2(sm_f(q[BXY]), sm_f(q[BXY + BX]));      // z1
    const float2 b1 = make_float2(sm_f(q[BXY + 1]), sm_f(q[BXY + BX + 1]));
    const float2 te = make_float2(aed.x, aed.x);
    const float2 e0 = lerp2(a0, b0, te);   // z0: (d0, d1)
    const float2 e1 = lerp2(a1, b1, te);   // z1: (d0, d1)
    const float2 dz = lerp2(make_float2(e0.x, e1.x), make_float2(e0.y, e1.y), make_float2(aed.y, aed.y));
    return fmaf(az, dz.y - dz.x, dz.x);
  }
};

// Samples of one ray inside one slab.  The number of samples the slab holds
// is found first (the first k whose d coordinate leaves the slab; d is
// monotone along the ray), then they are taken in a counted loop, kFwdUnroll
// independent evaluations per iteration, added to acc in ray order.
// (ce, cd, cz) are frame texel coordinates.
constexpr int kFwdUnroll = 2;

template <class V, int BX, int SGN, bool CHECK, int BY = kBoxY>
__device__ __forceinline__ void slab_samples(const V* __restrict__ s, float& kf, float Nf, float ce0, float cd0,
                                             float cz0, float dce, float dcd, float idcd, float dcz, float lo,
                                             float hi, float cmo, unsigned maxidx, float& acc, int& bad) {
  using SS = SlabSample<V, BX, BY>;
  const float2 c0 = make_float2(ce0, cd0), dc = make_float2(dce, dcd);
  // floor(x) >= hi <=> x >= hi and floor(x) < lo <=> x < lo, lo and hi being integers.
  auto out_at = [&](float k) {
    const float x = fmaf(k, dcd, cd0);
    return SGN > 0 ? (x >= hi) : (x < lo);
  };
  // Estimate (idcd = 1 / dcd), then the exact boundary: out_at is monotone in k.
  float ke = ceilf(((SGN > 0 ? hi : lo) - cd0) * idcd);
  ke = fminf(fmaxf(ke, kf), Nf);
  while (ke > kf && out_at(ke - 1.f)) ke -= 1.f;
  while (ke < Nf && !out_at(ke)) ke += 1.f;
  float k = kf;
  for (; k + float(kFwdUnroll - 1) < ke; k += float(kFwdUnroll)) {
    float v[kFwdUnroll];
#pragma unroll
    for (int q = 0; q < kFwdUnroll; ++q) {
      const float kq = k + float(q);
      const float2 pq = __ffma2_rn(make_float2(kq, kq), dc, c0);
      const float czq = fmaf(kq, dcz, cz0);
      v[q] = SS::eval(s, pq, czq, floor_small(pq.x), floor_small(pq.y), floor_small(czq), cmo, maxidx, bad, CHECK);
    }
#pragma unroll
    for (int q = 0; q < kFwdUnroll; ++q) acc += v[q];
  }
  for (; k < ke; k += 1.f) {
    const float2 pq = __ffma2_rn(make_float2(k, k), dc, c0);
    const float czq = fmaf(k, dcz, cz0);
    acc += SS::eval(s, pq, czq, floor_small(pq.x), floor_small(pq.y), floor_small(czq), cmo, maxidx, bad, CHECK);
  }
  kf = ke;
}

// First sample of a ray past the slab [lo, hi), at least k: an estimate, then
// the exact test (monotone in k; floor(x) >= hi <=> x >= hi and floor(x) < lo <=>
// x < lo, lo and hi being integers).
__device__ __forceinline__ float slab_end(float k, float Nf, float cd0, float dcd, bool up, float lo, float hi) {
  auto out_at = [&](float q) {
    const float x = fmaf(q, dcd, cd0);
    return up ? (x >= hi) : (x < lo);
  };
  float ke = ceilf(__fdividef((up ? hi : lo) - cd0, dcd));
  ke = fminf(fmaxf(ke, k), Nf);
  while (ke > k && out_at(ke - 1.f)) ke -= 1.f;
  while (ke < Nf && !out_at(ke)) ke += 1.f;
  return ke;
}

__device__ __forceinline__ float2 floor2_small(float2 x) {
  const float2 c = make_float2(kRoundC, kRoundC);
  return __fadd2_rn(__fadd2_rd(x, c), make_float2(-kRoundC, -kRoundC));
}

// a - b (one rounding, as the scalar difference).
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }

// Form of the in-plane interpolation.  kLerpFrame: along e, then d, a lerp as
// (a - t a) + t b.  kLerpXisE and kLerpXisD: the gather kernel's, along x, then y, a lerp
// as a + t (b - a), in views whose x is the frame's e or d; launches that the gather
// kernel could take as well use these (forward_lerp_gather), so that rays through the
// volume are its rays.  Along z all are a + t (b - a).
enum LerpForm { kLerpFrame = 0, kLerpXisE = 1, kLerpXisD = 2 };

// Calls f(std::integral_constant<int, LerpForm>) for a view's form.  Kernels branch on the
// view around their sample loops.  (A body per order was 4 % better at 36 views of 511x383
// from 255x253x251 voxels, 2.74 against 2.86 ms, and 3 % worse at 40 views of 301x211 from
// 150x141x93, 1.07 against 1.03; strides known at run time 3.00 and 1.00; the frame form,
// whose results differ from the gather kernel's in rounding, 2.71 and 0.97.)
template <bool GATHER, class F>
__device__ __forceinline__ void with_form(int dom, F&& f) {
  if constexpr (!GATHER) f(std::integral_constant<int, kLerpFrame>{});
  else if (dom) f(std::integral_constant<int, kLerpXisE>{});
  else f(std::integral_constant<int, kLerpXisD>{});
}

// a + t (b - a), packed.
__device__ __forceinline__ float2 lerp2_gather(float2 a, float2 b, float2 t) {
  return __ffma2_rn(t, __fadd2_rn(b, make_float2(-a.x, -a.y)), a);
}

// In-plane interpolation at q0 and q1, two planes packed.
template <class V, int BX, int FORM>
__device__ __forceinline__ float2 planes2(const V* __restrict__ q0, const V* __restrict__ q1, float2 te, float2 nte,
                                          float2 td, float2 ntd) {
  const float2 a = make_float2(sm_f(q0[0]), sm_f(q1[0])), b = make_float2(sm_f(q0[1]), sm_f(q1[1]));
  const float2 c = make_float2(sm_f(q0[BX]), sm_f(q1[BX])), d = make_float2(sm_f(q0[BX + 1]), sm_f(q1[BX + 1]));
  if (FORM == kLerpXisE) return lerp2_gather(lerp2_gather(a, b, te), lerp2_gather(c, d, te), td);
  if (FORM == kLerpXisD) return lerp2_gather(lerp2_gather(a, c, td), lerp2_gather(b, d, td), te);
  const float2 x = __ffma2_rn(te, b, __ffma2_rn(nte, a, a));
  const float2 y = __ffma2_rn(te, d, __ffma2_rn(nte, c, c));
  return __ffma2_rn(td, y, __ffma2_rn(ntd, x, x));
}

}  // namespace

}  // namespace cbct
