// forward_slab.cuh -- per-ray slab forward projector (device code; instantiated and
// launched by forward_slab.cu): the kernel of launches with too few rays to fill the
// GPU and of detectors whose rows are far apart.
//
// What bounds it.  A launch of one or a few small views fits the GPU at once, so its
// time is that of its slowest warp.  Every ray has N samples, wherever it enters, so
// rays that cut a corner have all of them in a slab or two, and with a barrier per
// slab over a 16x16 tile each slab lasted as long as its slowest ray: corner tiles of
// a one-view call ran two and a half times as long as the middle ones, themselves at
// a third of the issue slots.  Hence
//  * warps do not wait for one another: each has its own small box (8 x 4 rays) and
//    barrier, and goes through its own slabs;
//  * long runs of samples in a slab are dealt over the warp (deal_long_runs), rays
//    along the silhouette four at a time (grown_rays4);
//  * one box per warp: the other warps of the SM cover a warp's wait for its next
//    slab, and two or three boxes only took their places (one 256x192 view into 128^3:
//    45, 46 and 62 us for one, two and three; 8 views of 128x96 into 64^3: 33, 39, 55);
//  * slabs of 8 voxels (slabs of 5: 55 and 35 us), four warps per CTA (1, 2 and 8: 45,
//    45, 60 and 38, 36, 34 us; fewer would need more partial sums);
//  * no index clamp: a slab's samples are checked at their two ends, coordinates being
//    monotone along a ray.
// One 256x192 view into 128^3, whole call: 107 us with 16x16 tiles, 95 once silhouette
// rays were taken by whole warps, 49 now; 8 views of 128x96 into 64^3, the kernel alone:
// 59 us before, 33 now; 32 views of 1.5 mm pixels into 128^3: 0.59 ms before, 0.43 now.
#pragma once

#include "forward_device.cuh"

namespace cbct {

namespace {

// A CTA is four warps on top of one another, each with 8 columns x 4 rows of rays, a
// box and a barrier of its own.  Box rows (the slab's kSlabTS + 1, padded) and widths
// are chosen for the banks; registers are bounded for five CTAs per SM.
constexpr int kSlabWarps = 4, kSlabU = 8, kSlabV = 4 * kSlabWarps, kSlabThreads = 32 * kSlabWarps;
constexpr int kSlabTS = 8, kSlabBoxY = 10, kSlabMinb = 5, kSlabUnroll = 2;

struct SlabShared {
  uint64_t bars[kSlabWarps];
  int abort_flag;
  double red[8];
};

// Four rays at a time: the lanes of a warp in groups of eight, group g on the
// g-th ray of mask m (groups without one repeat the first).  Returns the lane
// that holds the group's ray; rays_done takes the four off the mask, and
// to_owner brings a group's value to the lane that holds its ray.
__device__ __forceinline__ int group_ray(unsigned m) {
  unsigned g = m;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i < int(threadIdx.x >> 3 & 3)) g &= g - 1;
  return __ffs(g ? g : m) - 1;
}
__device__ __forceinline__ unsigned rays_done(unsigned m) {
#pragma unroll
  for (int i = 0; i < 4; ++i) m &= m - 1;
  return m;
}
__device__ __forceinline__ bool to_owner(int src, float group_value, float& value) {
  const int lane = threadIdx.x & 31;
  bool mine = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float x = __shfl_sync(0xffffffffu, group_value, 8 * i);
    if (__shfl_sync(0xffffffffu, src, 8 * i) == lane) {
      value = x;
      mine = true;
    }
  }
  return mine;
}

// Sums of a warp's rays that miss the volume but pass within half a voxel of
// it (their samples read border texels): zero for the other lanes.  All lanes of
// the warp call it; `miss` marks the lanes whose ray (u, v) misses.  The warp
// takes these rays four at a time, lane l of a group sampling k0 + l, k0 + l + 8,
// ... with four samples in flight: one ray per lane leaves a silhouette tile with
// one or two busy lanes for N samples of dependent global loads, and one ray per
// warp pays the load latency once per ray (a tile edge along the silhouette has up
// to 32 of them in one warp: 34k cycles, three quarters of an 8-view 128x96 launch).
// The order of the sum does not depend on the kernel or the tile: 32 partial sums
// of every 32nd sample, added as a tree.
template <class V>
__device__ __forceinline__ float grown_rays4(const V* __restrict__ vol, const ViewParams& vp, const GridConst& gc,
                                            int u, int v, bool miss) {
  constexpr unsigned FULL = 0xffffffffu;
  const int l = threadIdx.x & 7;
  bool need = false;
  int k0 = 0, k1 = -1;
  Ray r{};
  if (miss) {
    r = make_ray(vp, gc, u, v);
    need = grown_range(vp, gc, u, v, r, k0, k1);
  }
  float val = 0.f;
  for (unsigned m = __ballot_sync(FULL, need); m; m = rays_done(m)) {
    const int src = group_ray(m);
    const float cx = __shfl_sync(FULL, r.c0x, src), dx = __shfl_sync(FULL, r.dcx, src);
    const float cy = __shfl_sync(FULL, r.c0y, src), dy = __shfl_sync(FULL, r.dcy, src);
    const float cz = __shfl_sync(FULL, r.c0z, src), dz = __shfl_sync(FULL, r.dcz, src);
    const int last = __shfl_sync(FULL, k1, src);
    float part[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k = __shfl_sync(FULL, k0, src) + l; __any_sync(FULL, k <= last); k += 32) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float kf = float(min(k + 8 * j, last));
        const float x = fetch3_global(vol, gc.nx, gc.ny, gc.nz, fmaf(kf, dx, cx), fmaf(kf, dy, cy), fmaf(kf, dz, cz));
        part[j] += k + 8 * j <= last ? x : 0.f;
      }
    }
    float sum = (part[0] + part[2]) + (part[1] + part[3]);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
    to_owner(src, sum, val);
  }
  return need ? val * r.delta : 0.f;
}

// Long runs.  Every ray takes N samples over its own chord, so a ray that cuts
// an edge or a corner of the volume has most of them in one slab (192 against the
// 11 or so of a ray through the middle), and a lane that took them alone would
// hold up its warp (measured with 16x16 tiles and a barrier per slab: corner tiles
// of a 128^3 one-view call ran 155k cycles, tiles through the middle 58k).
// So rays with more than kLongRun samples in the slab are taken by the whole
// warp, four at a time and 32 samples of each per round, the values added in ray
// order by shuffles: about 270 instructions per round against 50 per sample and
// warp, which pays for up to kDealtRays such rays.  (Raising the bar until no more
// than kDealtRays are left, or taking a round's samples while the last are added,
// gained nothing.)
// All lanes call it; eval(k, c0, dc, z0, dz) is the value of a ray's k-th sample.
constexpr float kLongRun = 24.f;
constexpr int kDealtRays = 16;

template <class Eval>
__device__ __forceinline__ void deal_long_runs(float& k, float ke, float2 c0, float2 dc, float z0, float dz,
                                               float& acc, Eval eval) {
  constexpr unsigned FULL = 0xffffffffu;
  unsigned m = __ballot_sync(FULL, ke - k > kLongRun);
  if (__popc(m) > kDealtRays) return;
  const float l = float(threadIdx.x & 7);
  for (; m; m = rays_done(m)) {
    const int src = group_ray(m);
    const float2 c = make_float2(__shfl_sync(FULL, c0.x, src), __shfl_sync(FULL, c0.y, src));
    const float2 d = make_float2(__shfl_sync(FULL, dc.x, src), __shfl_sync(FULL, dc.y, src));
    const float z = __shfl_sync(FULL, z0, src), zd = __shfl_sync(FULL, dz, src);
    const float qe = __shfl_sync(FULL, ke, src);
    float sum = __shfl_sync(FULL, acc, src);
    for (float q = __shfl_sync(FULL, k, src); __any_sync(FULL, q < qe); q += 32.f) {
      float x[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float kq = q + (l + float(8 * j));
        x[j] = eval(fminf(kq, qe - 1.f), c, d, z, zd);
        x[j] = kq < qe ? x[j] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int t = 0; t < 8; ++t) sum += __shfl_sync(FULL, x[j], t, 8);
    }
    if (to_owner(src, sum, acc)) k = ke;
  }
}

// Samples k .. ke-1 of one ray (all lanes of the warp call it; k == ke: none).
template <class V, int BX, int BY, int FORM>
__device__ __forceinline__ void slab_march(const V* __restrict__ s, float k, float ke, float2 c0, float2 dc, float z0,
                                           float dz, float cmo, float& acc) {
  constexpr int BXY = BX * BY, U = kSlabUnroll;
  auto eval = [&](float q, float2 c, float2 d, float z, float zd) {
    const float2 pq = __ffma2_rn(make_float2(q, q), d, c);
    const float cz = fmaf(q, zd, z);
    const float2 f = floor2_small(pq);
    const float fz = floor_small(cz);
    const float2 t = sub2(pq, f);
    const V* b = s + (unsigned)int_of_biased(fmaf(fz, float(BXY), fmaf(f.y, float(BX), f.x)) + cmo);
    const float2 l = planes2<V, BX, FORM>(b, b + BXY, make_float2(t.x, t.x), make_float2(-t.x, -t.x),
                                    make_float2(t.y, t.y), make_float2(-t.y, -t.y));
    return fmaf(cz - fz, l.y - l.x, l.x);
  };
  deal_long_runs(k, ke, c0, dc, z0, dz, acc, eval);
  for (; k + float(U - 1) < ke; k += float(U)) {
    float v[U];
#pragma unroll
    for (int j = 0; j < U; ++j) v[j] = eval(k + float(j), c0, dc, z0, dz);
#pragma unroll
    for (int j = 0; j < U; ++j) acc += v[j];
  }
  for (; k < ke; k += 1.f) acc += eval(k, c0, dc, z0, dz);
}

// One CTA: ray tile `tile` of the call.  smem_raw is the 128-byte aligned dynamic
// shared memory: per warp a box and the slabs' box origins.  GATHER: the
// gather kernel's interpolation (see LerpForm).
template <class V, int BX, bool GATHER>
__device__ __forceinline__ void fwd_slab_body(const CUtensorMap* map_v, const CUtensorMap* map_t,
                                              const V* __restrict__ vol, const ViewParams* __restrict__ views,
                                              const GridConst& gc, int BZ, int nsl_max, bool check,
                                              const FwdOut& o, int* flags, const TileId& tile,
                                              unsigned char* smem_raw, SlabShared& sh) {
  constexpr int TS = kSlabTS, BY = kSlabBoxY, BXY = BX * BY;
  constexpr unsigned FULL = 0xffffffffu;
  const ViewParams vp = views[tile.z];
  const int dom = vp.dom;
  const bool up = vp.dsgn > 0;
  const CUtensorMap* map = dom ? map_v : map_t;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int u0 = tile.x * kSlabU, v0 = tile.y * kSlabV + 4 * warp;
  const int u = u0 + (lane & 7), v = v0 + (lane >> 3);
  const float Nf = float(gc.N);
  uint64_t* const bar = &sh.bars[warp];
  if (tid == 0) sh.abort_flag = 0;
  if (lane == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  __syncthreads();

  const bool active = u < gc.W && v < gc.H;
  const Ray r = make_ray(vp, gc, min(u, gc.W - 1), min(v, gc.H - 1));
  const bool hit = active && r.a2 > r.a1;
  // Frame coordinates: e = cross axis, d = slab axis (y for dom = 1, x for dom = 0).
  const float2 c0 = dom ? make_float2(r.c0x, r.c0y) : make_float2(r.c0y, r.c0x);
  const float2 dc = dom ? make_float2(r.dcx, r.dcy) : make_float2(r.dcy, r.dcx);
  int mlo = INT_MAX, mhi = INT_MIN;
  if (hit) {
    const int m0 = (max(int(floorf(c0.y)), kSlabBase) - kSlabBase) / TS;
    const int m1 = (max(int(floorf(fmaf(Nf - 1.f, dc.y, c0.y))), kSlabBase) - kSlabBase) / TS;
    mlo = min(m0, m1);
    mhi = max(m0, m1);
  }
  mlo = __reduce_min_sync(FULL, mlo);
  mhi = __reduce_max_sync(FULL, mhi);
  int nslab = (mhi >= mlo) ? (mhi - mlo + 1) : 0;
  if (nslab > nsl_max) {
    if (lane == 0) atomicAdd(&flags[0], 1);
    nslab = 0;
  }

  // Box origin (e, z) of every slab in marching order: the warp's four corner
  // rays at the slab's two bounding planes, clamped to the volume's texels.
  const uint32_t box_bytes = uint32_t(BXY * BZ * sizeof(V));
  const uint32_t box_stride = (box_bytes + 127u) & ~127u;
  unsigned char* const box = smem_raw + warp * (box_stride + ((uint32_t(nsl_max) * sizeof(int2) + 127u) & ~127u));
  int2* const org = reinterpret_cast<int2*>(box + box_stride);
  {
    const float ke_ = dom ? gc.kx : gc.ky, be = dom ? gc.bx : gc.by;
    const float kd = dom ? gc.ky : gc.kx, bd = dom ? gc.by : gc.bx;
    const float Se = dom ? vp.Sx : vp.Sy, Sd = dom ? vp.Sy : vp.Sx;
    const int ue = min(u0 + kSlabU, gc.W) - 1, ve = min(v0 + 4, gc.H) - 1;
    const int ne = dom ? gc.nx : gc.ny;
    const unsigned lanes = 0xffu << (lane & 24);
    for (int q = lane; q < nslab * 8; q += 32) {
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
  __syncwarp();

  auto slab_d = [&](int i) { return kSlabBase + (up ? mlo + i : mhi - i) * TS; };
  auto issue = [&](int i) {
    mbar_arrive_expect_tx(bar, box_bytes);
    tma_load_3d(box, map, org[i].x, slab_d(i), org[i].y, bar);
  };
  if (lane == 0 && nslab > 0) issue(0);

  const V* const s = reinterpret_cast<const V*>(box);
  float acc = 0.f, kf = 0.f;
  int bad = 0;
  for (int i = 0; i < nslab; ++i) {
    if (!__all_sync(FULL, mbar_wait_bounded(bar, i & 1, gc.wait_limit))) {
      if (lane == 0) {
        // The load in flight lands (bounded) before the warp leaves.
        atomicAdd(&flags[1], 1);
        atomicMax(&sh.abort_flag, mbar_wait_bounded(bar, i & 1, kWaitLimit) ? 1 : 2);
      }
      break;
    }
    const int oe = org[i].x, oz = org[i].y, od = slab_d(i);
    const float lo = float(od), hi = lo + float(TS);
    const float ke = hit ? slab_end(kf, Nf, c0.y, dc.y, up, lo, hi) : kf;
    bool run = ke > kf;
    if (run) {
      // Samples between two that lie in the box lie in it (coordinates are monotone
      // along a ray; d is inside by the choice of ke): e and z at both ends.
      const float kl = ke - 1.f;
      const float ea = fmaf(kf, dc.x, c0.x), eb = fmaf(kl, dc.x, c0.x);
      const float za = fmaf(kf, r.dcz, r.c0z), zb = fmaf(kl, r.dcz, r.c0z);
      run = fminf(ea, eb) >= float(oe) && fmaxf(ea, eb) < float(oe + BX - 1) && fminf(za, zb) >= float(oz) &&
            fmaxf(za, zb) < float(oz + BZ - 1);
      bad |= !run;
    }
    const float cmo = kRoundC - float(oe + od * BX + oz * BXY);
    with_form<GATHER>(dom, [&](auto form) {
      slab_march<V, BX, BY, decltype(form)::value>(s, run ? kf : ke, ke, c0, dc, r.c0z, r.dcz, cmo, acc);
    });
    kf = ke;
    __syncwarp();
    if (lane == 0 && i + 1 < nslab) {
      fence_proxy_async();
      issue(i + 1);
    }
  }
  if (check && hit && kf != Nf) bad = 1;  // every sample of a hit ray must be consumed
  if (bad) atomicAdd(&flags[0], 1);

  const float grown = grown_rays4(vol, vp, gc, u, v, active && !hit);
  const float val = hit ? acc * r.delta : grown;
  fwd_epilogue(o, gc, vp, tile.z, u, v, active, val, sh.red, tid, tile.bid);
}

template <class V, int BX, bool GATHER>
__global__ void __launch_bounds__(kSlabThreads, kSlabMinb)
    fwd_slab_kernel(const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_t,
                    const V* __restrict__ vol, const ViewParams* __restrict__ views, GridConst gc, int BZ,
                    int nsl_max, int check, FwdOut o, int* flags) {
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 127) & ~uintptr_t(127));
  __shared__ SlabShared sh;
  fwd_slab_body<V, BX, GATHER>(&map_v, &map_t, vol, views, gc, BZ, nsl_max, check != 0, o, flags, launch_tile(),
                       smem_raw, sh);
}

}  // namespace

}  // namespace cbct
