// forward.cu -- cone-beam forward projector (mult_M) for sm_100a.
//
// Semantics: conebeam_forwards_projection_kernel (xray/conebeam_projection.cu:412-528):
// one ray per detector pixel from the source to the pixel centre, clipped to
// the volume box, N = (int)(spp*nx) equidistant samples from the entry point,
// trilinear interpolation with border 0, result scaled by the sample spacing.
// Interpolation here is FP32 in software (not 9-bit texture weights).
//
// Variants (all but the gather kernel give bitwise equal results over aligned rows):
//  * fwd_slab_kernel (forward_slab.cuh): one thread per ray.  A warp marches a tile of
//    rays of one view through the volume in slabs of a few voxels along the view's
//    dominant in-plane axis.  Each slab's footprint (the box around the tile's ray
//    pyramid) is staged into shared memory by a 3-D TMA load; out-of-volume texels
//    arrive as zeros (the border rule for free).  Views whose rays run mostly along x
//    read an x/y-transposed copy of the volume, so every slab is a range of
//    memory rows and the box is never padded along its slab axis.  Samples are
//    taken in ray order, so each ray's sum has the reference's summation
//    order.  Pairs of lerps run as packed FP32 (FFMA2).
//  * fwd_pair_kernel: the same slabs, but one thread marches two vertically
//    adjacent rays of a detector column that share their in-plane sample
//    positions, interpolating them in e and d once.
//  * fwd_quad_kernel (forward_quad.cuh): four such rays per thread; the kernel of
//    launches that fill the GPU (quad_choose and launch_variant have the rules).
//  * fwd_fan_kernel (opt-in): the in-plane sharing across a whole column,
//    through shared-memory lines.
//  * fwd_gather_kernel: bounds-checked global loads, used when the geometry does not fit
//    the slab boxes or the volume's start is not TMA-aligned.  Volumes whose rows are not
//    a multiple of 16 bytes take the slab and quad kernels on row-padded copies, in the
//    gather kernel's form of interpolation (LerpForm): it took those launches before, and
//    an FP64 residual norm shows the difference of the forms.
#include <climits>
#include <cmath>
#include <cstring>

#include "forward_host.h"

namespace cbct {

namespace {

// ------------------------------------------------------------------ gather
template <class V>
__global__ void __launch_bounds__(256) fwd_gather_kernel(const V* __restrict__ vol,
                                                         const ViewParams* __restrict__ views,
                                                         GridConst gc, FwdOut o) {
  __shared__ double sh_red[8];
  const int tid = threadIdx.x;
  const int u = blockIdx.x * kTU + (tid % kTU);
  const int v = blockIdx.y * kTV + (tid / kTU);
  const int p = blockIdx.z;
  const ViewParams vp = views[p];
  const bool active = (u < gc.W) && (v < gc.H);
  float val = 0.f;
  if (active) {
    const Ray r = make_ray(vp, gc, u, v);
    int k0, k1;
    if (grown_range(vp, gc, u, v, r, k0, k1)) val = march_global(vol, gc, r, k0, k1) * r.delta;
  }
  fwd_epilogue(o, gc, vp, p, u, v, active, val, sh_red, tid, launch_block_id());
}

// ------------------------------------------------------------------ transpose
// volT[k][i][j] = vol[k][j][i]: the volume seen with x and y exchanged, rows
// pitchT elements apart.  With volP, also a copy of the volume whose rows are
// pitchP apart (TMA needs rows of a multiple of 16 bytes).
//
// What bounds it: HBM, given enough loads in flight.  A CTA of 256 threads takes a 32x32
// tile of four planes, sixteen loads per thread before the first is waited for (256^3
// fp32, 134 MB: 40 us with one plane per CTA, 28 with four).
constexpr int kCopyPlanes = 4;

template <class V>
__global__ void __launch_bounds__(256) volume_copies_kernel(const V* __restrict__ in, V* __restrict__ volT, int pitchT,
                                                            V* __restrict__ volP, int pitchP, int nx, int ny, int nz) {
  __shared__ V tile[kCopyPlanes][32][33];
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32, z0 = blockIdx.z * kCopyPlanes;
  const int x = x0 + threadIdx.x;
  V v[kCopyPlanes][4];
#pragma unroll
  for (int k = 0; k < kCopyPlanes; ++k)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int y = y0 + threadIdx.y + 8 * i, z = z0 + k;
      if (x < nx && y < ny && z < nz) v[k][i] = in[((size_t)z * ny + y) * nx + x];
    }
#pragma unroll
  for (int k = 0; k < kCopyPlanes; ++k)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = threadIdx.y + 8 * i, y = y0 + j, z = z0 + k;
      if (x < nx && y < ny && z < nz) {
        tile[k][j][threadIdx.x] = v[k][i];
        if (volP) volP[((size_t)z * ny + y) * pitchP + x] = v[k][i];
      }
    }
  if (!volT) return;
  __syncthreads();
  const int yt = y0 + threadIdx.x;
#pragma unroll
  for (int k = 0; k < kCopyPlanes; ++k)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = threadIdx.y + 8 * i, xt = x0 + j, z = z0 + k;
      if (xt < nx && yt < ny && z < nz) volT[((size_t)z * nx + xt) * pitchT + yt] = tile[k][threadIdx.x][j];
    }
}

// The same for 16-bit volumes with an even row length and a 4-byte aligned start: a
// CTA takes a 64x64 tile of two planes in words of two elements, so that each row of
// a tile is 128 bytes (512^3 bf16, 537 MB: 274 us element by element, 101 so).  Even
// and odd rows lie apart in shared memory, rows 33 words apart: a thread's two words
// (rows 2t, 2t + 1, columns 2c, 2c + 1) are on banks t + c, and two byte permutes make
// them the words of the output rows 2c and 2c + 1.
__global__ void __launch_bounds__(256) volume_copies16_kernel(const uint32_t* __restrict__ in, uint16_t* __restrict__ volT,
                                                              int pitchT, uint32_t* __restrict__ volP, int pitchP,
                                                              int nx, int ny, int nz) {
  constexpr int KZ = 2;
  __shared__ uint32_t tile[KZ][2][32][33];
  const int x0 = blockIdx.x * 64, y0 = blockIdx.y * 64, z0 = blockIdx.z * KZ;
  const int xw = x0 / 2 + threadIdx.x, nw = nx / 2;
  uint32_t v[KZ][8];
#pragma unroll
  for (int k = 0; k < KZ; ++k)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int y = y0 + threadIdx.y + 8 * i, z = z0 + k;
      v[k][i] = xw < nw && y < ny && z < nz ? in[((size_t)z * ny + y) * nw + xw] : 0u;
    }
#pragma unroll
  for (int k = 0; k < KZ; ++k)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int j = threadIdx.y + 8 * i, y = y0 + j, z = z0 + k;
      tile[k][j & 1][j >> 1][threadIdx.x] = v[k][i];
      if (volP && xw < nw && y < ny && z < nz) volP[((size_t)z * ny + y) * (pitchP / 2) + xw] = v[k][i];
    }
  if (!volT) return;
  __syncthreads();
  const int yt = y0 + 2 * threadIdx.x;
#pragma unroll
  for (int k = 0; k < KZ; ++k)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = threadIdx.y + 8 * i, xt = x0 + 2 * c, z = z0 + k;
      if (xt >= nx || yt >= ny || z >= nz) continue;
      const uint32_t w0 = tile[k][0][threadIdx.x][c], w1 = tile[k][1][threadIdx.x][c];
      uint16_t* const q = volT + ((size_t)z * nx + xt) * pitchT + yt;
      if (yt + 1 < ny) {
        *reinterpret_cast<uint32_t*>(q) = __byte_perm(w0, w1, 0x5410);
        *reinterpret_cast<uint32_t*>(q + pitchT) = __byte_perm(w0, w1, 0x7632);
      } else {
        q[0] = uint16_t(w0);
        q[pitchT] = uint16_t(w0 >> 16);
      }
    }
}

// x/y transposes of many scans' volumes in one launch: one CTA per 32x32 tile
// of one plane of one scan, scans numbered in order.
struct TransposeRec {
  const float* in;
  float* out;
  int nx, ny;
  int tx, ty;            // tiles per plane (x, y)
  int base;              // index of the scan's first CTA
};

__global__ void transpose_multi_kernel(const TransposeRec* __restrict__ recs, int n_recs) {
  __shared__ float tile[32][33];
  int lo = 0, hi = n_recs - 1;
  const int t = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (recs[mid].base <= t) lo = mid;
    else hi = mid - 1;
  }
  const TransposeRec& R = recs[lo];
  int l = t - R.base;
  const int x0 = l % R.tx * 32;
  l /= R.tx;
  const int y0 = l % R.ty * 32;
  const size_t plane = (size_t)(l / R.ty) * ((size_t)R.nx * R.ny);
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int x = x0 + threadIdx.x, y = y0 + j;
    if (x < R.nx && y < R.ny) tile[j][threadIdx.x] = R.in[plane + (size_t)y * R.nx + x];
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int y = y0 + threadIdx.x, x = x0 + j;
    if (x < R.nx && y < R.ny) R.out[plane + (size_t)x * R.ny + y] = tile[threadIdx.x][j];
  }
}

// ------------------------------------------------------------------ row pairs
// Two vertically adjacent rays of one detector column lie in the column's
// vertical plane.  When both leave the volume through its side faces their
// clip (a1, a2) is the column's, so their k-th samples share the in-plane
// position (e_k, d_k) and differ only in z; when in addition their z
// coordinates differ by less than one texel at every sample (checked at both
// ends; the difference is linear in k), the lower ray's planes fz, fz + 1 and
// the upper ray's planes are among fz, fz + 1, fz + 2.  One thread then marches
// the pair: one e/d position, three planes interpolated in e and d (12 shared
// loads instead of 16), and each ray's own z lerp.  Every value is the one the
// slab kernel computes for that ray (same texels, same operations, same
// order), so results are bitwise equal.  Other pairs (rays clipped by the top
// or bottom face, or far apart in z) run slab_samples for each ray.
// The row-pair kernel keeps one TMA stage: with 16x16 tiles its box is small
// enough for six CTAs per SM, and the other CTAs' work covers each CTA's wait
// for its next slab (two stages would halve the CTAs per SM).
#ifndef CBCT_PAIR_STAGES
#define CBCT_PAIR_STAGES 1
#endif
constexpr int kPairStages = CBCT_PAIR_STAGES;
// Rows of a row-pair box (the slab's kTS + 1 rows, padded to kBoxY by default).
#ifndef CBCT_PAIR_BOXY
#define CBCT_PAIR_BOXY 10
#endif
constexpr int kPairBoxY = CBCT_PAIR_BOXY;

struct PairShared {
  uint64_t bars[kPairStages];
  int mlo, mhi, abort_flag;
  double red[8];
};

// One sample of a paired ray: (lower ray's value, upper ray's value).
template <class V, int BX, bool CHECK, int BY = kBoxY>
__device__ __forceinline__ float2 pair_eval(const V* __restrict__ s, float k, float2 c0, float2 dc, float zl0,
                                            float dzl, float zu0, float dzu, float cmo, unsigned maxidx,
                                            unsigned maxidx3, int& bad) {
  constexpr int BXY = BX * BY;
  const float2 pq = __ffma2_rn(make_float2(k, k), dc, c0);
  const float czl = fmaf(k, dzl, zl0), czu = fmaf(k, dzu, zu0);
  const float fe = floor_small(pq.x), fd = floor_small(pq.y), fzl = floor_small(czl), fzu = floor_small(czu);
  const float2 aed = __fadd2_rn(pq, make_float2(-fe, -fd));
  const int idx0 = int_of_biased(fmaf(fzl, float(BXY), fmaf(fd, float(BX), fe)) + cmo);
  const bool up = fzu != fzl;
  if (CHECK) bad |= ((unsigned)idx0 > maxidx) | (up && (unsigned)idx0 + 2u * BXY > maxidx3) | (fzu - fzl > 1.f);
  const V* q = s + min((unsigned)idx0, maxidx);
  const V* q2 = s + min((unsigned)idx0 + 2u * BXY, maxidx3);
  const float2 te = make_float2(aed.x, aed.x);
  const float2 e0 = lerp2(make_float2(sm_f(q[0]), sm_f(q[BX])), make_float2(sm_f(q[1]), sm_f(q[BX + 1])), te);
  const float2 e1 = lerp2(make_float2(sm_f(q[BXY]), sm_f(q[BXY + BX])),
                          make_float2(sm_f(q[BXY + 1]), sm_f(q[BXY + BX + 1])), te);
  const float2 e2 = lerp2(make_float2(sm_f(q2[0]), sm_f(q2[BX])), make_float2(sm_f(q2[1]), sm_f(q2[BX + 1])), te);
  // d lerps of planes fz, fz + 1 (packed) and fz + 2: the slab kernel's formula
  const float2 d01 = lerp2(make_float2(e0.x, e1.x), make_float2(e0.y, e1.y), make_float2(aed.y, aed.y));
  const float d2 = fmaf(aed.y, e2.y, fmaf(-aed.y, e2.x, e2.x));
  const float bl = up ? d01.y : d01.x, bh = up ? d2 : d01.y;
  return make_float2(fmaf(czl - fzl, d01.y - d01.x, d01.x), fmaf(czu - fzu, bh - bl, bl));
}

#ifndef CBCT_PAIR_UNROLL
#define CBCT_PAIR_UNROLL 1
#endif
constexpr int kPairUnroll = CBCT_PAIR_UNROLL;

// The pair's samples inside one slab (counted as in slab_samples), each ray's
// values added in ray order.
template <class V, int BX, int SGN, bool CHECK, int BY = kBoxY>
__device__ __forceinline__ void pair_samples(const V* __restrict__ s, float& kf, float Nf, float ce0, float cd0,
                                             float dce, float dcd, float idcd, float zl0, float dzl, float zu0,
                                             float dzu, float lo, float hi, float cmo, unsigned maxidx,
                                             unsigned maxidx3, float& accl, float& accu, int& bad) {
  const float2 c0 = make_float2(ce0, cd0), dc = make_float2(dce, dcd);
  auto out_at = [&](float k) {
    const float x = fmaf(k, dcd, cd0);
    return SGN > 0 ? (x >= hi) : (x < lo);
  };
  float ke = ceilf(((SGN > 0 ? hi : lo) - cd0) * idcd);
  ke = fminf(fmaxf(ke, kf), Nf);
  while (ke > kf && out_at(ke - 1.f)) ke -= 1.f;
  while (ke < Nf && !out_at(ke)) ke += 1.f;
  float k = kf;
  if (kPairUnroll > 1) {
    for (; k + float(kPairUnroll - 1) < ke; k += float(kPairUnroll)) {
      float2 v[kPairUnroll];
#pragma unroll
      for (int q = 0; q < kPairUnroll; ++q)
        v[q] = pair_eval<V, BX, CHECK, BY>(s, k + float(q), c0, dc, zl0, dzl, zu0, dzu, cmo, maxidx, maxidx3, bad);
#pragma unroll
      for (int q = 0; q < kPairUnroll; ++q) {
        accl += v[q].x;
        accu += v[q].y;
      }
    }
  }
  for (; k < ke; k += 1.f) {
    const float2 v = pair_eval<V, BX, CHECK, BY>(s, k, c0, dc, zl0, dzl, zu0, dzu, cmo, maxidx, maxidx3, bad);
    accl += v.x;
    accu += v.y;
  }
  kf = ke;
}

// CTAs per SM the register budget is sized for: 80 registers (no spills) at
// six 128-thread CTAs, as many as the fp32 boxes of 16x16 tiles leave room for.
template <class V>
constexpr int pair_min_blocks() {
#ifdef CBCT_PAIR_MINB
  return CBCT_PAIR_MINB;
#else
  return kPairThreads >= 256 ? 3 : 6;
#endif
}

// One CTA of the row-pair kernel (see fwd_slab_body).
template <class V, int BX, bool CHECK>
__device__ __forceinline__ void fwd_pair_body(const CUtensorMap* map_v, const CUtensorMap* map_t,
                                              const V* __restrict__ vol, const ViewParams* __restrict__ views,
                                              const GridConst& gc, int BZ, int nsl_max, const FwdOut& o,
                                              int* flags, const TileId& tile, unsigned char* smem_raw,
                                              PairShared& sh) {
  constexpr int BXY = BX * kPairBoxY;
  const ViewParams vp = views[tile.z];
  const int dom = vp.dom;
  const CUtensorMap* map = dom ? map_v : map_t;
  const int tid = threadIdx.x;
  const int p = tile.z;
  const int u0 = tile.x * kPU, v0 = tile.y * kPV;
  const int u = u0 + (tid % kPU), va = v0 + 2 * (tid / kPU), vb = va + 1;
  const bool act_a = (u < gc.W) && (va < gc.H), act_b = (u < gc.W) && (vb < gc.H);
  const int uc = min(u, gc.W - 1);
  const Ray ra = make_ray(vp, gc, uc, min(va, gc.H - 1));
  const Ray rb = make_ray(vp, gc, uc, min(vb, gc.H - 1));
  const bool hit_a = act_a && (ra.a2 > ra.a1), hit_b = act_b && (rb.a2 > rb.a1);
  const float ke_ = dom ? gc.kx : gc.ky, be = dom ? gc.bx : gc.by;
  const float kd = dom ? gc.ky : gc.kx, bd = dom ? gc.by : gc.bx;
  const float Se = dom ? vp.Sx : vp.Sy, Sd = dom ? vp.Sy : vp.Sx;
  // Frame coordinates (e = cross axis, d = slab axis) of both rays.
  const float ce0a = dom ? ra.c0x : ra.c0y, dcea = dom ? ra.dcx : ra.dcy;
  const float cd0a = dom ? ra.c0y : ra.c0x, dcda = dom ? ra.dcy : ra.dcx;
  const float ce0b = dom ? rb.c0x : rb.c0y, dceb = dom ? rb.dcx : rb.dcy;
  const float cd0b = dom ? rb.c0y : rb.c0x, dcdb = dom ? rb.dcy : rb.dcx;
  const float idcda = 1.f / dcda, idcdb = 1.f / dcdb;
  const float Nf = float(gc.N);
  // Pairing: same clip, z difference in (0, 1) texel at both ends (the lower
  // ray first).  The margins cover the rounding of the sample coordinates.
  bool paired = false, a_low = true;
  if (hit_a && hit_b && ra.a1 == rb.a1 && ra.a2 == rb.a2) {
    const float d0 = rb.c0z - ra.c0z;
    const float d1 = fmaf(Nf - 1.f, rb.dcz, rb.c0z) - fmaf(Nf - 1.f, ra.dcz, ra.c0z);
    const bool ab = d0 >= 2e-3f && d0 <= 0.998f && d1 >= 2e-3f && d1 <= 0.998f;
    const bool ba = d0 <= -2e-3f && d0 >= -0.998f && d1 <= -2e-3f && d1 >= -0.998f;
    paired = ab || ba;
    a_low = ab;
  }
  const float zl0 = a_low ? ra.c0z : rb.c0z, dzl = a_low ? ra.dcz : rb.dcz;
  const float zu0 = a_low ? rb.c0z : ra.c0z, dzu = a_low ? rb.dcz : ra.dcz;

  if (tid == 0) {
    sh.mlo = INT_MAX;
    sh.mhi = INT_MIN;
    sh.abort_flag = 0;
    for (int s = 0; s < kPairStages; ++s) mbar_init(&sh.bars[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  {
    int mn = INT_MAX, mx = INT_MIN;
    if (hit_a) {
      const int m0 = (max(int(floorf(cd0a)), kSlabBase) - kSlabBase) / kTS;
      const int m1 = (max(int(floorf(fmaf(Nf - 1.f, dcda, cd0a))), kSlabBase) - kSlabBase) / kTS;
      mn = min(m0, m1);
      mx = max(m0, m1);
    }
    if (hit_b) {
      const int m0 = (max(int(floorf(cd0b)), kSlabBase) - kSlabBase) / kTS;
      const int m1 = (max(int(floorf(fmaf(Nf - 1.f, dcdb, cd0b))), kSlabBase) - kSlabBase) / kTS;
      mn = min(mn, min(m0, m1));
      mx = max(mx, max(m0, m1));
    }
    if (mn <= mx) {
      atomicMin(&sh.mlo, mn);
      atomicMax(&sh.mhi, mx);
    }
  }
  __syncthreads();
  const int mlo = sh.mlo, mhi = sh.mhi;
  int nslab = (mhi >= mlo) ? (mhi - mlo + 1) : 0;
  if (nslab > nsl_max) {
    if (tid == 0) atomicAdd(&flags[0], 1);
    nslab = 0;
  }
  // Per-slab footprints (e min, e max, z min, z max) after the boxes.
  const uint32_t box_bytes = uint32_t(BX * kPairBoxY * BZ * sizeof(V));
  const uint32_t stage_stride = (box_bytes + 127u) & ~127u;
  int* const emin = reinterpret_cast<int*>(smem_raw + kPairStages * stage_stride);
  int* const emax = emin + nsl_max;
  int* const zmin = emax + nsl_max;
  int* const zmax = zmin + nsl_max;
  for (int i = tid; i < nslab; i += blockDim.x) {
    emin[i] = INT_MAX; emax[i] = INT_MIN;
    zmin[i] = INT_MAX; zmax[i] = INT_MIN;
  }
  __syncthreads();
  // Footprint of every slab: the tile's four corner rays at the slab's two
  // bounding planes, clamped to the volume's texel range.
  const int ue = min(u0 + kPU, gc.W) - 1, ve = min(v0 + kPV, gc.H) - 1;
  const int ne = dom ? gc.nx : gc.ny;
  for (int q = tid; q < nslab * 8; q += blockDim.x) {
    const int i = q >> 3, c = q & 7;
    const int m = mlo + i;
    const float plane = float(kSlabBase + m * kTS + ((c & 4) ? kTS : 0));
    const int ucc = (c & 1) ? ue : u0, vcc = (c & 2) ? ve : v0;
    const float dx = fmaf(float(ucc), vp.Eux, vp.D0x);
    const float dy = fmaf(float(ucc), vp.Euy, vp.D0y);
    const float dz = fmaf(float(vcc), vp.Evz, vp.D0z);
    const float de = dom ? dx : dy, dd = dom ? dy : dx;
    const float t = ((plane - bd) / kd - Sd) / dd;
    const float ce = fmaf(fmaf(t, de, Se), ke_, be);
    const float cz = fmaf(t * dz, gc.kz, gc.bz);
    const int fe = min(max(int(floorf(fminf(fmaxf(ce, -1.0e5f), 1.0e5f))), -1), ne - 1);
    const int fz = min(max(int(floorf(fminf(fmaxf(cz, -1.0e5f), 1.0e5f))), -1), gc.nz - 1);
    atomicMin(&emin[i], fe);
    atomicMax(&emax[i], fe);
    atomicMin(&zmin[i], fz);
    atomicMax(&zmax[i], fz);
  }
  __syncthreads();

  const unsigned maxidx = unsigned(BXY * (BZ - 1) - BX - 2);   // two-plane loads stay in the box
  const unsigned maxidx3 = unsigned(BXY * BZ - BX - 2);        // the third plane's loads
  auto origin = [&](int i, int& oe, int& od, int& oz, int& m) {
    m = (vp.dsgn > 0) ? mlo + i : mhi - i;
    const int ii = m - mlo;
    oe = (emin[ii] - 1) & ~(int(16 / sizeof(V)) - 1);   // 16-byte aligned x start
    od = kSlabBase + m * kTS;
    oz = zmin[ii] - 1;
  };
  auto issue = [&](int i) {
    int oe, od, oz, m;
    origin(i, oe, od, oz, m);
    uint64_t* bar = &sh.bars[i % kPairStages];
    mbar_arrive_expect_tx(bar, box_bytes);
    tma_load_3d(smem_raw + (i % kPairStages) * stage_stride, map, oe, od, oz, bar);
  };
  if (tid == 0) {
    for (int i = 0; i < min(kPairStages, nslab); ++i) issue(i);
  }

  float acca = 0.f, accb = 0.f;   // paired: lower / upper ray
  float kfa = 0.f, kfb = 0.f;     // paired: kfa is the pair's next sample
  int bad = 0;
  int done = 0;
  for (int i = 0; i < nslab; ++i) {
    const int slot = i % kPairStages;
    const bool ok = mbar_wait_bounded(&sh.bars[slot], (i / kPairStages) & 1, gc.wait_limit);
    if (__syncthreads_or(!ok)) {
      if (tid == 0) { atomicAdd(&flags[1], 1); sh.abort_flag = 1; }
      break;
    }
    done = i + 1;
    int oe, od, oz, m;
    origin(i, oe, od, oz, m);
    if (CHECK && tid == 0) {
      const int ii = m - mlo;
      if (emax[ii] + 2 - oe >= BX || zmax[ii] + 2 - oz >= BZ) atomicAdd(&flags[0], 1);
    }
    const V* s = reinterpret_cast<const V*>(smem_raw + slot * stage_stride);
    const float lo = float(od), hi = lo + float(kTS);
    const float cmo = kRoundC - float(oe + od * BX + oz * BXY);
    constexpr int PY = kPairBoxY;
    if (paired) {
      if (vp.dsgn > 0)
        pair_samples<V, BX, 1, CHECK, PY>(s, kfa, Nf, ce0a, cd0a, dcea, dcda, idcda, zl0, dzl, zu0, dzu, lo, hi,
                                          cmo, maxidx, maxidx3, acca, accb, bad);
      else
        pair_samples<V, BX, -1, CHECK, PY>(s, kfa, Nf, ce0a, cd0a, dcea, dcda, idcda, zl0, dzl, zu0, dzu, lo, hi,
                                           cmo, maxidx, maxidx3, acca, accb, bad);
    } else {
      if (hit_a) {
        if (vp.dsgn > 0)
          slab_samples<V, BX, 1, CHECK, PY>(s, kfa, Nf, ce0a, cd0a, ra.c0z, dcea, dcda, idcda, ra.dcz, lo, hi, cmo,
                                            maxidx, acca, bad);
        else
          slab_samples<V, BX, -1, CHECK, PY>(s, kfa, Nf, ce0a, cd0a, ra.c0z, dcea, dcda, idcda, ra.dcz, lo, hi, cmo,
                                             maxidx, acca, bad);
      }
      if (hit_b) {
        if (vp.dsgn > 0)
          slab_samples<V, BX, 1, CHECK, PY>(s, kfb, Nf, ce0b, cd0b, rb.c0z, dceb, dcdb, idcdb, rb.dcz, lo, hi, cmo,
                                            maxidx, accb, bad);
        else
          slab_samples<V, BX, -1, CHECK, PY>(s, kfb, Nf, ce0b, cd0b, rb.c0z, dceb, dcdb, idcdb, rb.dcz, lo, hi, cmo,
                                             maxidx, accb, bad);
      }
    }
    __syncthreads();
    if (tid == 0 && i + kPairStages < nslab) {
      fence_proxy_async();
      issue(i + kPairStages);
    }
  }
  if (sh.abort_flag && tid == 0) {
    for (int i = done; i < min(done + kPairStages, nslab); ++i)
      if (!mbar_wait_bounded(&sh.bars[i % kPairStages], (i / kPairStages) & 1, kWaitLimit)) sh.abort_flag = 2;
  }
  if (CHECK) {
    // every sample of a hit ray must be consumed
    if (paired ? kfa != Nf : ((hit_a && kfa != Nf) || (hit_b && kfb != Nf))) bad = 1;
    if (bad) atomicAdd(&flags[0], 1);
  }
  float vala = 0.f, valb = 0.f;
  if (paired) {
    vala = (a_low ? acca : accb) * ra.delta;
    valb = (a_low ? accb : acca) * rb.delta;
  } else {
    if (hit_a) vala = acca * ra.delta;
    if (hit_b) valb = accb * rb.delta;
  }
  const float grown_a = grown_rays(vol, vp, gc, u, va, act_a && !hit_a);
  const float grown_b = grown_rays(vol, vp, gc, u, vb, act_b && !hit_b);
  if (!hit_a) vala = grown_a;
  if (!hit_b) valb = grown_b;
  double sq = 0.0;
  if (act_a) sq += fwd_store(o, gc, vp, p, u, va, vala);
  if (act_b) sq += fwd_store(o, gc, vp, p, u, vb, valb);
  fwd_block_partial(o, sq, sh.red, tid, tile.bid);
}

template <class V, int BX, bool CHECK>
__global__ void __launch_bounds__(kPairThreads, pair_min_blocks<V>())
    fwd_pair_kernel(const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_t,
                    const V* __restrict__ vol, const ViewParams* __restrict__ views, GridConst gc, int BZ,
                    int nsl_max, FwdOut o, int* flags) {
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 127) & ~uintptr_t(127));
  __shared__ PairShared sh;
  fwd_pair_body<V, BX, CHECK>(&map_v, &map_t, vol, views, gc, BZ, nsl_max, o, flags, launch_tile(), smem_raw, sh);
}

// ------------------------------------------------------------------ fan
// The rays of one detector column lie in one vertical plane (the detector's
// v axis is the world z axis).  A ray that enters and leaves the volume
// through its side faces has the clip (a1, a2) of the column's in-plane path,
// so its k-th sample sits at the column's k-th in-plane position (e_k, d_k);
// only z differs between the rows.  The fan kernel gives each warp one column
// of a kFU x kFV tile (lane = detector row).  Per slab, the warp first
// interpolates the column's samples in e and d on every z plane its rays
// reach ("lines", one value per sample and plane), then every ray takes its
// samples as linear interpolations in z between two line entries.  This is
// the slab kernel's trilinear tree (e, then d, then z) with the e/d part
// shared by the column's rays, so results are bitwise those of the per-ray
// kernels.  Rays clipped by the top or bottom face (their own a1/a2) take the
// per-ray trilinear path on the same box.
struct FanShared {
  uint64_t bars[kNStage];
  int mlo, mhi, abort_flag;
  double red[8];
  float tile[kFV][kFU + 1];  // results, transposed for a coalesced epilogue
};

// The column's samples inside one slab, in chunks of kFKC (warp-level; every
// lane of the warp calls it).  kcol: the column's next sample (warp-uniform).
template <class V, int BX, int SGN, bool CHECK>
__device__ __forceinline__ void fan_slab(const V* __restrict__ s, float* __restrict__ lines, int LZ, int BZ,
                                         int lane, int N, int& kcol, float2 c0, float2 dc, bool shared, float c0z,
                                         float dcz, float lo, float hi, int oz, float orgf, float& acc, int& bad) {
  constexpr int BXY = BX * kBoxY;
  constexpr unsigned FULL = 0xffffffffu;
  const unsigned maxidx = unsigned(BXY * BZ - BX - 2);
  auto outside = [&](float fd) { return SGN > 0 ? (fd >= hi) : (fd < lo); };
  for (;;) {
    if (kcol >= N) return;
    // Samples of the chunk still inside the slab (a prefix, floor(d) being
    // monotone along the ray).
    bool in = false;
    if (lane < kFKC && kcol + lane < N) {
      const float kj = float(kcol + lane);
      in = !outside(floorf(fmaf(kj, dc.y, c0.y)));
    }
    const int nk = __ffs(~__ballot_sync(FULL, in)) - 1;
    if (nk <= 0) return;
    // z planes the shared rays reach over the chunk.
    int zl = INT_MAX, zh = INT_MIN;
    if (shared) {
      const int fa = int(floorf(fmaf(float(kcol), dcz, c0z)));
      const int fb = int(floorf(fmaf(float(kcol + nk - 1), dcz, c0z)));
      zl = min(fa, fb);
      zh = max(fa, fb);
    }
    zl = __reduce_min_sync(FULL, zl);
    zh = __reduce_max_sync(FULL, zh);
    int nz = zh - zl + 2;
    if (CHECK && (nz > LZ || zl < oz || zh + 1 >= oz + BZ)) bad = 1;
    nz = min(nz, LZ);
    // Lines: lane (j, g) interpolates sample j on planes g, g + G, ...
    const int G = 32 / nk;
    const int j = lane % nk, g = lane / nk;
    if (g < G) {
      const float kfj = float(kcol + j);
      const float2 pa = __ffma2_rn(make_float2(kfj, kfj), dc, c0);
      const float fe = floor_small(pa.x), fd = floor_small(pa.y);
      const float2 aed = __fadd2_rn(pa, make_float2(-fe, -fd));
      const float2 te = make_float2(aed.x, aed.x);
      const float td = aed.y;
      int idx = int(fmaf(float(zl + g), float(BXY), fmaf(fd, float(BX), fe)) - orgf);
      float* L = lines + j * LZ;
      for (int z = g; z < nz; z += G, idx += G * BXY) {
        if (CHECK) bad |= (unsigned)idx > maxidx;
        const V* q = s + min((unsigned)idx, maxidx);
        const float2 a0 = make_float2(sm_f(q[0]), sm_f(q[BX]));
        const float2 b0 = make_float2(sm_f(q[1]), sm_f(q[BX + 1]));
        const float2 e = lerp2(a0, b0, te);  // (d0, d1) rows on plane z
        L[z] = fmaf(td, e.y, fmaf(-td, e.x, e.x));
      }
    }
    __syncwarp();
    if (shared) {
      const float* L = lines;
      for (int jj = 0; jj < nk; ++jj, L += LZ) {
        const float cz = fmaf(float(kcol + jj), dcz, c0z);
        const float fz = floor_small(cz);
        const float az = cz - fz;
        int iz = int(fz) - zl;
        if (CHECK) bad |= (unsigned)iz > (unsigned)(nz - 2);
        iz = min(max(iz, 0), nz - 2);
        acc += fmaf(az, L[iz + 1] - L[iz], L[iz]);
      }
    }
    kcol += nk;
    __syncwarp();
    if (nk < kFKC) return;
  }
}

template <class V, int BX, bool CHECK>
__global__ void __launch_bounds__(256, 3) fwd_fan_kernel(const __grid_constant__ CUtensorMap map_v,
                                                      const __grid_constant__ CUtensorMap map_t,
                                                      const V* __restrict__ vol,
                                                      const ViewParams* __restrict__ views, GridConst gc,
                                                      int BZ, int LZ, int nsl_max, FwdOut o, int* flags) {
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  __shared__ FanShared sh;
  unsigned char* smem_raw =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 127) & ~uintptr_t(127));
  constexpr int BXY = BX * kBoxY;
  const ViewParams vp = views[blockIdx.z];
  const int dom = vp.dom;
  const CUtensorMap* map = dom ? &map_v : &map_t;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int p = blockIdx.z;
  const int u0 = blockIdx.x * kFU, v0 = blockIdx.y * kFV;
  const int u = u0 + warp, v = v0 + lane;
  const bool active = (u < gc.W) && (v < gc.H);
  const int uc = min(u, gc.W - 1);
  const Ray r = make_ray(vp, gc, uc, min(v, gc.H - 1));
  const bool hit = active && (r.a2 > r.a1);
  // The column's in-plane clip: make_ray's without the z faces.
  const float dx = fmaf(float(uc), vp.Eux, vp.D0x);
  const float dy = fmaf(float(uc), vp.Euy, vp.D0y);
  const float tx1 = __fdiv_rn(gc.hx - vp.Sx, dx), tx2 = __fdiv_rn(-gc.hx - vp.Sx, dx);
  const float ty1 = __fdiv_rn(gc.hy - vp.Sy, dy), ty2 = __fdiv_rn(-gc.hy - vp.Sy, dy);
  const float a1c = fmaxf(fmaxf(fminf(tx1, tx2), fminf(ty1, ty2)), 0.f);
  const float a2c = fminf(fminf(fmaxf(tx1, tx2), fmaxf(ty1, ty2)), 1.f);
  const bool shared = hit && r.a1 == a1c && r.a2 == a2c;
  const bool own = hit && !shared;
  const bool any_shared = __any_sync(0xffffffffu, shared);
  // Frame coordinates (e = cross axis, d = slab axis) of this lane's ray; for
  // shared rays they are the column's.
  const float ce0 = dom ? r.c0x : r.c0y, dce = dom ? r.dcx : r.dcy;
  const float cd0 = dom ? r.c0y : r.c0x, dcd = dom ? r.dcy : r.dcx;
  const float idcd = 1.f / dcd;
  // The column's frame coordinates, from the first shared lane.
  const int src = any_shared ? __ffs(__ballot_sync(0xffffffffu, shared)) - 1 : 0;
  const float2 cc0 = make_float2(__shfl_sync(0xffffffffu, ce0, src), __shfl_sync(0xffffffffu, cd0, src));
  const float2 cdc = make_float2(__shfl_sync(0xffffffffu, dce, src), __shfl_sync(0xffffffffu, dcd, src));

  if (tid == 0) {
    sh.mlo = INT_MAX;
    sh.mhi = INT_MIN;
    sh.abort_flag = 0;
    for (int s = 0; s < kNStage; ++s) mbar_init(&sh.bars[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (hit) {
    const int f0 = int(floorf(cd0));
    const int f1 = int(floorf(fmaf(float(gc.N - 1), dcd, cd0)));
    const int m0 = (max(f0, kSlabBase) - kSlabBase) / kTS;
    const int m1 = (max(f1, kSlabBase) - kSlabBase) / kTS;
    atomicMin(&sh.mlo, min(m0, m1));
    atomicMax(&sh.mhi, max(m0, m1));
  }
  __syncthreads();
  const int mlo = sh.mlo, mhi = sh.mhi;
  int nslab = (mhi >= mlo) ? (mhi - mlo + 1) : 0;
  if (nslab > nsl_max) {
    if (tid == 0) atomicAdd(&flags[0], 1);
    nslab = 0;
  }
  // Per-slab footprints (e min, e max, z min, z max) live after the lines.
  const uint32_t box_bytes = uint32_t(BX * kBoxY * BZ * sizeof(V));
  const uint32_t stage_stride = (box_bytes + 127u) & ~127u;
  int* foot = reinterpret_cast<int*>(smem_raw + kNStage * stage_stride + (size_t)kFU * kFKC * LZ * sizeof(float));
  const float ke = dom ? gc.kx : gc.ky, be = dom ? gc.bx : gc.by;
  const float kd = dom ? gc.ky : gc.kx, bd = dom ? gc.by : gc.bx;
  const float Se = dom ? vp.Sx : vp.Sy, Sd = dom ? vp.Sy : vp.Sx;
  for (int i = tid; i < nslab; i += blockDim.x) {
    foot[i] = INT_MAX; foot[nsl_max + i] = INT_MIN;
    foot[2 * nsl_max + i] = INT_MAX; foot[3 * nsl_max + i] = INT_MIN;
  }
  __syncthreads();
  // Footprint of every slab: the four corner rays of the tile at the slab's
  // two bounding planes.
  const int ue = min(u0 + kFU, gc.W) - 1, ve = min(v0 + kFV, gc.H) - 1;
  const int ne = dom ? gc.nx : gc.ny;  // volume extent along e
  for (int q = tid; q < nslab * 8; q += blockDim.x) {
    const int i = q >> 3, c = q & 7;
    const int m = mlo + i;
    const float plane = float(kSlabBase + m * kTS + ((c & 4) ? kTS : 0));
    const int ucc = (c & 1) ? ue : u0, vcc = (c & 2) ? ve : v0;
    const float ddx = fmaf(float(ucc), vp.Eux, vp.D0x);
    const float ddy = fmaf(float(ucc), vp.Euy, vp.D0y);
    const float ddz = fmaf(float(vcc), vp.Evz, vp.D0z);
    const float de = dom ? ddx : ddy, dd = dom ? ddy : ddx;
    const float t = ((plane - bd) / kd - Sd) / dd;
    float ce = fmaf(fmaf(t, de, Se), ke, be);
    float cz = fmaf(t * ddz, gc.kz, gc.bz);
    // Samples lie inside the volume (texel floors in [-1, n-1]; outside it the
    // border reads 0), so the box only has to cover the footprint's part in it.
    const int fe = min(max(int(floorf(fminf(fmaxf(ce, -1.0e5f), 1.0e5f))), -1), ne - 1);
    const int fz = min(max(int(floorf(fminf(fmaxf(cz, -1.0e5f), 1.0e5f))), -1), gc.nz - 1);
    atomicMin(&foot[i], fe);
    atomicMax(&foot[nsl_max + i], fe);
    atomicMin(&foot[2 * nsl_max + i], fz);
    atomicMax(&foot[3 * nsl_max + i], fz);
  }
  __syncthreads();

  const unsigned maxidx = unsigned(BXY * (BZ - 1) - BX - 2);
  float* lines = reinterpret_cast<float*>(smem_raw + kNStage * stage_stride) + warp * (kFKC * LZ);
  auto origin = [&](int i, int& oe, int& od, int& oz, int& m) {
    m = (vp.dsgn > 0) ? mlo + i : mhi - i;
    const int ii = m - mlo;
    oe = (foot[ii] - 1) & ~(int(16 / sizeof(V)) - 1);
    od = kSlabBase + m * kTS;
    oz = foot[2 * nsl_max + ii] - 1;
  };
  auto issue = [&](int i) {
    int oe, od, oz, m;
    origin(i, oe, od, oz, m);
    uint64_t* bar = &sh.bars[i % kNStage];
    mbar_arrive_expect_tx(bar, box_bytes);
    tma_load_3d(smem_raw + (i % kNStage) * stage_stride, map, oe, od, oz, bar);
  };
  if (tid == 0) {
    for (int i = 0; i < min(kNStage, nslab); ++i) issue(i);
  }

  float acc = 0.f;
  float kf = 0.f;   // own rays: next sample
  int kcol = 0;     // the column's next sample
  const float Nf = float(gc.N);
  int bad = 0;
  int done = 0;
  for (int i = 0; i < nslab; ++i) {
    const int slot = i % kNStage;
    const bool ok = mbar_wait_bounded(&sh.bars[slot], (i / kNStage) & 1, gc.wait_limit);
    if (__syncthreads_or(!ok)) {
      if (tid == 0) { atomicAdd(&flags[1], 1); sh.abort_flag = 1; }
      break;
    }
    done = i + 1;
    int oe, od, oz, m;
    origin(i, oe, od, oz, m);
    if (CHECK && tid == 0) {
      const int ii = m - mlo;
      if (foot[nsl_max + ii] + 2 - oe >= BX || foot[3 * nsl_max + ii] + 2 - oz >= BZ) atomicAdd(&flags[0], 1);
    }
    const V* s = reinterpret_cast<const V*>(smem_raw + slot * stage_stride);
    const float lo = float(od), hi = lo + float(kTS);
    const float orgf = float(oe + od * BX + oz * BXY);
    if (any_shared) {
      if (vp.dsgn > 0)
        fan_slab<V, BX, 1, CHECK>(s, lines, LZ, BZ, lane, gc.N, kcol, cc0, cdc, shared, r.c0z, r.dcz, lo, hi, oz,
                                  orgf, acc, bad);
      else
        fan_slab<V, BX, -1, CHECK>(s, lines, LZ, BZ, lane, gc.N, kcol, cc0, cdc, shared, r.c0z, r.dcz, lo, hi, oz,
                                   orgf, acc, bad);
    }
    if (own) {
      const float cmo = kRoundC - orgf;
      if (vp.dsgn > 0)
        slab_samples<V, BX, 1, CHECK>(s, kf, Nf, ce0, cd0, r.c0z, dce, dcd, idcd, r.dcz, lo, hi, cmo, maxidx, acc,
                                        bad);
      else
        slab_samples<V, BX, -1, CHECK>(s, kf, Nf, ce0, cd0, r.c0z, dce, dcd, idcd, r.dcz, lo, hi, cmo, maxidx, acc,
                                         bad);
    }
    __syncthreads();
    if (tid == 0 && i + kNStage < nslab) {
      fence_proxy_async();
      issue(i + kNStage);
    }
  }
  if (sh.abort_flag && tid == 0) {
    for (int i = done; i < min(done + kNStage, nslab); ++i)
      (void)mbar_wait_bounded(&sh.bars[i % kNStage], (i / kNStage) & 1, kWaitLimit);
  }
  if (CHECK && !sh.abort_flag) {
    if ((shared && kcol != gc.N) || (own && kf != Nf)) bad = 1;  // every sample of a hit ray is consumed
    if (bad) atomicAdd(&flags[0], 1);
  }

  const float grown = grown_rays(vol, vp, gc, u, v, active && !hit);
  const float val = hit ? acc * r.delta : grown;
  // Transpose through shared memory so that the epilogue's accesses run along u.
  sh.tile[lane][warp] = val;
  __syncthreads();
  const int tu = tid % kFU, tv = tid / kFU;
  const int eu = u0 + tu, ev = v0 + tv;
  fwd_epilogue(o, gc, vp, p, eu, ev, eu < gc.W && ev < gc.H, sh.tile[tv][tu], sh.red, tid, launch_block_id());
}

// ------------------------------------------------------------------ host
CUtensorMapDataType tma_dtype(cbct_dtype dt) {
  switch (dt) {
    case CBCT_F32: return CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    case CBCT_F16: return CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    default: return CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  }
}

// ------------------------------------------------------------------ work list
// Work-list (persistent) forward projector over many scans: resident CTAs
// take items -- one ray tile of one view of one scan -- from an atomic counter
// until the list is empty and run the one-scan kernel's body on them, so every
// ray gets the arithmetic of its own launch.  A scan's items are numbered in
// its one-scan launch order (x fastest), which is also its partial-sum slot.
template <int BX>
__global__ void __launch_bounds__(kPairThreads, pair_min_blocks<float>())
    fwd_multi_kernel(const FwdScanRec* __restrict__ recs, int n_recs, int total, int* __restrict__ counter) {
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 127) & ~uintptr_t(127));
  __shared__ PairShared sh;
  __shared__ int item;
  __shared__ int base[kMultiMaxRecs];
  for (int i = threadIdx.x; i < n_recs; i += blockDim.x) base[i] = recs[i].base;
  int last = -1;
  for (;;) {
    if (threadIdx.x == 0) item = atomicAdd(counter, 1);
    __syncthreads();
    const int t = item;
    if (t >= total) break;
    // Broadcast: the compiler may then keep the record's fields uniform.
    const int lo = __shfl_sync(0xffffffffu, find_rec(base, n_recs, t), 0);
    const FwdScanRec& R = recs[lo];
    int l = t - base[lo];
    TileId tile;
    tile.bid = (size_t)l;
    tile.x = l % R.tx;
    l /= R.tx;
    tile.y = l % R.ty;
    tile.z = l / R.ty;
    if (threadIdx.x == 0 && lo != last) {   // the thread that issues the TMA loads
      tensormap_acquire(&R.map_v);
      tensormap_acquire(&R.map_t);
      last = lo;
    }
    fwd_pair_body<float, BX, false>(&R.map_v, &R.map_t, static_cast<const float*>(R.vol), R.views, R.gc, R.BZ,
                                    R.nsl_max, R.o, R.flags, tile, smem_raw, sh);
    __syncthreads();
    // A wait that gave up is counted in the scan's flag word and its loads
    // drained; only a CTA whose drain also gave up (a copy may still land in
    // its shared memory) stops taking items.
    const bool ok = sh.abort_flag != 2;
    if (threadIdx.x == 0) {
      for (int i = 0; i < kPairStages; ++i) mbar_inval(&sh.bars[i]);
    }
    if (!ok) break;
  }
}

}  // namespace

CUtensorMap make_volume_map(cbct_dtype dt, const void* vol, int n0, int n1, int n2, const SlabBox& b) {
  CUtensorMap m;
  std::memset(&m, 0, sizeof(m));
  const size_t es = dtype_size(dt);
  cuuint64_t dims[3] = {(cuuint64_t)n0, (cuuint64_t)n1, (cuuint64_t)n2};
  const cuuint64_t pitch = (cuuint64_t)tma_pitch(n0, es) * es;
  cuuint64_t strides[2] = {pitch, pitch * n1};
  cuuint32_t box[3] = {(cuuint32_t)b.bx, (cuuint32_t)b.by, (cuuint32_t)b.bz};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult res = tensor_map_encoder()(&m, tma_dtype(dt), 3, const_cast<void*>(vol), dims, strides, box, estr,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (res != CUDA_SUCCESS)
    throw Error(CBCT_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)res));
  return m;
}

namespace {

// Dynamic shared memory of a fan launch: kNStage TMA stages of the
// box (128-byte aligned) + the fan kernel's lines + alignment slack.
static size_t forward_smem(const SlabBox& b, size_t es, int lz, int nsl = 0) {
  return kNStage * ((b.bx * b.by * b.bz * es + 127) & ~size_t(127)) + (size_t)kFU * kFKC * lz * sizeof(float) +
         4 * sizeof(int) * (size_t)nsl + 128;
}

// Dynamic shared memory of a row-pair launch: kPairStages boxes (128-byte
// aligned), the per-slab footprints, alignment slack.
static size_t pair_smem(const SlabBox& b, size_t es, int nsl) {
  return kPairStages * ((b.bx * b.by * b.bz * es + 127) & ~size_t(127)) + 4 * sizeof(int) * (size_t)nsl + 128;
}

template <class V>
const SlabBox& pair_box_for(const cbct_plan* p) { return sizeof(V) == 4 ? p->pair : p->pair16; }

template <class V, int BX>
void launch_pair(cbct_plan* p, const V* vol, const V* volP, const V* volT, const FwdOut& o, int first, int cnt, cudaStream_t st,
                 cbct_dtype dt) {
  const SlabBox& b = pair_box_for<V>(p);
  const CUtensorMap mv = make_volume_map(dt, volP, p->g.nx, p->g.ny, p->g.nz, b);
  const CUtensorMap mt = volT ? make_volume_map(dt, volT, p->g.ny, p->g.nx, p->g.nz, b) : mv;
  const int nsl = forward_slabs(p->g, kTS);
  const size_t smem = pair_smem(b, sizeof(V), nsl);
  const dim3 grid((p->g.width + kPU - 1) / kPU, (p->g.height + kPV - 1) / kPV, cnt);
  if (p->debug_checks) {
    auto k = fwd_pair_kernel<V, BX, true>;
    ensure_smem_attr((const void*)k, smem);
    k<<<grid, kPairThreads, smem, st>>>(mv, mt, vol, p->d_views + first, p->gc, b.bz, nsl, o, p->d_flags);
  } else {
    auto k = fwd_pair_kernel<V, BX, false>;
    ensure_smem_attr((const void*)k, smem);
    k<<<grid, kPairThreads, smem, st>>>(mv, mt, vol, p->d_views + first, p->gc, b.bz, nsl, o, p->d_flags);
  }
  check_launch("fwd_pair_kernel");
}

template <class V>
const SlabBox& fan_box_for(const cbct_plan* p) { return sizeof(V) == 4 ? p->fan : p->fan16; }

template <class V, int BX>
void launch_fan(cbct_plan* p, const V* vol, const V* volP, const V* volT, const FwdOut& o, int first, int cnt, cudaStream_t st,
                cbct_dtype dt) {
  const SlabBox& b = fan_box_for<V>(p);
  const CUtensorMap mv = make_volume_map(dt, volP, p->g.nx, p->g.ny, p->g.nz, b);
  const CUtensorMap mt = volT ? make_volume_map(dt, volT, p->g.ny, p->g.nx, p->g.nz, b) : mv;
  const int nsl = forward_slabs(p->g, kTS);
  const size_t smem = forward_smem(b, sizeof(V), p->fan_lz, nsl);
  const dim3 grid((p->g.width + kFU - 1) / kFU, (p->g.height + kFV - 1) / kFV, cnt);
  if (p->debug_checks) {
    auto k = fwd_fan_kernel<V, BX, true>;
    ensure_smem_attr((const void*)k, smem);
    k<<<grid, kFU * 32, smem, st>>>(mv, mt, vol, p->d_views + first, p->gc, b.bz, p->fan_lz, nsl, o, p->d_flags);
  } else {
    auto k = fwd_fan_kernel<V, BX, false>;
    ensure_smem_attr((const void*)k, smem);
    k<<<grid, kFU * 32, smem, st>>>(mv, mt, vol, p->d_views + first, p->gc, b.bz, p->fan_lz, nsl, o, p->d_flags);
  }
  check_launch("fwd_fan_kernel");
}

// A volume TMA cannot read in place: rows or start off a 16-byte boundary.  The
// TMA kernels then read a row-padded copy, made with the transposed one in one pass
// (8 to 12 bytes per voxel, HBM-bound): 40 views of 301x211 from 150x141x93 voxels
// take 1.03 ms, the gather kernel's bounds-checked global loads 2.36 ms.
bool needs_padded_rows(const void* vol, int nx, size_t es) {
  return (nx * es) % 16 != 0 || reinterpret_cast<uintptr_t>(vol) % 16 != 0;
}

// Plan buffer for a row-padded copy of a volume of element size es, or NULL.
// 16-bit volumes keep theirs behind the transposed copy (d_volT has fp32 room).
void* padded_rows(const cbct_plan* p, size_t es) {
  if (p->g.nx % 4 != 0) return p->d_volP;
  if (es == 2 && p->g.nx % 8 != 0 && p->d_volT && !p->volT_plain) return static_cast<char*>(p->d_volT) + volT16_bytes(p->g);
  return nullptr;
}

template <class V>
void launch_typed(cbct_plan* p, int s, const void* vol_v, const FwdOut& o, cudaStream_t st, cbct_dtype dt,
                  int variant) {
  const V* vol = static_cast<const V*>(vol_v);
  const int first = p->first[s], cnt = p->count[s];
  dim3 grid((p->g.width + kTU - 1) / kTU, (p->g.height + kTV - 1) / kTV, cnt);
  if (variant == 0) {
    fwd_gather_kernel<V><<<grid, 256, 0, st>>>(vol, p->d_views + first, p->gc, o);
    check_launch("fwd_gather_kernel");
    return;
  }
  // Copies the TMA boxes come from: the x/y-transposed volume for x-dominant
  // views, and a row-padded one where the caller's rows are not TMA-aligned.
  const int pitchT = tma_pitch(p->g.ny, sizeof(V)), pitchP = tma_pitch(p->g.nx, sizeof(V));
  V* const volT = p->subset_has_xdom[s] ? static_cast<V*>(p->d_volT) : nullptr;
  V* const pad = needs_padded_rows(vol, p->g.nx, sizeof(V)) ? static_cast<V*>(padded_rows(p, sizeof(V))) : nullptr;
  // Odd sizes: calls that the gather kernel would take without scratch may come from
  // several streams.
  ScratchUse use(p->fwd_order, st, (volT || pad) && (p->g.nx % 8 || p->g.ny % 8));
  if (volT || pad) {
    const int nx = p->g.nx, ny = p->g.ny, nz = p->g.nz;
    if (sizeof(V) == 2 && nx % 2 == 0 && reinterpret_cast<uintptr_t>(vol) % 4 == 0) {
      const dim3 tg((nx + 63) / 64, (ny + 63) / 64, (nz + 1) / 2);
      volume_copies16_kernel<<<tg, dim3(32, 8), 0, st>>>(reinterpret_cast<const uint32_t*>(vol),
                                                         reinterpret_cast<uint16_t*>(volT), pitchT,
                                                         reinterpret_cast<uint32_t*>(pad), pitchP, nx, ny, nz);
    } else {
      const dim3 tg((nx + 31) / 32, (ny + 31) / 32, (nz + kCopyPlanes - 1) / kCopyPlanes);
      volume_copies_kernel<V><<<tg, dim3(32, 8), 0, st>>>(vol, volT, pitchT, pad, pitchP, nx, ny, nz);
    }
    check_launch("volume_copies_kernel");
  }
  const V* const volP = pad ? pad : vol;
  if (variant == 4) {
    quad_launch(p, dt, vol, volP, volT, o, first, cnt, st);
    return;
  }
  if (variant == 3) {
    switch (pair_box_for<V>(p).bx) {
      case 40: launch_pair<V, 40>(p, vol, volP, volT, o, first, cnt, st, dt); break;
      case 56: launch_pair<V, 56>(p, vol, volP, volT, o, first, cnt, st, dt); break;
      case 72: launch_pair<V, 72>(p, vol, volP, volT, o, first, cnt, st, dt); break;
      case 104: launch_pair<V, 104>(p, vol, volP, volT, o, first, cnt, st, dt); break;
      case 136: launch_pair<V, 136>(p, vol, volP, volT, o, first, cnt, st, dt); break;
      default: throw Error(CBCT_ERR_INTERNAL, "unsupported pair box width");
    }
    return;
  }
  if (variant == 2) {
    switch (fan_box_for<V>(p).bx) {
      case 24: launch_fan<V, 24>(p, vol, volP, volT, o, first, cnt, st, dt); break;
      case 40: launch_fan<V, 40>(p, vol, volP, volT, o, first, cnt, st, dt); break;
      case 56: launch_fan<V, 56>(p, vol, volP, volT, o, first, cnt, st, dt); break;
      case 72: launch_fan<V, 72>(p, vol, volP, volT, o, first, cnt, st, dt); break;
      default: throw Error(CBCT_ERR_INTERNAL, "unsupported fan box width");
    }
    return;
  }
  slab_launch(p, dt, vol, volP, volT, o, first, cnt, st);
}

template <class V, int BX>
void prepare_pair_width(size_t smem) {
  ensure_smem_attr((const void*)fwd_pair_kernel<V, BX, false>, smem);
  ensure_smem_attr((const void*)fwd_pair_kernel<V, BX, true>, smem);
}

template <class V, int BX>
void prepare_fan_width(size_t smem) {
  ensure_smem_attr((const void*)fwd_fan_kernel<V, BX, false>, smem);
  ensure_smem_attr((const void*)fwd_fan_kernel<V, BX, true>, smem);
}

template <class V>
void prepare_typed(const cbct_plan* p) {
  if (p->fwd_variant == 3) {
    const SlabBox& b = pair_box_for<V>(p);
    const size_t ps = pair_smem(b, sizeof(V), forward_slabs(p->g, kTS));
    switch (b.bx) {
      case 40: prepare_pair_width<V, 40>(ps); break;
      case 56: prepare_pair_width<V, 56>(ps); break;
      case 72: prepare_pair_width<V, 72>(ps); break;
      case 104: prepare_pair_width<V, 104>(ps); break;
      case 136: prepare_pair_width<V, 136>(ps); break;
      default: break;
    }
  }
  if (p->fwd_variant == 2) {
    const SlabBox& f = fan_box_for<V>(p);
    const size_t fs = forward_smem(f, sizeof(V), p->fan_lz, forward_slabs(p->g, kTS));
    switch (f.bx) {
      case 24: prepare_fan_width<V, 24>(fs); break;
      case 40: prepare_fan_width<V, 40>(fs); break;
      case 56: prepare_fan_width<V, 56>(fs); break;
      case 72: prepare_fan_width<V, 72>(fs); break;
      default: break;
    }
  }
}

}  // namespace

int forward_slabs(const cbct_geometry& g, int TS) {
  return (std::max(g.nx, g.ny) + 1 - kSlabBase + TS - 1) / TS + 1;
}

// Largest footprint of one slab over every view and tile of a TU x TV tiling
// (corner-ray bounding box in the view's frame, computed in FP64): e extent
// and z extent in elements, including margins.  False when some view cannot
// use slabs (a ray not dominated by its view's slab axis, or too many slabs).
bool slab_extents(const cbct_plan* p, int TU, int TV, int TS, int& ext_e, int& ext_z, bool beside) {
  const cbct_geometry& g = p->g;
  const double kx = g.nx / (double)g.lx, ky = g.ny / (double)g.ly, kz = g.nz / (double)g.lz;
  const double bx = g.nx / 2.0 - 0.5, by = g.ny / 2.0 - 0.5, bz = g.nz / 2.0 - 0.5;
  const int tiles_u = (g.width + TU - 1) / TU, tiles_v = (g.height + TV - 1) / TV;
  struct Acc { int e = 0, z = 0, ok = 1; };
  std::vector<Acc> acc(host_threads());
  // The in-plane coordinate of a ray does not depend on the detector row, so the
  // e extent is a function of (view, tile column, slab); the z extent comes from
  // the products t * dz at the extreme path parameters and rows of each tile.
  parallel_for(p->n_views, [&](int lo, int hi, int tid) {
    Acc& a = acc[tid];
    std::vector<double> dz0(tiles_v), dz1(tiles_v);
    for (int iv = lo; iv < hi && a.ok; ++iv) {
      const ViewParams& vp = p->hviews[iv];
      const int dom = vp.dom;
      const int Nd = dom ? g.ny : g.nx, Ne = dom ? g.nx : g.ny;
      const double ke = dom ? kx : ky, be = dom ? bx : by, kd = dom ? ky : kx, bd = dom ? by : bx;
      const double Se = dom ? vp.Sx : vp.Sy, Sd = dom ? vp.Sy : vp.Sx, ikd = 1.0 / kd;
      const int nsl = (Nd + 1 - kSlabBase + TS - 1) / TS + 1;
      if (nsl * TS > kMaxSlabs * kTS) { a.ok = 0; break; }
      for (int tv = 0; tv < tiles_v; ++tv) {
        const int v0 = tv * TV, ve = std::min(v0 + TV, g.height) - 1;
        dz0[tv] = vp.D0z + v0 * (double)vp.Evz;
        dz1[tv] = vp.D0z + ve * (double)vp.Evz;
      }
      const double dzabs = std::max(std::fabs(dz0[0]), std::fabs(dz1[tiles_v - 1]));
      const double dzspan = (TV - 1) * (double)vp.Evz;
      // Distances of the first and last slab plane from the source along the slab axis,
      // and the largest |dz| of a row that meets the volume.
      const double near = (kSlabBase - bd) * ikd - Sd, far = (kSlabBase + nsl * TS - bd) * ikd - Sd;
      const double pmax = std::max(std::fabs(near), std::fabs(far)), pmin = std::min(std::fabs(near), std::fabs(far));
      const bool ahead = near * vp.dsgn > 0 && far * vp.dsgn > 0;
      for (int tu = 0; tu < tiles_u && a.ok; ++tu) {
        const int uc[2] = {tu * TU, std::min(tu * TU + TU, g.width) - 1};
        double de[2], dd[2];
        for (int c = 0; c < 2; ++c) {
          const double dx = vp.D0x + uc[c] * (double)vp.Eux, dy = vp.D0y + uc[c] * (double)vp.Euy;
          de[c] = dom ? dx : dy;
          dd[c] = dom ? dy : dx;
          // The slab axis must dominate every ray of the view with a uniform sign.
          if (dd[c] * vp.dsgn <= 0 || dd[c] * vp.dsgn < 0.25 * std::fabs(de[c])) a.ok = 0;
        }
        if (!a.ok) break;
        // Ray parameters t and e coordinates of the tile's two edge columns at a
        // slab's first plane; the last plane is the next slab's first.
        const double idd[2] = {1.0 / dd[0], 1.0 / dd[1]};
        // No slab of this tile spans more than these: skip the tile where neither can
        // exceed what was found so far (most tiles: two thirds of the time over random plans).
        const double s0 = de[0] * idd[0], s1 = de[1] * idd[1], ai = std::max(std::fabs(idd[0]), std::fabs(idd[1]));
        const double dmost = beside || !ahead
                                 ? dzabs
                                 : std::min(dzabs, (g.nz + 1.0 - bz) / (kz * pmin * std::min(std::fabs(idd[0]), std::fabs(idd[1]))));
        const double se = ke * (TS * ikd * std::max(std::fabs(s0), std::fabs(s1)) + pmax * std::fabs(s0 - s1));
        const double sz = kz * ((TS * ikd * ai + pmax * std::fabs(idd[0] - idd[1])) * dmost + pmax * ai * dzspan);
        if (std::min(std::ceil(se + 1e-9) + 3 + 2, Ne + 4.0) <= a.e && std::min(std::ceil(sz + 1e-9) + 3 + 2, g.nz + 4.0) <= a.z)
          continue;
        double t0[2], e0[2], t1[2], e1[2];
        auto at_plane = [&](int m, double (&t)[2], double (&e)[2]) {
          const double pl = (kSlabBase + m * TS - bd) * ikd - Sd;
          for (int c = 0; c < 2; ++c) {
            t[c] = pl * idd[c];
            e[c] = (Se + t[c] * de[c]) * ke + be;
          }
        };
        at_plane(0, t1, e1);
        for (int m = 0; m < nsl; ++m) {
          for (int c = 0; c < 2; ++c) { t0[c] = t1[c]; e0[c] = e1[c]; }
          at_plane(m + 1, t1, e1);
          const double emn = std::min(std::min(e0[0], e0[1]), std::min(e1[0], e1[1]));
          const double emx = std::max(std::max(e0[0], e0[1]), std::max(e1[0], e1[1]));
          const double tmn = std::min(std::min(t0[0], t0[1]), std::min(t1[0], t1[1]));
          const double tmx = std::max(std::max(t0[0], t0[1]), std::max(t1[0], t1[1]));
          // elements from floor(min)-1 to floor(max)+1 inclusive, +2 margin; the
          // kernels clamp footprints to the volume, whose extent bounds the box
          // a slab where the tile's rays are beside the volume holds no samples
          if (!beside && (emx < -1.0 || emn > Ne)) continue;
          a.e = std::max(a.e, std::min((int)(std::floor(emx) - std::floor(emn)) + 3 + 2, Ne + 4));
          // A tile row inside the volume spans at most this in z: skip the rows
          // where none can exceed the extent found so far.
          const double dmax =
              beside ? dzabs : std::min(dzabs, (g.nz + 1.0 - bz) / (kz * std::max(tmn, 1e-9)));
          if (tmn > 0 && std::ceil(kz * ((tmx - tmn) * dmax + tmx * dzspan)) + 3 + 2 <= a.z) continue;
          // One tile row; false where the rows towards the centre, whose extent is
          // smaller, cannot exceed the extent found so far.
          auto row = [&](int tv) {
            const double z00 = tmn * dz0[tv], z01 = tmn * dz1[tv], z10 = tmx * dz0[tv], z11 = tmx * dz1[tv];
            const double zmn = std::min(std::min(z00, z01), std::min(z10, z11)) * kz + bz;
            const double zmx = std::max(std::max(z00, z01), std::max(z10, z11)) * kz + bz;
            if (!beside && (zmx < -1.0 || zmn > g.nz)) return true;
            if (std::ceil(zmx - zmn) + 3 + 2 <= a.z) return false;
            const int ez = (int)(std::floor(zmx) - std::floor(zmn)) + 3 + 2;
            a.z = std::max(a.z, std::min(ez, g.nz + 4));
            return true;
          };
          row(tiles_v - 1);   // may hold fewer rays than the others
          int lo_v = 0, hi_v = tiles_v - 2;
          if (tmn > 0) {
            while (lo_v <= hi_v && dz1[lo_v] <= 0 && row(lo_v)) ++lo_v;
            while (hi_v >= lo_v && dz0[hi_v] >= 0 && row(hi_v)) --hi_v;
            while (lo_v <= hi_v && dz1[lo_v] <= 0) ++lo_v;
            while (hi_v >= lo_v && dz0[hi_v] >= 0) --hi_v;
          }
          for (int tv = lo_v; tv <= hi_v; ++tv) row(tv);
        }
      }
    }
  }, 16000 / std::max(1, tiles_u * forward_slabs(g, TS)));
  ext_e = ext_z = 0;
  bool ok = true;
  for (const Acc& a : acc) {
    ext_e = std::max(ext_e, a.e);
    ext_z = std::max(ext_z, a.z);
    ok = ok && a.ok;
  }
  return ok;
}

// Whether the detector's pixels are so wide that a box of 16 x 16 rays and kTS voxels,
// two of them a CTA, has no room in shared memory anywhere along the rays.  A bound of
// its extents from each view's outer columns settles it for all but such detectors.
static bool wide_pixels(const cbct_plan* p) {
  const cbct_geometry& g = p->g;
  const double kx = g.nx / (double)g.lx, ky = g.ny / (double)g.ly, kz = g.nz / (double)g.lz;
  auto fits = [](int e, int z) {
    int w32 = 0, w16 = 0;
    for (int w : kBoxWidths) {
      if (!w32 && w >= e + 3) w32 = w;
      if (!w16 && w >= e + 7) w16 = w;
    }
    auto smem = [&](int w, int es) { return kNStage * (((size_t)w * kBoxY * z * es + 127) & ~size_t(127)) + 128; };
    return w32 && w16 && z <= 256 && smem(w32, 4) <= (size_t)kSmemBudget && smem(w16, 2) <= (size_t)kSmemBudget;
  };
  double be = 0, bz = 0;
  for (int iv = 0; iv < p->n_views; ++iv) {
    const ViewParams& vp = p->hviews[iv];
    const bool dom = vp.dom;
    const int Nd = dom ? g.ny : g.nx;
    const double ke = dom ? kx : ky, kd = dom ? ky : kx, Sd = dom ? vp.Sy : vp.Sx;
    const double Ee = dom ? vp.Eux : vp.Euy, Ed = dom ? vp.Euy : vp.Eux;
    const double D0e = dom ? vp.D0x : vp.D0y, D0d = dom ? vp.D0y : vp.D0x;
    // depth of the farthest slab plane from the source, least depth of a ray at t = 1
    const double depth = std::fabs(Sd) + (0.5 * Nd + 2.0 * kTS + 2.0) / kd;
    double dd = 1e30, slope = 0;
    for (double u : {0.0, g.width - 1.0}) {
      dd = std::min(dd, std::fabs(D0d + u * Ed));
      slope = std::max(slope, std::fabs((D0e + u * Ee) / (D0d + u * Ed)));
    }
    const double dz = std::max(std::fabs((double)vp.D0z), std::fabs(vp.D0z + (g.height - 1.0) * vp.Evz));
    be = std::max(be, kTS * slope * ke / kd + depth * ke * (kTU - 1) * std::fabs(Ee * D0d - D0e * Ed) / (dd * dd));
    bz = std::max(bz, kz * ((kTS / kd / dd + depth * (kTU - 1) * std::fabs(Ed) / (dd * dd)) * dz +
                            depth / dd * (kTV - 1) * std::fabs((double)vp.Evz)));
  }
  auto ext = [](double span, int n) { return int(std::min(std::ceil(std::min(span, 1e6)) + 3 + 2, n + 4.0)); };
  if (fits(ext(be, std::max(g.nx, g.ny)), std::max(ext(bz, g.nz), 2))) return false;
  int e, z;
  return slab_extents(p, kTU, kTV, kTS, e, z, true) && !fits(e, std::max(z, 2));
}

bool forward_lerp_gather(const cbct_plan* p, size_t es) {
  return p->fwd_wide || ((size_t)p->g.nx * es) % 16 != 0 || ((size_t)p->g.ny * es) % 16 != 0;
}

// Largest z distance (texels) between the rays of adjacent detector rows at a
// point of the volume.  A point P lies at ray parameter t = (P - S).n / SDD,
// n the unit vector from the source towards the detector centre, so over the
// volume t <= (SAD + hx |sin| + hy |cos|) / SDD; rows are dv apart at t = 1.
static double row_dz_max(const cbct_plan* p) {
  const cbct_geometry& g = p->g;
  const double kz = g.nz / (double)g.lz, dv = double(g.fov_v) / g.height;
  double m = 0;
  for (int iv = 0; iv < p->n_views; ++iv) {
    const double th = double(p->angles[iv]) * (3.14159265358979323846 / 180.0);
    const double tmax = (g.SAD + 0.5 * g.lx * std::fabs(std::sin(th)) + 0.5 * g.ly * std::fabs(std::cos(th))) / g.SDD;
    m = std::max(m, tmax * dv * kz);
  }
  return m;
}

// Row distances (texels) from which launches take the slab kernel at any size (see
// launch_variant), fp32 and 16-bit volumes.
constexpr double kRowsApart = 1.2, kRowsApart16 = 1.0;

// Chooses the forward variant and its TMA boxes from the plan geometry: the
// row-quad kernel by quad_choose's rule, else the row-pair kernel where adjacent
// detector rows are less than one z texel apart over the whole volume (so pairs
// share their planes) and its boxes fit, else the per-ray slab kernel where its
// boxes fit, else the gather kernel.  CBCT_OPT_FORWARD_KERNEL forces slab (1),
// gather (2), fan (3), pairs (4) or quads (5).
void forward_choose_variant(cbct_plan* p) {
  p->fwd_variant = 0;
  p->slab = SlabBox{0, 0, 0, 0};
  p->fan = SlabBox{0, 0, 0, 0};
  p->pair = p->pair16 = SlabBox{0, 0, 0, 0};
  p->quad = p->quad16 = SlabBox{0, 0, 0, 0};
  // Per view range (subsets, the all-views entry and bin segments).
  p->subset_has_xdom.assign(p->first.size(), 0);
  for (size_t s = 0; s < p->first.size(); ++s)
    for (int i = p->first[s]; i < p->first[s] + p->count[s]; ++i)
      if (p->hviews[i].dom == 0) p->subset_has_xdom[s] = 1;
  p->fwd_wide = 0;
  if (p->force_gather || p->fwd_pref == 2) return;
  p->fwd_wide = wide_pixels(p);   // off again for a forced kernel of another form
  // The x start of a box is rounded down to a 16-byte boundary (4 fp32 or 8
  // 16-bit elements), which widens the box by up to 3 or 7 elements.
  auto width = [](const auto& list, int ext, int slack) {
    for (int w : list)
      if (w >= ext + slack) return w;
    return 0;
  };
  const double row_dz = p->fwd_row_dz = row_dz_max(p);
  const double height = double(p->g.fov_v) * (p->g.SAD / p->g.SDD) * p->g.nz / p->g.lz;
  p->fwd_fill_rays = height <= p->g.nz ? 8e5 : row_dz < 0.9 ? 2e6 : 3e6;
  // Rows so far apart that no launch would take quads (launch_variant), where the slab
  // kernel's boxes fit.
  const bool apart = p->fwd_pref == 0 && row_dz >= kRowsApart && slab_choose(p);
  if (!apart && (p->fwd_pref == 0 || p->fwd_pref == 5) && quad_choose(p, row_dz, p->fwd_pref == 5)) {
    p->fwd_variant = 4;
    // The slab kernel's boxes, where launch_variant may take it for some view range.
    bool slab = row_dz >= kRowsApart16;
    for (int c : p->count) slab = slab || (c > 0 && double(p->g.width) * p->g.height * c < p->fwd_fill_rays);
    if (p->fwd_pref == 5) p->fwd_wide = 0;
    if ((p->fwd_pref == 0 && slab) || p->fwd_tuned_views) slab_choose(p);
    return;
  }
  int e, z;
  if (slab_choose(p)) p->fwd_variant = 1;
  if ((p->fwd_pref == 4 || (p->fwd_pref == 0 && p->fwd_variant == 1 && row_dz < 0.99)) &&
      slab_extents(p, kPU, kPV, kTS, e, z)) {
    const int w32 = width(kBoxWidths, e, 3), w16 = width(kBoxWidths, e, 7);
    const int boxz = std::max(z, 3);
    const SlabBox b32{w32, kPairBoxY, boxz, 1}, b16{w16, kPairBoxY, boxz, 1};
    const int nsl = forward_slabs(p->g, kTS);
    if (w32 && w16 && boxz <= 256 && pair_smem(b32, 4, nsl) <= (size_t)kSmemBudget &&
        pair_smem(b16, 2, nsl) <= (size_t)kSmemBudget) {
      p->pair = b32;
      p->pair16 = b16;
      p->fwd_variant = 3;
      if (p->fwd_pref == 4) p->fwd_wide = 0;
    }
  }
  if (p->fwd_pref == 3 && slab_extents(p, kFU, kFV, kTS, e, z)) {
    const int w32 = width(kFanWidths, e, 3), w16 = width(kFanWidths, e, 7);
    const int boxz = std::max(z, 2);
    const int lz = (boxz + 1) | 1;  // odd: consecutive lines start in different banks
    const SlabBox b32{w32, kBoxY, boxz, 1}, b16{w16, kBoxY, boxz, 1};
    const int nsl = forward_slabs(p->g, kTS);
    if (w32 && w16 && boxz <= 256 && forward_smem(b32, 4, lz, nsl) <= (size_t)kSmemBudget &&
        forward_smem(b16, 2, lz, nsl) <= (size_t)kSmemBudget) {
      p->fan = b32;
      p->fan16 = b16;
      p->fan_lz = lz;
      p->fwd_variant = 2;
      p->fwd_wide = 0;
    }
  }
}

// Variant of a launch of cnt views.  Row pairs and quads need many rays: a thread
// marches two or four one after another, and rays cut by the volume's top or bottom
// face are marched by themselves.  Below fwd_fill_rays rays an automatically chosen
// plan's launches run the per-ray slab kernel, whose results are bitwise the same.
// Measured in ms, slab against the better of pairs and quads: detectors that the volume's
// height covers, threshold 0.8 million rays: 2 views of 0.9 mm pixels into 128^3
// (0.12 M rays) 0.088 to 0.173, 8 views (0.47 M) 0.223 to 0.232, 32 views (1.9 M) 0.829
// to 0.692; 2 views of 0.75 mm into 256^3 (0.68 M) 0.54 to 0.71, 8 views (2.7 M) 2.07 to
// 1.48.  Taller detectors, whose outer rays are cut, 2 million, between
// break-evens of 1 and 3 million by volume and detector: 4 views of 512x512 into 256^3 (1.0
// M) 0.89 to 0.81, 8 views (2.1 M) 1.71 to 1.52; 304x208 into 152x144x96 20 views (1.3 M)
// 0.57 to 0.60, 32 views (2.0 M) 0.88 to 0.86; 256x256 into 128^3 32 views (2.1 M) 0.86 to
// 0.90, 48 views (3.1 M) 1.27 to 1.27; 3 million for rows 0.9 texel or more apart:
// 2 views of 1.5 mm into 256^3 (0.2 M) 0.25 to 0.55, 64 views of 256x192 into 128^3
// (3.1 M) 1.06 to 1.01.
// Rows beyond 1.2 texels (16-bit volumes: 1) share too few planes at any size: 40 views of
// 400x300 into 256^3, 1.34 texels, 3.78 to 3.75, 1.5 texels 3.30 to 3.76; bf16 at 1.1 texels 4.01
// to 4.19, 1.18 texels 3.73 to 4.38.
static int launch_variant(const cbct_plan* p, int cnt, size_t es) {
  const bool rows = p->fwd_variant == 3 || p->fwd_variant == 4;
  const double rays = double(p->g.width) * p->g.height * cnt;
  const bool automatic = p->fwd_pref == 0 || cnt < p->fwd_tuned_views;
  if (rows && automatic && p->slab.bx && (rays < p->fwd_fill_rays || p->fwd_row_dz >= (es == 2 ? kRowsApart16 : kRowsApart)))
    return 1;
  // The gather form is compiled for the slab and quad kernels.
  if (forward_lerp_gather(p, es) && (p->fwd_variant == 2 || p->fwd_variant == 3)) return p->slab.bx ? 1 : 0;
  return p->fwd_variant;
}

static int variant_of(const cbct_plan* p, int s, cbct_dtype dt, const void* vol) {
  const size_t es = dtype_size(dt);
  const bool tma = (!needs_padded_rows(vol, p->g.nx, es) || padded_rows(p, es) != nullptr) &&
                   (!p->subset_has_xdom[s] || (p->d_volT != nullptr && !(p->volT_plain && forward_lerp_gather(p, es))));
  return tma ? launch_variant(p, p->count[s], es) : 0;
}

int forward_variant_of(const cbct_plan* p, int s, cbct_dtype dt) { return variant_of(p, s, dt, nullptr); }

void forward_prepare(cbct_plan* p) {
  if (p->fwd_variant < 1) return;
  prepare_typed<float>(p);
  prepare_typed<__half>(p);
  prepare_typed<__nv_bfloat16>(p);
  if (p->slab.bx) slab_prepare(p);
  if (p->fwd_variant == 4) quad_prepare(p);
  bool any_x = false;
  for (size_t s = 0; s < p->subset_has_xdom.size(); ++s) any_x = any_x || p->subset_has_xdom[s];
  // Row-padded copies are made where the device has room for them: without, launches over
  // rows that TMA cannot read run the gather kernel, whose rays through the volume they
  // are anyway.
  const size_t plain = (size_t)p->g.nx * p->g.ny * p->g.nz * 4;
  const bool padded = volT_bytes(p->g) > plain || volP_bytes(p->g);
  if (any_x && !p->d_volT) {
    if (!padded) p->d_volT = plan_alloc(p, plain);
    else if (p->pads) p->d_volT = plan_try_alloc(p, volT_bytes(p->g));
    if (!p->d_volT && p->g.nx % 4 == 0 && p->g.ny % 4 == 0) {   // aligned fp32 launches need theirs
      p->d_volT = plan_alloc(p, plain);
      p->volT_plain = 1;
    }
  }
  if (volP_bytes(p->g) && !p->d_volP && p->pads && (!any_x || p->d_volT)) p->d_volP = plan_try_alloc(p, volP_bytes(p->g));
}

void forward_launch(cbct_plan* p, int s, cbct_dtype dt, const void* vol, float* out, const float* b,
                    float scale, int mode, int apply_offset, int accumulate, double* norm2_out,
                    cudaStream_t st) {
  forward_launch_ex(p, s, dt, vol, out, b, nullptr, scale, mode, apply_offset, accumulate, norm2_out, st);
}

void forward_launch_ex(cbct_plan* p, int s, cbct_dtype dt, const void* vol, float* out, const void* b,
                       const float* pw, float scale, int mode, int apply_offset, int accumulate,
                       double* norm2_out, cudaStream_t st, cbct_dtype b_dtype) {
  FwdOut o;
  o.out = out;
  o.pw = pw;
  o.b = b;
  o.b_dtype = b_dtype;
  o.scale = scale;
  o.mode = mode;
  o.apply_offset = apply_offset;
  o.accumulate = accumulate;
  o.partials = nullptr;
  const int cnt = p->count[s];
  if (cnt == 0) return;
  o.wproj = p->d_pweights ? p->d_pweights + (size_t)p->g.width * p->g.height * p->first[s] : nullptr;
  const int variant = variant_of(p, s, dt, vol);
  // One partial sum per block of the kernel that will run.
  int TU = kTU, TV = kTV;
  if (variant == 1) slab_tile(TU, TV);
  else if (variant == 2) { TU = kFU; TV = kFV; }
  else if (variant == 3) { TU = kPU; TV = kPV; }
  else if (variant == 4) quad_tile(p->quad_shape, TU, TV);
  const size_t nblocks = (size_t)((p->g.width + TU - 1) / TU) * ((p->g.height + TV - 1) / TV) * cnt;
  if (norm2_out) {
    if (nblocks > p->n_partials) throw Error(CBCT_ERR_INTERNAL, "partials buffer too small");
    o.partials = p->d_partials;
  }
  switch (dt) {
    case CBCT_F32: launch_typed<float>(p, s, vol, o, st, dt, variant); break;
    case CBCT_F16: launch_typed<__half>(p, s, vol, o, st, dt, variant); break;
    case CBCT_BF16: launch_typed<__nv_bfloat16>(p, s, vol, o, st, dt, variant); break;
    default: throw Error(CBCT_ERR_INVALID_ARGUMENT, "unknown volume dtype");
  }
  if (norm2_out) finalize_partials(p->d_partials, (int)nblocks, norm2_out, st);
}

namespace {

// Work-list launch of kernel k over the records of one group.
void add_fwd_group(WorkArena& A, FwdMultiKernel k, int threads, const std::vector<FwdScanRec>& recs, int total,
                   size_t smem) {
  ensure_smem_attr((const void*)k, smem);
  const size_t off = A.add(recs.data(), recs.size() * sizeof(FwdScanRec));
  const int ci = A.n_counters++;
  const int grid = std::min(total, resident_grid((const void*)k, threads, smem));
  const int n = (int)recs.size();
  A.ops.push_back([&A, k, off, ci, grid, threads, n, total, smem](cudaStream_t st) {
    k<<<grid, threads, smem, st>>>(reinterpret_cast<const FwdScanRec*>(A.dev + off), n, total, A.counter(ci));
    check_launch("forward work-list kernel");
  });
}

FwdMultiKernel fwd_multi_ptr(int bx) {
  switch (bx) {
    case 40: return fwd_multi_kernel<40>;
    case 56: return fwd_multi_kernel<56>;
    case 72: return fwd_multi_kernel<72>;
    case 104: return fwd_multi_kernel<104>;
    case 136: return fwd_multi_kernel<136>;
    default: throw Error(CBCT_ERR_INTERNAL, "unsupported forward box width");
  }
}

// Small scans that fill the GPU together run quads where their rows share enough planes.
// Their rays are bitwise the slab kernel's; a norm is summed tile by tile, so scans that
// want theirs keep the kernel of their own launches.  Whole batches of 2, 4 or 6 scans, us,
// with quads and with the slab kernel:
//  detectors that the volume's height covers, rows up to 0.9 texel, 300,000 rays a step: 0.45
//  texel, 0.06 M rays 765, 720; 0.25 M 1487, 2045; 1.4 M 5493, 9486; 0.66 texel, 0.83 M 4559,
//  6606; 0.77 texel, 0.9 M 4218, 3979; 0.85 texel, 0.52 M 3855, 4061; 1.2 M 7763, 8903;
//  taller detectors, whose outer rays are cut, rows up to half a texel, 0.6 from three
//  million rays a step: 0.42 texel, 0.08 M
//  1247, 834; 0.31 M 2243, 2423; 1.7 M 11649, 11968; 0.53 texel, 0.81 M 7428, 6561; 0.56
//  texel, 0.59 M 3923, 3731; 1.8 M 11084, 9221; 4.4 M 21097, 22172.
constexpr double kMultiQuadRays = 3e5;

// The scans of one kernel (kind, shape and box width).
struct FwdGroup {
  FwdMultiKernel k;
  int threads;
  std::vector<FwdScanRec> recs;
  int total = 0;
  size_t smem = 0;
};

}  // namespace

void forward_multi(WorkArena& A, const std::vector<MultiFwdJob>& jobs) {
  std::vector<FwdGroup> groups;
  double all_rays = 0;
  for (const MultiFwdJob& j : jobs) all_rays += double(j.p->g.width) * j.p->g.height * j.p->count[j.s];
  // Transposes of the volumes the next launches read, one launch for all.
  std::vector<TransposeRec> tr;
  int tr_total = 0;
  auto flush_transposes = [&]() {
    if (tr.empty()) return;
    const size_t off = A.add(tr.data(), tr.size() * sizeof(TransposeRec));
    const int n = (int)tr.size(), total = tr_total;
    A.ops.push_back([&A, off, n, total](cudaStream_t st) {
      transpose_multi_kernel<<<total, dim3(32, 8), 0, st>>>(reinterpret_cast<const TransposeRec*>(A.dev + off), n);
      check_launch("transpose_multi_kernel");
    });
    tr.clear();
    tr_total = 0;
  };
  auto flush = [&](FwdGroup& g) {
    if (g.recs.empty()) return;
    flush_transposes();
    add_fwd_group(A, g.k, g.threads, g.recs, g.total, g.smem);
    g.recs.clear();
    g.total = 0;
    g.smem = 0;
  };
  std::vector<std::function<void(cudaStream_t)>> after;
  for (const MultiFwdJob& j : jobs) {
    cbct_plan* p = j.p;
    const int s = j.s, first = p->first[s], cnt = p->count[s];
    if (cnt == 0) continue;
    const bool tma = p->fwd_variant >= 1 && !forward_lerp_gather(p, sizeof(float)) &&
                     (reinterpret_cast<uintptr_t>(j.vol) % 16 == 0) && (!p->subset_has_xdom[s] || p->d_volT);
    int fv = launch_variant(p, cnt, sizeof(float));
    if (fv == 1 && p->fwd_variant == 4 && (p->fwd_pref == 0 || p->fwd_tuned_views) && !j.norm2_out && all_rays >= kMultiQuadRays &&
        p->fwd_row_dz < (p->fwd_fill_rays < 1e6 ? 0.9 : all_rays < 3e6 ? 0.5 : 0.6))
      fv = 4;
    auto one_scan = [&A](const MultiFwdJob& jj) {
      A.ops.push_back([jj](cudaStream_t st) {
        forward_launch_ex(jj.p, jj.s, CBCT_F32, jj.vol, jj.out, jj.b, nullptr, 1.f, kModeResidual, jj.apply_offset,
                          0, jj.norm2_out, st, jj.b_dtype);
      });
    };
    if (!tma || fv == 2 || p->debug_checks) {
      one_scan(j);
      continue;
    }
    int nsl = forward_slabs(p->g, kTS), TU, TV, threads;
    SlabBox b;
    size_t sm = 0;
    FwdMultiKernel kernel;
    if (fv == 4) {
      const ForwardMulti q = quad_multi(p);
      b = p->quad; kernel = q.kernel; nsl = q.nsl; sm = q.smem; threads = q.threads;
      quad_tile(p->quad_shape, TU, TV);
    } else if (fv == 3) {
      b = p->pair; TU = kPU; TV = kPV; sm = pair_smem(b, 4, nsl); threads = kPairThreads;
      kernel = fwd_multi_ptr(b.bx);
    } else {
      const ForwardMulti q = slab_multi(p);
      b = p->slab; kernel = q.kernel; nsl = q.nsl; sm = q.smem; threads = q.threads;
      slab_tile(TU, TV);
    }
    const int tx = (p->g.width + TU - 1) / TU, ty = (p->g.height + TV - 1) / TV;
    const int nblocks = tx * ty * cnt;
    ensure_smem_attr((const void*)kernel, sm);
    if (nblocks >= kMultiFillWaves * resident_grid((const void*)kernel, threads, sm)) {
      one_scan(j);
      continue;
    }
    auto gi = std::find_if(groups.begin(), groups.end(), [&](const FwdGroup& g) { return g.k == kernel; });
    if (gi == groups.end()) {
      FwdGroup ng;
      ng.k = kernel;
      ng.threads = threads;
      gi = groups.insert(groups.end(), std::move(ng));
    }
    FwdGroup& g = *gi;
    const float* volT = nullptr;
    if (p->subset_has_xdom[s]) {
      float* t = static_cast<float*>(p->d_volT);
      if ((int)tr.size() == kMultiMaxRecs) flush_transposes();
      TransposeRec q{j.vol, t, p->g.nx, p->g.ny, (p->g.nx + 31) / 32, (p->g.ny + 31) / 32, tr_total};
      tr_total += q.tx * q.ty * p->g.nz;
      tr.push_back(q);
      volT = t;
    }
    FwdOut o{};
    o.out = j.out;
    o.b = j.b;
    o.b_dtype = j.b_dtype;
    o.pw = nullptr;
    o.scale = 1.f;
    o.mode = kModeResidual;
    o.apply_offset = j.apply_offset;
    o.accumulate = 0;
    o.partials = nullptr;
    o.wproj = p->d_pweights ? p->d_pweights + (size_t)p->g.width * p->g.height * first : nullptr;
    FwdScanRec r;
    std::memset(&r, 0, sizeof(r));
    r.map_v = make_volume_map(CBCT_F32, j.vol, p->g.nx, p->g.ny, p->g.nz, b);
    r.map_t = make_volume_map(CBCT_F32, volT ? (const void*)volT : (const void*)j.vol, volT ? p->g.ny : p->g.nx,
                       volT ? p->g.nx : p->g.ny, p->g.nz, b);
    r.vol = j.vol;
    r.views = p->d_views + first;
    r.flags = p->d_flags;
    r.gc = p->gc;
    r.BZ = b.bz;
    r.nsl_max = nsl;
    r.tx = tx;
    r.ty = ty;
    if (j.norm2_out) {
      if ((size_t)nblocks > p->n_partials) throw Error(CBCT_ERR_INTERNAL, "partials buffer too small");
      o.partials = p->d_partials;
      double* part = p->d_partials;
      double* out = j.norm2_out;
      after.push_back([part, nblocks, out](cudaStream_t st) { finalize_partials(part, nblocks, out, st); });
    }
    r.o = o;
    if ((int)g.recs.size() == kMultiMaxRecs) flush(g);
    r.base = g.total;
    g.total += nblocks;
    g.smem = std::max(g.smem, sm);
    g.recs.push_back(r);
  }
  for (FwdGroup& g : groups) flush(g);
  flush_transposes();
  for (auto& f : after) A.ops.push_back(std::move(f));
}

}  // namespace cbct
