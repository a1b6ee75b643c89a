// forward_quad.cu -- choice, instantiation and launches of the row-quad forward
// projector (device code in forward_quad.cuh).
#include <cmath>
#include <cstring>

#include "forward_host.h"
#include "forward_quad.cuh"

namespace cbct {

namespace {

struct QuadDims { int TU, TV, TS, BY, threads; };
template <int SHAPE>
constexpr QuadDims dims_of() {
  using C = typename ShapeOf<SHAPE>::C;
  return QuadDims{C::TU, C::TV, C::TS, C::BY, C::threads};
}
constexpr QuadDims kDims[kQuadShapes] = {dims_of<kQuadWide>(), dims_of<kQuadWarp>(), dims_of<kQuadThin>(),
                                          dims_of<kQuadSkew>()};

// One box (128-byte aligned), the slabs' box origins, alignment slack.
size_t quad_smem(const SlabBox& b, size_t es, int nsl) {
  return ((b.bx * b.by * b.bz * es + 127) & ~size_t(127)) + sizeof(int2) * (size_t)nsl + 128;
}

template <class V>
QuadKernel<V> quad_kernel(const cbct_plan* p) {
  if (forward_lerp_gather(p, sizeof(V))) return quad_kernel_gather<V>(p);
  QuadKernel<V> k = nullptr;
  with_quad<V>(p, [&](auto BX, auto SHAPE) { k = quad_kernel_of<V, decltype(BX)::value, decltype(SHAPE)::value, false>(); });
  return k;
}

template <class V>
void prepare_typed(const cbct_plan* p) {
  const SlabBox& b = sizeof(V) == 4 ? p->quad : p->quad16;
  const size_t smem = quad_smem(b, sizeof(V), forward_slabs(p->g, kDims[p->quad_shape].TS));
  ensure_smem_attr((const void*)quad_kernel<V>(p), smem);
}

template <class V>
void launch_typed(cbct_plan* p, const V* vol, const V* volP, const V* volT, const FwdOut& o, int first, int cnt, cudaStream_t st,
                  cbct_dtype dt) {
  const SlabBox& b = sizeof(V) == 4 ? p->quad : p->quad16;
  const CUtensorMap mv = make_volume_map(dt, volP, p->g.nx, p->g.ny, p->g.nz, b);
  const CUtensorMap mt = volT ? make_volume_map(dt, volT, p->g.ny, p->g.nx, p->g.nz, b) : mv;
  const QuadDims& d = kDims[p->quad_shape];
  const int nsl = forward_slabs(p->g, d.TS);
  const size_t smem = quad_smem(b, sizeof(V), nsl);
  const dim3 grid((p->g.width + d.TU - 1) / d.TU, (p->g.height + d.TV - 1) / d.TV, cnt);
  const QuadKernel<V> k = quad_kernel<V>(p);
  ensure_smem_attr((const void*)k, smem);
  k<<<grid, d.threads, smem, st>>>(mv, mt, vol, p->d_views + first, p->gc, b.bz, nsl, p->debug_checks, o, p->d_flags);
  check_launch("fwd_quad_kernel");
}

// Work list over many scans of one shape and box width (see fwd_multi_kernel).
template <int BX, int SHAPE>
__global__ void __launch_bounds__(ShapeOf<SHAPE>::C::threads, ShapeOf<SHAPE>::minb)
    quad_multi_kernel(const FwdScanRec* __restrict__ recs, int n_recs, int total, int* __restrict__ counter) {
  using C = typename ShapeOf<SHAPE>::C;
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 127) & ~uintptr_t(127));
  __shared__ QuadShared<C::NS> sh;
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
    fwd_quad_body<float, BX, C, false>(&R.map_v, &R.map_t, static_cast<const float*>(R.vol), R.views, R.gc, R.BZ, R.nsl_max,
                                false, R.o, R.flags, tile, smem_raw, sh);
    __syncthreads();
    // A wait that gave up is counted in the scan's flag word and its loads
    // drained; only a CTA whose drain also gave up stops taking items.
    const bool ok = sh.abort_flag != 2;
    if (threadIdx.x == 0) {
      for (int i = 0; i < C::NS; ++i) mbar_inval(&sh.bars[i]);
    }
    if (!ok) break;
  }
}

}  // namespace

void quad_tile(int shape, int& TU, int& TV) {
  TU = kDims[shape].TU;
  TV = kDims[shape].TV;
}

// Whether (and in which shape) the row-quad kernel projects this plan; sets its
// boxes.  row_dz: largest distance of adjacent rows (texels).  Launches with too few
// rays to fill the GPU run the slab kernel all the same (launch_variant).
//  row_dz < 0.66: always (4 planes per quad).  Up to 0.9 where the largest subset has
//  150,000 rays, up to 1.4 where it has a million (from 1.2 on the caller prefers the slab
//  kernel where its boxes fit): others have no launch that quads would gain on (180 views
//  of 256x192 into 128^3 at 1.09 texel: 2.42 ms, slab kernel 2.47, row pairs 3.36; 8 views
//  0.22, 0.14 and 0.22).
//  Shape: wide where its tiles are three waves and row_dz < 0.66 (20 views of 512x384
//  into 160^3: 1.10 ms against 1.17 with the warp shape; 10 views of 192x144 into 64^3,
//  0.3 waves: 0.139 against 0.115); warp up to 0.9 texel (25 views of 320x240 into
//  160x144x112: 0.86 ms, wide 0.92, row pairs 1.00); thin to 1 texel (40 views of 360x220
//  into 200^3 at 0.99 texel: 1.52 ms, skewed 1.66), skewed beyond (180 views of 256x192
//  into 128^3 at 1.09 texel: 2.31 ms, thin 2.42, warp 2.71, wide 3.69).  The next shape where
//  boxes do not fit or its index would leave its range.
bool quad_choose(cbct_plan* p, double row_dz, bool forced) {
  const double rays = double(p->g.width) * p->g.height * p->max_subset;
  if (!forced && !(row_dz < 0.66 || (row_dz < 0.9 && rays >= 1.5e5) || (row_dz < 1.4 && rays >= 1e6))) return false;
  const QuadDims& w = kDims[kQuadWide];
  const double wide = std::ceil(p->g.width / double(w.TU)) * std::ceil(p->g.height / double(w.TV)) * p->max_subset;
  int order[kQuadShapes] = {kQuadWide, kQuadWarp, kQuadThin, kQuadSkew};
  if (row_dz >= 1.0) std::swap(order[0], order[3]), std::swap(order[1], order[2]);
  else if (row_dz >= 0.9) std::swap(order[0], order[2]);
  else if (row_dz >= 0.66 || wide < 3.0 * 148 * ShapeOf<kQuadWide>::minb) std::swap(order[0], order[1]);
  for (int s : order) {
    const QuadDims& d = kDims[s];
    int e, z;
    if (!slab_extents(p, d.TU, d.TV, d.TS, e, z)) return false;
    // The x start of a box is rounded down to a 16-byte boundary.
    auto width = [](const int (&list)[2], int ext) { return list[0] >= ext ? list[0] : list[1] >= ext ? list[1] : 0; };
    const int w32 = width(kQuadWidths32[s], e + 3), w16 = width(kQuadWidths16[s], e + 7);
    const int boxz = std::max(z, 4), nsl = forward_slabs(p->g, d.TS);
    const SlabBox b32{w32, d.BY, boxz, 1}, b16{w16, d.BY, boxz, 1};
    if (!w32 || !w16 || boxz > 256 || quad_smem(b32, 4, nsl) > (size_t)kSmemBudget ||
        quad_smem(b16, 2, nsl) > (size_t)kSmemBudget || box_index_bound(p->g, b32) >= size_t(1) << 22 ||
        box_index_bound(p->g, b16) >= size_t(1) << 22)
      continue;   // (the index bound: volumes of more than 8,000 to 20,000 planes)
    p->quad = b32;
    p->quad16 = b16;
    p->quad_shape = s;
    return true;
  }
  return false;
}

void quad_prepare(const cbct_plan* p) {
  prepare_typed<float>(p);
  prepare_typed<__half>(p);
  prepare_typed<__nv_bfloat16>(p);
}

void quad_launch(cbct_plan* p, cbct_dtype dt, const void* vol, const void* volP, const void* volT, const FwdOut& o,
                 int first, int cnt, cudaStream_t st) {
  auto go = [&](auto v) {
    using V = decltype(v);
    launch_typed<V>(p, static_cast<const V*>(vol), static_cast<const V*>(volP), static_cast<const V*>(volT), o, first,
                    cnt, st, dt);
  };
  if (dt == CBCT_F32) go(float{});
  else if (dt == CBCT_F16) go(__half{});
  else go(__nv_bfloat16{});
}

ForwardMulti quad_multi(const cbct_plan* p) {
  ForwardMulti m{};
  const QuadDims& d = kDims[p->quad_shape];
  m.nsl = forward_slabs(p->g, d.TS);
  m.smem = quad_smem(p->quad, 4, m.nsl);
  m.threads = d.threads;
  with_quad<float>(p, [&](auto BX, auto SHAPE) {
    m.kernel = quad_multi_kernel<decltype(BX)::value, decltype(SHAPE)::value>;
  });
  return m;
}

}  // namespace cbct
