// forward_slab.cu -- instantiation, choice and launch of the per-ray slab forward
// projector (forward_slab.cuh).
#include <algorithm>

#include "forward_host.h"
#include "forward_slab.cuh"

namespace cbct {

namespace {

// Box widths (elements).  fp32: BX * kSlabBoxY is 8 or 24 words mod 32, so that the four
// rows of a warp, about a plane apart, fall on different banks.
constexpr int kSlabWidths32[] = {28, 36, 52, 84, 132};
constexpr int kSlabWidths16[] = {24, 40, 56, 88, 136};

// Per warp a box (128-byte aligned) and the slabs' box origins; alignment slack.
size_t slab_smem(const SlabBox& b, size_t es, int nsl) {
  const size_t box = (b.bx * b.by * b.bz * es + 127) & ~size_t(127);
  return kSlabWarps * (box + ((sizeof(int2) * nsl + 127) & ~size_t(127))) + 128;
}

// Calls f(std::integral_constant<int, BX>) for the compiled width bx.
template <class V, class F>
void with_slab(int bx, F&& f) {
  constexpr const int(&w)[5] = sizeof(V) == 4 ? kSlabWidths32 : kSlabWidths16;
  if (bx == w[0]) f(std::integral_constant<int, w[0]>{});
  else if (bx == w[1]) f(std::integral_constant<int, w[1]>{});
  else if (bx == w[2]) f(std::integral_constant<int, w[2]>{});
  else if (bx == w[3]) f(std::integral_constant<int, w[3]>{});
  else if (bx == w[4]) f(std::integral_constant<int, w[4]>{});
  else throw Error(CBCT_ERR_INTERNAL, "unsupported slab box width");
}

template <class V>
const SlabBox& box_of(const cbct_plan* p) { return sizeof(V) == 4 ? p->slab : p->slab16; }

template <class V>
void prepare_typed(const cbct_plan* p) {
  const SlabBox& b = box_of<V>(p);
  const size_t smem = slab_smem(b, sizeof(V), forward_slabs(p->g, kSlabTS));
  with_slab<V>(b.bx, [&](auto BX) {
    ensure_smem_attr(forward_lerp_gather(p, sizeof(V)) ? (const void*)fwd_slab_kernel<V, decltype(BX)::value, true>
                                                       : (const void*)fwd_slab_kernel<V, decltype(BX)::value, false>,
                     smem);
  });
}

template <class V>
void launch_typed(cbct_plan* p, const V* vol, const V* volP, const V* volT, const FwdOut& o, int first, int cnt,
                  cudaStream_t st, cbct_dtype dt) {
  const SlabBox& b = box_of<V>(p);
  const CUtensorMap mv = make_volume_map(dt, volP, p->g.nx, p->g.ny, p->g.nz, b);
  const CUtensorMap mt = volT ? make_volume_map(dt, volT, p->g.ny, p->g.nx, p->g.nz, b) : mv;
  const int nsl = forward_slabs(p->g, kSlabTS);
  const size_t smem = slab_smem(b, sizeof(V), nsl);
  const dim3 grid((p->g.width + kSlabU - 1) / kSlabU, (p->g.height + kSlabV - 1) / kSlabV, cnt);
  with_slab<V>(b.bx, [&](auto BX) {
    auto k = forward_lerp_gather(p, sizeof(V)) ? fwd_slab_kernel<V, decltype(BX)::value, true>
                                               : fwd_slab_kernel<V, decltype(BX)::value, false>;
    ensure_smem_attr((const void*)k, smem);
    k<<<grid, kSlabThreads, smem, st>>>(mv, mt, vol, p->d_views + first, p->gc, b.bz, nsl, p->debug_checks, o,
                                        p->d_flags);
  });
  check_launch("fwd_slab_kernel");
}

// Work list over many scans of one box width (see fwd_multi_kernel).
template <int BX>
__global__ void __launch_bounds__(kSlabThreads, kSlabMinb)
    slab_multi_kernel(const FwdScanRec* __restrict__ recs, int n_recs, int total, int* __restrict__ counter) {
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 127) & ~uintptr_t(127));
  __shared__ SlabShared sh;
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
    if ((threadIdx.x & 31) == 0 && lo != last) {   // the threads that issue the TMA loads
      tensormap_acquire(&R.map_v);
      tensormap_acquire(&R.map_t);
      last = lo;
    }
    fwd_slab_body<float, BX, false>(&R.map_v, &R.map_t, static_cast<const float*>(R.vol), R.views, R.gc, R.BZ, R.nsl_max,
                             false, R.o, R.flags, tile, smem_raw, sh);
    __syncthreads();
    // A wait that gave up is counted in the scan's flag word and its loads
    // drained; only a CTA whose drain also gave up stops taking items.
    const bool ok = sh.abort_flag != 2;
    if (threadIdx.x == 0) {
      for (int w = 0; w < kSlabWarps; ++w) mbar_inval(&sh.bars[w]);
    }
    if (!ok) break;
  }
}

}  // namespace

void slab_tile(int& TU, int& TV) {
  TU = kSlabU;
  TV = kSlabV;
}

// Sets the slab kernel's boxes; false where some view or box does not fit.
bool slab_choose(cbct_plan* p) {
  int e, z;
  if (!slab_extents(p, kSlabU, 4, kSlabTS, e, z)) return false;
  // The x start of a box is rounded down to a 16-byte boundary (4 fp32 or 8
  // 16-bit elements), which widens the box by up to 3 or 7 elements.
  auto width = [](const int (&list)[5], int ext) {
    for (int w : list)
      if (w >= ext) return w;
    return 0;
  };
  const int nsl = forward_slabs(p->g, kSlabTS);
  const SlabBox b32{width(kSlabWidths32, e + 3), kSlabBoxY, std::max(z, 2), 1};
  const SlabBox b16{width(kSlabWidths16, e + 7), kSlabBoxY, std::max(z, 2), 1};
  if (!b32.bx || !b16.bx || b32.bz > 256 || slab_smem(b32, 4, nsl) > (size_t)kSmemBudget ||
      slab_smem(b16, 2, nsl) > (size_t)kSmemBudget || box_index_bound(p->g, b32) >= size_t(1) << 24 ||
      box_index_bound(p->g, b16) >= size_t(1) << 24)
    return false;
  p->slab = b32;
  p->slab16 = b16;
  return true;
}

void slab_prepare(const cbct_plan* p) {
  prepare_typed<float>(p);
  prepare_typed<__half>(p);
  prepare_typed<__nv_bfloat16>(p);
}

void slab_launch(cbct_plan* p, cbct_dtype dt, const void* vol, const void* volP, const void* volT, const FwdOut& o,
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

ForwardMulti slab_multi(const cbct_plan* p) {
  ForwardMulti m{};
  m.nsl = forward_slabs(p->g, kSlabTS);
  m.smem = slab_smem(p->slab, 4, m.nsl);
  m.threads = kSlabThreads;
  with_slab<float>(p->slab.bx, [&](auto BX) { m.kernel = slab_multi_kernel<decltype(BX)::value>; });
  return m;
}

}  // namespace cbct
