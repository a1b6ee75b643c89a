// forward_host.h -- host-side declarations shared by the forward projector's
// translation units.
#pragma once

#include <algorithm>

#include "forward_device.cuh"

namespace cbct {

// A scan's entry in a work-list launch over many scans: the arguments of its
// one-scan launch and where its tiles start in the list.
struct alignas(128) FwdScanRec {
  CUtensorMap map_v, map_t;    // volume and x/y-transposed volume, the plan's box
  const void* vol;
  const ViewParams* views;     // the subset's views
  int* flags;
  GridConst gc;
  FwdOut o;
  int BZ, nsl_max;
  int tx, ty;                  // ray tiles per view (x, y)
  int base;                    // work-list index of the scan's first tile
};

// Tensor map of a volume (n0, n1, n2) with box b.
CUtensorMap make_volume_map(cbct_dtype dt, const void* vol, int n0, int n1, int n2, const SlabBox& b);

// Largest footprint of a slab of TS voxels over every view and tile of a TU x TV
// tiling, margins included; false when some view cannot use slabs.  beside: also over
// tiles and slabs whose rays pass beside the volume.
bool slab_extents(const cbct_plan* p, int TU, int TV, int TS, int& ext_e, int& ext_z, bool beside = false);

// Whether launches of element size es interpolate in the gather kernel's form (see
// LerpForm): the plan's rows or pixels are such that the gather kernel is the one that
// reads the caller's volume as it lies.
bool forward_lerp_gather(const cbct_plan* p, size_t es);

// Bound of a sample's element index counted from the volume's corner with box b's strides.
// Kernels form it as an exact FP32 sum: below 2^24, or below 2^22 in the mantissa of a
// sum biased by 1.5 * 2^23 whose box origin is taken off afterwards.
inline size_t box_index_bound(const cbct_geometry& g, const SlabBox& b) {
  return ((size_t)g.nz + 1) * b.bx * b.by + ((size_t)std::max(g.nx, g.ny) + 1) * (b.bx + 1);
}

// Slabs of TS voxels a ray can cross in the larger in-plane direction.
int forward_slabs(const cbct_geometry& g, int TS);

using FwdMultiKernel = void (*)(const FwdScanRec*, int, int, int*);
struct ForwardMulti {
  FwdMultiKernel kernel;       // work-list kernel of the plan's shape and box width
  int nsl, threads;
  size_t smem;
};

// Per-ray slab projector (forward_slab.cu).
void slab_tile(int& TU, int& TV);
bool slab_choose(cbct_plan* p);
void slab_prepare(const cbct_plan* p);
// vol: the caller's volume; volP: the copy TMA reads it from (or vol itself).
void slab_launch(cbct_plan* p, cbct_dtype dt, const void* vol, const void* volP, const void* volT, const FwdOut& o,
                 int first, int cnt, cudaStream_t st);
ForwardMulti slab_multi(const cbct_plan* p);

// Row-quad projector (forward_quad.cu).
enum QuadShape { kQuadWide = 0, kQuadWarp = 1, kQuadThin = 2, kQuadSkew = 3, kQuadShapes = 4 };
void quad_tile(int shape, int& TU, int& TV);
bool quad_choose(cbct_plan* p, double row_dz, bool forced);
void quad_prepare(const cbct_plan* p);
// vol: the caller's volume; volP: the copy TMA reads it from (or vol itself).
void quad_launch(cbct_plan* p, cbct_dtype dt, const void* vol, const void* volP, const void* volT, const FwdOut& o,
                 int first, int cnt, cudaStream_t st);

ForwardMulti quad_multi(const cbct_plan* p);

}  // namespace cbct
