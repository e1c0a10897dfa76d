/*
 * scene_host.h -- host-side scene (src/scene.zig) with its binned-SAH BVH
 * (src/bvh.zig) and emitter table (src/light.zig), plus the flattening into
 * the device layout of zt_types.h.
 */
#ifndef ZT_SCENE_HOST_H
#define ZT_SCENE_HOST_H

#include <math.h>
#include <stdlib.h>
#include <sys/mman.h>

#include <new>
#include <string>
#include <utility>
#include <vector>

#include "../../include/zigtrace_b200.h"
#include "zt_types.h"

struct zt_device_buffers;
struct zt_device_tree;  /* defined by the CUDA side */
struct zt_host_staging;    /* pinned flattened copy, defined by the CUDA side */

namespace zt {

/* Allocator of the scene's large arrays (shapes, nodes, permutation).  From
 * 4 MB up they lie on huge pages where the system grants them on request
 * (MADV_HUGEPAGE), and elements added by resize are left uninitialised: the
 * caller fills them.  A fresh 82 MB array of a million shapes otherwise costs
 * 20,000 page faults when it is filled and as many pages to give back: adding
 * the shapes, receiving the nodes and freeing both took 89 ms, with this and
 * the copies on several threads 10 ms. */
template <typename T>
struct ArrayAllocator {
  using value_type = T;
  ArrayAllocator() = default;
  template <typename U>
  ArrayAllocator(const ArrayAllocator<U>&) {}
  T* allocate(size_t n) {
    constexpr size_t huge = 2u << 20;
    if (n > SIZE_MAX / sizeof(T)) throw std::bad_alloc();
    const size_t bytes = n * sizeof(T);
    void* p;
    if (bytes < 2 * huge) {
      p = malloc(bytes > 0 ? bytes : 1);
    } else {
      if (bytes > SIZE_MAX - huge) throw std::bad_alloc();
      p = aligned_alloc(huge, (bytes + huge - 1) / huge * huge);
      if (p) madvise(p, bytes, MADV_HUGEPAGE); /* a hint: failing costs only time */
    }
    if (!p) throw std::bad_alloc();
    return static_cast<T*>(p);
  }
  void deallocate(T* p, size_t) { free(p); }
  template <typename U>
  void construct(U* p) {
    ::new (static_cast<void*>(p)) U;
  }
  template <typename U, typename... A>
  void construct(U* p, A&&... a) {
    ::new (static_cast<void*>(p)) U(std::forward<A>(a)...);
  }
  template <typename U>
  bool operator==(const ArrayAllocator<U>&) const { return true; }
  template <typename U>
  bool operator!=(const ArrayAllocator<U>&) const { return false; }
};
template <typename T>
using Array = std::vector<T, ArrayAllocator<T>>;

struct HostNode {  /* Bvh.Node, bvh.zig:22-33 */
  double bmin[3], bmax[3];
  uint32_t first, count;
};

struct HostLight {  /* Light, light.zig:30-35 */
  zt_shape shape;
  double radiance[3];
  double weight;
};

/* Flattened arrays in the device layout (zt_types.h). */
struct FlatScene {
  std::vector<DPrim> prims;
  std::vector<int32_t> prim_ids;
  std::vector<DPair> pairs;
  std::vector<FPair> fpairs; /* conservative float copy of pairs (empty when the fast traversal cannot be used) */
  std::vector<DPrim> planes;
  std::vector<DMat> mats;
  std::vector<DLight> lights;
  std::vector<FLight> flights;
  std::vector<double> cdf;
  double fast_eps[3]; /* margins of the float records */
  DevScene view;  /* pointers unset; counts, root, total, background set */
};

}  // namespace zt

struct zt_scene {
  std::vector<zt_material> materials;
  zt::Array<zt_shape> shapes;    /* bounded, insertion order */
  std::vector<zt_shape> planes;  /* unbounded, insertion order */
  zt_camera_config camera;
  zt_background background;
  bool built = false;
  zt::Array<zt::HostNode> nodes;
  zt::Array<uint32_t> indices;
  bool boxes_nested = false;  /* every node's box holds its children's and its primitives' boxes */
  double leaf_extent[3] = {INFINITY, INFINITY, INFINITY}; /* of the leaves' boxes, about: geometric means */
  bool leaves_ordered = false; /* a left child's primitives come right before its sibling's in `indices` */
  std::vector<zt::HostLight> lights;
  std::vector<double> cdf;
  double total = 0;
  zt_device_buffers* device = nullptr;  /* resident copy, owned */
  bool pilot_valid = false;             /* mean_path is current for this build, camera and background */
  double mean_path = 0;                 /* mean path length of the pilot that ZT_MODE_AUTO reads */
  zt_host_staging* staging = nullptr;   /* pinned flattened copy, owned */
  zt_device_tree* device_tree = nullptr; /* shapes and tree left on the device by a device build, owned */
  bool uploaded = false;                /* since the last build */
  uint64_t primal_cache_limit = 1ull << 30; /* bytes zt_forward may keep for zt_backward */
};

namespace zt {

void set_error(const std::string& msg);
zt_status fail(zt_status code, const std::string& msg);

/* Scene.build (scene.zig:92-96); with device = true the BVH is built on the
 * current CUDA device when it can be (see device_build_bvh), else on the
 * host.  *used_device tells which. */
zt_status build_scene(zt_scene* s, bool device = false, bool* used_device = nullptr, double* build_ms = nullptr);
/* Bvh.build on the current CUDA device (bvh_build.cu): the same nodes and
 * indices as the host build.  Returns ZT_DEVICE_BUILD_FALLBACK for input
 * the device build leaves to the host (splitMedian nodes, non-finite
 * boxes). */
constexpr zt_status ZT_DEVICE_BUILD_FALLBACK = 1;
zt_status device_build_bvh(zt_scene* s, double* build_ms);
/* Camera.init (camera.zig:29-55) for the given aspect ratio. */
DCamera camera_init(const zt_camera_config& cfg, double aspect);
/* Flattens a built scene into the device layout.  with_tree = false leaves
 * prims, prim_ids, pairs and fpairs empty for the device to fill
 * (flatten_on_device, bvh_build.cu) and sets the view's root and the float
 * records' root and margins (fast_eps) as far as the root box decides them. */
void flatten_scene(const zt_scene* s, FlatScene* out, bool with_tree = true);
/* Writes to every page of [p, p + bytes), from several threads where it is
 * large. */
void touch_pages(void* p, size_t bytes);
/* Shapes, permutation and nodes of a scene in device memory. */
struct DeviceTree {
  const zt_shape* shapes;
  const uint32_t* indices;
  const HostNode* nodes;
};
/* Drops what a device build left on the device. */
void release_device_tree(zt_scene* s);
/* The tree a device build left on the current device, if it did. */
bool device_tree(const zt_scene* s, DeviceTree* out);
/* Fills the tree's part of the device layout from t on the legacy default
 * stream: the same bytes as flatten_scene's.  fpairs may be NULL; ordered:
 * the scene's leaves_ordered.
 * *max_leaf: the largest leaf; *nan: a primitive holds a NaN. */
zt_status flatten_on_device(const DeviceTree& t, uint32_t n_prims, uint32_t n_nodes, const double eps[3], bool ordered,
                            DPrim* prims, int32_t* ids, DPair* pairs, FPair* fpairs, uint32_t* max_leaf, bool* nan);
/* Drops the resident device copy (implemented with the CUDA code). */
void release_device(zt_scene* s);
/* Drops the device copy and the pinned staging copy (scene changed). */
void release_staging(zt_scene* s);

}  // namespace zt

#endif
