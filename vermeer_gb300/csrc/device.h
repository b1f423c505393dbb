// device.h - device-side data layout of libvmr (shared by host and kernels).
//
// HBM layout of one mesh (all arrays 128-byte aligned, resident for the
// lifetime of the context):
//   static mesh
//     GNode   nodes[n_nodes]       128 B: the 24 child-box floats of qbvh.Node
//                                  as 6 float4 (minx,miny,minz,maxx,maxy,maxz
//                                  over the 4 children), children as int4,
//                                  split axes packed in one word
//     float4  tris[3*n_tris]       leaf order: v0,v1,v2 (w unused), 48 B per
//                                  triangle, so a leaf is one contiguous run
//   motion mesh
//     MNode   mnodes[n_mnodes]     32 B: children int4 + packed axes
//     float4  mboxes[keys][n][6]   96 B per node per key
//     float4  mtris[keys][3*n]     leaf-position order, per key
//     int32   elem[n]              leaf position -> reported ElemID
#pragma once
#include <cstdint>

#include "animdecomp.h"

#ifndef __CUDACC__
struct float4_host { float x, y, z, w; };
#endif

namespace vmr {

// Leaf code in GNode/MNode children: bit 31 set, bits 4..30 first element,
// bits 0..3 count-1.  -1 is an empty child.  The reference packs the first
// element into 23 bits (LeafBase, qbvh/qbvh.go:64); the device format keeps
// 27, the upload path checks that reference trees decode unchanged.
constexpr int32_t kEmptyChild = -1;

struct alignas(128) GNode {
  float box[24];        // box[c + 4*axis] = min, box[12 + c + 4*axis] = max
  int32_t child[4];
  uint32_t axes;        // axis0 | axis1<<2 | axis2<<4
  uint32_t rank[2];     // push rank of each child per ray octant: byte o
                        // (o = sign bits of D) holds rank(c) at bits 2c
  uint32_t pad;
};
static_assert(sizeof(GNode) == 128, "GNode must be 128 bytes");

// A static node as the rays of one direction octant read it (o = the sign
// bits of D): the children in push order (slot 0 pushed first, so slot 3 is
// visited first), and per child the near and far box planes of that octant
// instead of min and max, so a visit needs neither the min/max of each plane
// pair nor the rank arithmetic of the push.  A mesh holds one such array per
// octant (o * n_nodes + node): 8 x 128 B per node, about the size of the
// triangle table.  An absent child's planes are never hit (near +inf, far
// -inf along D).  A motion mesh holds the same per key ((o * keys + key) *
// n_nodes + node): the near planes of two keys lerp to the near plane at the
// ray's time, as the boxes of every key are ordered; its absent children are
// told by their code.
struct alignas(128) ONode {
  float slot[4][6];     // near x, near y, far x, far y, near z, far z
  int32_t child[4];
  uint32_t pad[4];
};
static_assert(sizeof(ONode) == 128, "ONode must be 128 bytes");

struct alignas(32) MNode {
  int32_t child[4];
  uint32_t axes;
  uint32_t rank[2];
  uint32_t pad;
};
static_assert(sizeof(MNode) == 32, "MNode must be 32 bytes");

// Where octant o's copy holds child c of a node, and the child there.
VMR_HD unsigned octant_slot(const uint32_t rank[2], unsigned c, unsigned o) {
  return (rank[o >> 2] >> (8u * (o & 3u) + 2u * c)) & 3u;
}
// Static: a plane pair given in the wrong order is put in order and a NaN plane
// takes the other's value, as the min and max of the products would; a child all
// of whose planes are NaN is never hit.
VMR_HD void octant_child(const GNode& N, unsigned c, unsigned o, ONode& r) {
  const float inf = INFINITY;
  const unsigned slot = octant_slot(N.rank, c, o);
  const int at_near[3] = {0, 1, 4}, at_far[3] = {2, 3, 5};
  float lo[3], hi[3];
  int nans = 0;
  for (int a = 0; a < 3; ++a) {
    const float mn = N.box[c + 4 * a], mx = N.box[12 + c + 4 * a];
    lo[a] = fminf(mn, mx);
    hi[a] = fmaxf(mn, mx);
    nans += lo[a] != lo[a] ? 1 : 0;
  }
  const bool absent = N.child[c] == kEmptyChild || nans == 3;
  for (int a = 0; a < 3; ++a) {
    const bool neg = (o >> a) & 1u;
    // absent: near +inf and far -inf along D, whichever way D points
    r.slot[slot][at_near[a]] = absent ? (neg ? -inf : inf) : (neg ? hi[a] : lo[a]);
    r.slot[slot][at_far[a]] = absent ? (neg ? inf : -inf) : (neg ? lo[a] : hi[a]);
  }
  r.child[slot] = N.child[c];
  r.pad[slot] = 0;
}
// Motion, one key's boxes (float[24], laid out as GNode::box); false when a
// present child has a plane out of order, a NaN or an infinity (0 * inf at a key is
// a NaN), where lerped near and far planes would not be the lerped box's: such a
// tree keeps to its mnodes.
VMR_HD bool octant_mchild(const MNode& N, const float* box, unsigned c, unsigned o, ONode& r) {
  const unsigned slot = octant_slot(N.rank, c, o);
  const int at_near[3] = {0, 1, 4}, at_far[3] = {2, 3, 5};
  bool ok = true;
  for (int a = 0; a < 3; ++a) {
    const float mn = box[c + 4 * a], mx = box[12 + c + 4 * a];
    const bool neg = (o >> a) & 1u;
    ok = ok && mn <= mx && mn > -INFINITY && mx < INFINITY;
    r.slot[slot][at_near[a]] = neg ? mx : mn;
    r.slot[slot][at_far[a]] = neg ? mn : mx;
  }
  r.child[slot] = N.child[c];
  r.pad[slot] = 0;
  return ok || N.child[c] == kEmptyChild;
}

// The octant copies a context may hold, of a device with total bytes of memory:
// a sixteenth, so a program that fills the device with geometry and workspaces of
// its own still finds room for them.  (They are the faster walk at any mesh size:
// 4,194,304 incoherent rays on 1, 2, 4 and 8.4 million triangles 7.10 -> 6.22, 7.62
// -> 6.80, 8.42 -> 7.61, 9.32 -> 8.46 ms, a million coherent ones 1.71 -> 1.43 to
// 1.94 -> 1.67, at 1.8 to 1.9 times the mesh's memory: 814 against 449 MB at most.)
constexpr bool octant_room(uint64_t held, uint64_t more, uint64_t total) { return held + more <= total / 16; }

// One mesh as the kernels see it.
struct DMesh {
  const GNode* nodes;       // static
  const ONode* onodes;      // [8][keys][n_nodes]; null: the kernels walk nodes / mnodes
  uint32_t n_nodes;
  uint32_t pad0;
  const void* tris;         // float4[3*n_tris] (static)
  const MNode* mnodes;      // motion
  const void* mboxes;       // float4[keys][n_mnodes][6]
  const void* mtris;        // float4[keys][3*n_tris]
  const int32_t* elem;      // motion: leaf position -> ElemID
  uint32_t n_tris;
  uint32_t n_mnodes;
  uint32_t keys;            // 1 = static
  float lower_static;       // EpsilonFloat32 + RayBias (trace.go:182)
  float ray_bias;           // motion lower bound (trace.go:612)
  uint32_t iter_cap;        // 4 * nodes + 2: a traversal pops each entry once
  uint32_t kind;            // kTriangles, kSphere, or kGroup
  float sphere[4];          // centre, radius
  uint32_t has_xf;          // PolyMesh.Transform: rays enter through xf_inv
  uint32_t xf_nkeys;        // >= 2: the transform is blended per ray from xf_keys
  uint32_t pad;
  // Matrix4Inverse of the transform, columns 0..3 rows 0..2 (column-major
  // elements 0,1,2, 4,5,6, 8,9,10, 12,13,14)
  float xf_inv[12];
  const anim::Decomp* xf_keys;  // decomposed transform keys (xf_nkeys >= 2)
  // kGroup (GeomInstance: group 1, Proc: group 2): the transform (has_xf /
  // xf_keys as above), the geoms traced in order and the geom id a hit in
  // each reports
  const uint32_t* children;
  const int32_t* child_hit;
  uint32_t n_children;
  uint32_t group;
};
enum MeshKind : uint32_t { kTriangles = 0, kSphere = 1, kGroup = 2 };

// Top level of a scene (builtin/scene): static GNodes or motion MNodes with
// boxes; leaves index geom_order (leaf position -> geom id).
struct DTop {
  const GNode* nodes;
  const ONode* onodes;      // as DMesh::onodes, of the top level
  uint32_t n_nodes;
  uint32_t pad0;
  const MNode* mnodes;
  const void* mboxes;
  const uint32_t* geom_order;
  const DMesh* meshes;      // indexed by geom id
  uint32_t keys;
  uint32_t n_mnodes;
  uint32_t n_geoms;
  uint32_t iter_cap;
  uint32_t all_static;  // static top level and only static meshes: the
                        // while-while scene kernel applies
  uint32_t simple_only; // instances, Procs or keyed transforms: the
                        // single-loop scene kernel only
};

struct RaySoA {
  const float *px, *py, *pz, *dx, *dy, *dz, *tmax, *time;
  // If set: the rays as two 16-byte records each, (px, py, pz, dx) and
  // (dy, dz, tmax, input index as bits), the key-ordered copy of a static
  // mesh trace (the arrays above are then unused; time is 0)
  const void* rec = nullptr;
};
struct HitSoA {
  int32_t* prim;
  int32_t* geom;
  float *t, *u, *v, *w;
};

// Device scratch of one context: the persistent kernels' work counter, the
// status word and the visit counters (reset before every launch).
struct DScratch {
  unsigned long long next_ray;
  int status;
  int pad;
  unsigned long long node_visits;
  unsigned long long leaf_visits;
  unsigned long long tri_tests;
};

enum DeviceStatus : int {
  kStatusOk = 0,
  kStatusStackOverflow = 1,
  kStatusIterationCap = 2,
};

constexpr int kStackCapacity = 90;  // RenderTask.Traversal.Stack (core/ray.go:158)

// Traversal kernel variants (vmr_tuning.kernel bits).
enum TraceKernel : int {
  kKernelScheduled = 0,
  kKernelWhileWhile = 1,
  kKernelPrefetch = 2,
  kKernelRegCap = 4,
  kKernelSort = 8,
  kKernelSharedStack = 16,  // while-while: the top of the stack in shared memory
  kKernelCoopLeaf = 32,     // while-while, static meshes: warp-cooperative leaf scan
};
constexpr int kSharedStackEntries = 16;

// Ray reordering (raysort.cu): 6 permutation classes x (2^b)^3 origin cells,
// b = 3..5, x the octant of the class's other two signs for b <= 4.
constexpr int kSortMaxBits = 5;
constexpr int kSortOctantBits = 4;
constexpr int kSortBucketsMax = 2 * (6 << (3 * kSortMaxBits));  // the histogram, then its scan
constexpr uint32_t sort_buckets(int bits) { return (6u << (3 * bits)) * (bits <= kSortOctantBits ? 4u : 1u); }
// The width a tuning of 0 takes: 16^3 cells, or 8^3 for batches in which that
// many buckets (98,304) hold a few rays each.  The two are within 2% of each other
// from 65,536 to 1.5 million rays: 8^3 is 0.4 to 1.8% ahead for scenes up to 800,000
// rays (300,007: 247 against 252 us; 1,000,003: 463 against 453; 3,000,000: 1,132
// against 1,087), 16^3 0.5 to 1.3% for meshes from 300,000 (300,007: 619 against 615
// us; 65,536: 348 against 351).
constexpr int default_sort_bits(uint64_t n) { return n < 700000u ? 3 : 4; }
constexpr uint64_t kSortMinRays = 1u << 16;  // smaller batches are traced unsorted

// Launch entry points (traverse.cu).
struct TraceLaunch {
  RaySoA rays;
  HitSoA hits;
  const uint32_t* order;  // rays[i] is input ray order[i] (nullptr: identity)
  uint64_t n;
  const unsigned long long* n_dev;  // if set, the ray count is read from device
                                    // memory when the kernel starts (wavefront
                                    // queues; n is then a capacity); scene
                                    // traces and the while-while mesh kernels
  int any_hit;
  int count;
  DScratch* scratch;
  int grid;             // resident blocks per SM wanted (0 = occupancy maximum)
  int block;
  int kernel;
  int refill_min;
  int walk_tail;
  void* stream;
  // scene traces in job mode (batched renders): no top level; ray i enters
  // mesh path_geom[ray_path[i]] directly (both set or both null)
  const uint32_t* ray_path;
  const uint32_t* path_geom;
};
int launch_trace_mesh(const DMesh& mesh, const TraceLaunch& l);
// n_dev (optional): the ray count on the device, at most n (a wavefront queue
// length); the grid is sized for n.  sorted_out.rec set: the key-ordered copy
// is written as records (RaySoA::rec, 32 bytes a ray) and order is not
// written; else as arrays, with order[i] = the input index of position i.
int launch_ray_sort(const RaySoA& rays, uint64_t n, const float bounds[6], int bits, uint32_t* keys, uint32_t* hist,
                    uint32_t* order, const RaySoA& sorted_out, void* stream,
                    const unsigned long long* n_dev = nullptr);
// n rays of 8 floats (16-byte aligned device memory) -> out's eight arrays.
int launch_ray_columns(const float* rows, uint64_t n, const RaySoA& out, void* stream);
int launch_trace_scene(const DTop& top, const TraceLaunch& l);
// out[8][n]: the octant copies of n nodes (octant.cu).
int launch_octant_nodes(const GNode* nodes, uint32_t n, ONode* out, void* stream);
// out[8][keys][n] of n motion nodes; *bad is set when the tree keeps to its mnodes
// (octant_mchild).
int launch_octant_mnodes(const MNode* nodes, const void* mboxes, uint32_t keys, uint32_t n, ONode* out, int* bad,
                         void* stream);
int device_sm_count();

// One job of a batched trace (vmr_trace_jobs): its rays and hits (device
// SoA, its own buffers) and its first position in the gathered ray stream.
struct JobDesc {
  RaySoA rays;
  HitSoA hits;
  uint64_t n;
  uint64_t ray0;  // the job's first position in the gathered ray stream
};
// Gathered rays and hits of a batched trace, the per-ray job index and the
// job -> geom table (the scene kernel's job mode reads job_geom[ray_job[i]]).
struct JobWork {
  RaySoA rays;
  HitSoA hits;
  uint32_t* ray_job;
  uint32_t* job_geom;
};
// l: the launch settings (stream, kernel, walk tail, scratch, any_hit); top:
// the mesh table indexed by geom id (keys = 1, no top level).
int launch_trace_jobs(const JobDesc* jobs, uint32_t n_jobs, uint64_t n_rays, const DTop& top, const JobWork& w,
                      TraceLaunch l);

}  // namespace vmr
