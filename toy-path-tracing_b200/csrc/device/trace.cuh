// Two-level 4-wide BVH traversal on the device, one ray per thread.
//
// Semantics follow the reference exactly (bit-for-bit on the same tree):
//  - slab test of qbvh.rs:578-607 with SSE minps/maxps NaN rules; rays whose
//    reciprocal direction has an infinite lane take the exact select path,
//    all others the cheaper fminf/fmaxf path (identical when no NaN can arise);
//  - per node, hit lanes are ordered by entry distance (stable), leaves are
//    visited far-to-near and interior nodes pushed so the nearest pops first
//    (qbvh.rs:640-671).  Leaves are pushed onto the stack above the interior
//    children, which gives the same leaf order and the same t_max for every
//    later box test as calling them in place;
//  - TLAS leaves expand to instance markers; an instance marker transforms the
//    ray (glam Mat4::transform_point3/_vector3 order) and traverses its BLAS
//    with the shared running t_max (scene/mod.rs:340-395, 686-723);
//  - pbrt-v4 watertight triangle test with the f64 fallback (math/ray.rs:107-209);
//    ties on t keep the later-tested triangle;
//  - closest_mesh_hit_with_filter's alpha test (scene/mod.rs:360-377, 686-723):
//    when the caller passes an AuxRng state, a candidate hit on an instance
//    whose material has an alpha test draws u from it (aux_rng.rs:21-28) and
//    is kept iff u < the material's opacity, in the candidates' test order.
// The library is compiled with -fmad=false so that no multiply-add is fused
// unless written as fmaf (the reference's `mul_add`).
//
// What bounds it is not DRAM (the tree is L2-resident) but the L1 data pipe and
// then the issue slots: lanes of incoherent rays read different nodes, and a
// lane's load takes one cycle of the SM's load pipe whether it is 16 or 32 bytes
// wide (measured: 7 x 16 B = 6.9 cycles per node and lane, 3 x 32 + 16 B = 3.9).
// Hence 32-byte loads: four per node instead of seven, two per triangle instead
// of three.  For the issue slots: packed two-lane subtracts and multiplies,
// three-input min/max, and a branch-free ranking of the children.
//
// Every index that goes to memory is clamped to the scene's arrays (nodes,
// triangles, instances).  The upload has checked the trees and a stack entry is
// written before it is read, so no clamp changes an index; they make a read outside
// the scene impossible whatever a ray or a word of the stack holds.  As minimum
// instructions they cost nothing (2^24 incoherent rays 5.87 -> 5.85 ms, Cornell box
// 1.88 -> 1.89, 2.1M-triangle scene 3.52 -> 3.53); as tests with an error flag 1-2 %.
#pragma once
#include "dev_types.cuh"

namespace tpt {

__device__ __forceinline__ float safe_inv(float d) { return d == 0.0f ? __int_as_float(0x7f800000) : 1.0f / d; }

// Per-(local-)ray data reused by every box and triangle test.
struct RayPre {
  float ox, oy, oz;     // origin
  float ix, iy, iz;     // safe reciprocal direction
  float sx, sy, sz;     // shear constants of the watertight test
  int kz;               // axis of the largest |d| component; x, y follow it cyclically
  bool exact;           // an infinite reciprocal lane: use select min/max
  bool no_tri;          // permuted d.z == 0: no triangle can be hit
  bool tris_ready;      // sx, sy, sz, kz and no_tri are set; before, (sx, sy, sz) is the direction
};

// (kx, ky, kz) components, kx = kz + 1 and ky = kz + 2 modulo 3
__device__ __forceinline__ void permute3(float x, float y, float z, int kz, float& px, float& py, float& pz) {
  px = kz == 0 ? y : (kz == 1 ? z : x);
  py = kz == 0 ? z : (kz == 1 ? x : y);
  pz = kz == 0 ? x : (kz == 1 ? y : z);
}

// A ray's setup comes in two parts, each made where it is first read: the
// reciprocals for box tests (an instance whose tree is a single leaf has none, and
// the world ray needs them back only for a TLAS node), and the permutation and
// shear for triangle tests (most instances a ray enters show it no leaf).  Each
// part is three divisions.
__device__ __forceinline__ void ray_setup_boxes(RayPre& r, float dx, float dy, float dz) {
  r.ix = safe_inv(dx); r.iy = safe_inv(dy); r.iz = safe_inv(dz);
  // NaN can only come from 0 * inf in (b - o) * inv, i.e. from a reciprocal
  // lane that is infinite (or zero, for an infinite direction component).
  r.exact = !(isfinite(r.ix) && isfinite(r.iy) && isfinite(r.iz) && r.ix != 0.0f && r.iy != 0.0f && r.iz != 0.0f);
}
// The direction waits in (sx, sy, sz) until then.
__device__ __forceinline__ void ray_setup_tris(RayPre& r) {
  const float dx = r.sx, dy = r.sy, dz = r.sz;
  const float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
  r.kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);  // math/mod.rs:148-156
  float pdx, pdy, pdz;
  permute3(dx, dy, dz, r.kz, pdx, pdy, pdz);
  r.no_tri = (pdz == 0.0f);
  r.sx = -pdx / pdz;
  r.sy = -pdy / pdz;
  r.sz = 1.0f / pdz;
  r.tris_ready = true;
}

__device__ __forceinline__ float dop(float a, float b, float c, float d) {
  float cd = c * d;
  float e = fmaf(a, b, -cd);
  float err = fmaf(-c, d, cd);
  return e + err;
}

// math/ray.rs:107-209 with the ray-only work hoisted into RayPre.
__device__ __forceinline__ bool tri_test(const RayPre& r, float t_max, const DevTri& tri, float& t_out, float& b0,
                                         float& b1, float& b2) {
  // degenerate flag precomputed on the host with the reference's formula
  if (tri.v1.w != 0.0f || r.no_tri) return false;
  // permute, then translate: each component's subtraction as the reference's
  float ox, oy, oz, p0x, p0y, p0z, p1x, p1y, p1z, p2x, p2y, p2z;
  permute3(r.ox, r.oy, r.oz, r.kz, ox, oy, oz);
  permute3(tri.v0.x, tri.v0.y, tri.v0.z, r.kz, p0x, p0y, p0z);
  permute3(tri.v1.x, tri.v1.y, tri.v1.z, r.kz, p1x, p1y, p1z);
  permute3(tri.v2.x, tri.v2.y, tri.v2.z, r.kz, p2x, p2y, p2z);
  p0x -= ox; p0y -= oy; p0z -= oz;
  p1x -= ox; p1y -= oy; p1z -= oz;
  p2x -= ox; p2y -= oy; p2z -= oz;
  p0x = p0x + r.sx * p0z; p0y = p0y + r.sy * p0z;
  p1x = p1x + r.sx * p1z; p1y = p1y + r.sy * p1z;
  p2x = p2x + r.sx * p2z; p2y = p2y + r.sy * p2z;
  float e0 = dop(p1x, p2y, p1y, p2x);
  float e1 = dop(p2x, p0y, p2y, p0x);
  float e2 = dop(p0x, p1y, p0y, p1x);
  if (e0 == 0.0f || e1 == 0.0f || e2 == 0.0f) {
    e0 = (float)((double)p2y * (double)p1x - (double)p2x * (double)p1y);
    e1 = (float)((double)p0y * (double)p2x - (double)p0x * (double)p2y);
    e2 = (float)((double)p1y * (double)p0x - (double)p1x * (double)p0y);
  }
  if ((e0 < 0.0f || e1 < 0.0f || e2 < 0.0f) && (e0 > 0.0f || e1 > 0.0f || e2 > 0.0f)) return false;
  float det = e0 + e1 + e2;
  if (det == 0.0f) return false;
  p0z = p0z * r.sz; p1z = p1z * r.sz; p2z = p2z * r.sz;
  float ts = e0 * p0z + e1 * p1z + e2 * p2z;
  if ((det < 0.0f && (ts >= 0.0f || ts < t_max * det)) || (det > 0.0f && (ts <= 0.0f || ts > t_max * det)))
    return false;
  float inv_det = 1.0f / det;
  float t = ts * inv_det;
  const float eps = 5.9604644775390625e-08f;  // f32::EPSILON / 2
  const float g2 = (2.0f * eps) / (1.0f - 2.0f * eps);
  const float g3 = (3.0f * eps) / (1.0f - 3.0f * eps);
  const float g5 = (5.0f * eps) / (1.0f - 5.0f * eps);
  float max_zt = fmaxf(fmaxf(fabsf(p0z), fabsf(p1z)), fabsf(p2z));
  float delta_z = g3 * max_zt;
  float max_xt = fmaxf(fmaxf(fabsf(p0x), fabsf(p1x)), fabsf(p2x));
  float max_yt = fmaxf(fmaxf(fabsf(p0y), fabsf(p1y)), fabsf(p2y));
  float delta_x = g5 * (max_xt + max_zt);
  float delta_y = g5 * (max_yt + max_zt);
  float delta_e = 2.0f * (g2 * max_xt * max_yt + delta_y * max_xt + delta_x * max_yt);
  float max_e = fmaxf(fmaxf(fabsf(e0), fabsf(e1)), fabsf(e2));
  float delta_t = 3.0f * (g3 * max_e * max_zt + delta_e * max_zt + delta_z * max_e) * fabsf(inv_det);
  if (t <= delta_t) return false;
  t_out = t;
  b0 = e0 * inv_det; b1 = e1 * inv_det; b2 = e2 * inv_det;
  return true;
}

// One 32-byte read-only load (32-byte aligned).
__device__ __forceinline__ void ldg32(const void* p, float (&v)[8]) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
      : "l"(p));
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// (b[k] - o) * i for the four lanes of a plane vector, two lanes per
// instruction; each rounds as the scalar subtract and multiply do (b - o is
// b + (-o)).
__device__ __forceinline__ void slab4(const float* b, float o, float i, float (&t)[4]) {
  asm("{\n\t"
      ".reg .b64 p, q, n, m;\n\t"
      "mov.b64 p, {%4, %5};\n\t"
      "mov.b64 q, {%6, %7};\n\t"
      "mov.b64 n, {%8, %8};\n\t"
      "mov.b64 m, {%9, %9};\n\t"
      "add.rn.f32x2 p, p, n;\n\t"
      "add.rn.f32x2 q, q, n;\n\t"
      "mul.rn.f32x2 p, p, m;\n\t"
      "mul.rn.f32x2 q, q, m;\n\t"
      "mov.b64 {%0, %1}, p;\n\t"
      "mov.b64 {%2, %3}, q;\n\t"
      "}"
      : "=f"(t[0]), "=f"(t[1]), "=f"(t[2]), "=f"(t[3])
      : "f"(b[0]), "f"(b[1]), "f"(b[2]), "f"(b[3]), "f"(-o), "f"(i));
}

// Slab test of one 4-wide node: returns the lane hit mask, lane entry
// distances in tmin[], child words in ch[].
__device__ __forceinline__ uint32_t box4(const DevNode* __restrict__ n, const RayPre& r, float t_max, float tmin[4],
                                         uint32_t ch[4]) {
  float q0[8], q1[8], q2[8];  // lo_x lo_y | lo_z hi_x | hi_y hi_z
  ldg32(&n->lo_x, q0);
  ldg32(&n->lo_z, q1);
  ldg32(&n->hi_y, q2);
  const uint4 c = __ldg(&n->child);
  ch[0] = c.x; ch[1] = c.y; ch[2] = c.z; ch[3] = c.w;
  float t1x[4], t1y[4], t1z[4], t2x[4], t2y[4], t2z[4];
  slab4(q0, r.ox, r.ix, t1x);
  slab4(q0 + 4, r.oy, r.iy, t1y);
  slab4(q1, r.oz, r.iz, t1z);
  slab4(q1 + 4, r.ox, r.ix, t2x);
  slab4(q2, r.oy, r.iy, t2y);
  slab4(q2 + 4, r.oz, r.iz, t2z);
  uint32_t mask = 0;
  if (!r.exact) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const float a = fmaxf(max3f(fminf(t1x[s], t2x[s]), fminf(t1y[s], t2y[s]), fminf(t1z[s], t2z[s])), 0.0f);
      const float b = fminf(min3f(fmaxf(t1x[s], t2x[s]), fmaxf(t1y[s], t2y[s]), fmaxf(t1z[s], t2z[s])), t_max);
      tmin[s] = a;
      // lanes whose child word decodes to Empty (leaf bit, zero count) never count
      if (a <= b && (ch[s] >> 24) != 0x80u) mask |= 1u << s;
    }
  } else {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const float mnx = t1x[s] < t2x[s] ? t1x[s] : t2x[s], mxx = t1x[s] > t2x[s] ? t1x[s] : t2x[s];
      const float mny = t1y[s] < t2y[s] ? t1y[s] : t2y[s], mxy = t1y[s] > t2y[s] ? t1y[s] : t2y[s];
      const float mnz = t1z[s] < t2z[s] ? t1z[s] : t2z[s], mxz = t1z[s] > t2z[s] ? t1z[s] : t2z[s];
      float a = mnx > mny ? mnx : mny; a = a > mnz ? a : mnz; a = a > 0.0f ? a : 0.0f;
      float b = mxx < mxy ? mxx : mxy; b = b < mxz ? b : mxz; b = b < t_max ? b : t_max;
      tmin[s] = a;
      if (a <= b && (ch[s] >> 24) != 0x80u) mask |= 1u << s;
    }
  }
  return mask;
}

// Triangle g (index over all meshes) of the paired records: two loads, of 32 and
// 16 bytes.
__device__ __forceinline__ DevTri load_tri(const DevTriPair* __restrict__ tris, uint32_t g) {
  const DevTriPair* p = tris + (g >> 1);
  float q[8];
  ldg32(&p->v01[g & 1u][0], q);
  DevTri t;
  t.v0 = make_float4(q[0], q[1], q[2], q[3]);
  t.v1 = make_float4(q[4], q[5], q[6], q[7]);
  t.v2 = __ldg(&p->v2[g & 1u]);
  return t;
}

struct TraceResult {
  float t;
  int32_t tri;
  int32_t inst;
  float b0, b1, b2;
};

struct TraceCounters {
  uint32_t nodes;
  uint32_t tris;
};

// Per-thread traversal stack: the first SH entries live in shared memory
// (entry k of thread i at base[k * STRIDE], bank-conflict free; STRIDE is the
// block size), deeper entries in a local-memory spill area.  Total depth
// kStackDepth (qbvh.rs:609).
template <int SH, int STRIDE>
struct SplitStack {
  static constexpr int kShared = SH, kStride = STRIDE;
  uint32_t* sh;
  uint32_t spill[kStackDepth - SH];
  __device__ __forceinline__ void set(int k, uint32_t v) {
    if (k < SH) sh[k * STRIDE] = v;
    else spill[k - SH] = v;
  }
  __device__ __forceinline__ uint32_t get(int k) const { return k < SH ? sh[k * STRIDE] : spill[k - SH]; }
};

// Stack entries: interior node (bit 31 clear), BLAS/TLAS leaf (bit 31, count
// >= 1), instance marker (bit 31, count 0, instance id), or kNone.  kNone can
// never be a real leaf word: the upload rejects leaf ranges past 2^24.
constexpr uint32_t kNone = 0xFFFFFFFFu;

// Traversal of one ray, advanced one entry at a time.  `next` holds the entry
// to process next (the would-be top of the stack kept in a register).
struct TravState {
  float wox, woy, woz, wdx, wdy, wdz;  // world-space ray
  RayPre r;                            // ray of the current level (world at the TLAS, instance space in a BLAS)
  float closest;                       // running t_max
  TraceResult res;                     // all but t, which hit_distance() gives
  uint32_t next;
  int sp, floor_sp;
  bool in_blas;
  bool boxes_ready;                    // the current level's ray is set up for box tests
  uint32_t node_base;                  // first node of the current level (TLAS or BLAS)
  uint32_t tri_base, inst_id;
  // ALPHA instantiations only
  bool alpha_on;                       // the scene has alpha tests
  float alpha;                         // the current instance's opacity (1: no test)
  uint32_t aux;                        // AuxRng state
};

// The hit's distance (+inf: no hit): the running t_max of the last accepted hit.
__device__ __forceinline__ float hit_distance(const TravState& s) {
  return s.res.tri >= 0 ? s.closest : __int_as_float(0x7f800000);
}

// AuxRng::next_f32 (aux_rng.rs:21-28)
__device__ __forceinline__ float aux_next_f32(uint32_t& state) {
  state = state * 747796405u + 2891336453u;
  uint32_t s = state;
  s ^= s >> (4u + (s >> 28));
  s *= 277803737u;
  s ^= s >> 22;
  return (float)(s >> 8) * (1.0f / 16777216.0f);
}

// Enter instance `id`'s BLAS with the ray transformed by world_to_local
// (glam Mat4::transform_point3 / transform_vector3 order), scene/mod.rs:357.
template <bool ALPHA>
__device__ __forceinline__ void enter_instance(const DevGeometry& G, TravState& s, uint32_t id) {
  s.inst_id = id;
  if (ALPHA) s.alpha = s.alpha_on ? __ldg(G.inst_alpha + id) : 1.0f;
  const DevInstance* I = G.instances + id;
  float q0[8], q1[8];
  ldg32(&I->m0, q0);
  ldg32(&I->m2, q1);
  const float4 m0 = make_float4(q0[0], q0[1], q0[2], q0[3]), m1 = make_float4(q0[4], q0[5], q0[6], q0[7]);
  const float4 m2 = make_float4(q1[0], q1[1], q1[2], q1[3]);
  const float ox = s.wox, oy = s.woy, oz = s.woz, dx = s.wdx, dy = s.wdy, dz = s.wdz;
  float lox = m0.x * ox, loy = m0.y * ox, loz = m0.z * ox;
  lox = m0.w * oy + lox; loy = m1.x * oy + loy; loz = m1.y * oy + loz;
  lox = m1.z * oz + lox; loy = m1.w * oz + loy; loz = m2.x * oz + loz;
  lox = m2.y + lox; loy = m2.z + loy; loz = m2.w + loz;
  float ldx = m0.x * dx, ldy = m0.y * dx, ldz = m0.z * dx;
  ldx = m0.w * dy + ldx; ldy = m1.x * dy + ldy; ldz = m1.y * dy + ldz;
  ldx = m1.z * dz + ldx; ldy = m1.w * dz + ldy; ldz = m2.x * dz + ldz;
  s.r.ox = lox; s.r.oy = loy; s.r.oz = loz;
  s.r.sx = ldx; s.r.sy = ldy; s.r.sz = ldz;
  s.r.tris_ready = false;
  s.node_base = __float_as_uint(q1[4]);
  s.tri_base = __float_as_uint(q1[5]);
  s.in_blas = true;
  s.floor_sp = s.sp;
  s.next = __float_as_uint(q1[6]);
  s.boxes_ready = !(s.next & kLeafBit);
  if (s.boxes_ready) ray_setup_boxes(s.r, ldx, ldy, ldz);
}

template <class Stack>
__device__ __forceinline__ void trav_pop(const DevGeometry& G, TravState& s, Stack& st) {
  if (s.sp == 0) {
    s.next = kNone;
    return;
  }
  if (s.in_blas && s.sp == s.floor_sp) {
    // the instance's BLAS is done: back to the TLAS with the world ray
    s.in_blas = false;
    s.node_base = G.tlas_node_base;
    s.boxes_ready = false;
  }
  s.next = st.get(--s.sp);
  if (!s.boxes_ready && !(s.next & kLeafBit)) {  // a TLAS node after an instance
    s.r.ox = s.wox; s.r.oy = s.woy; s.r.oz = s.woz;
    ray_setup_boxes(s.r, s.wdx, s.wdy, s.wdz);
    s.boxes_ready = true;
  }
}

// ALPHA: the caller has AuxRng states (aux: the ray's, NULL = none), which the
// alpha tests of the scene's materials advance; without, no alpha test is made.
template <bool ALPHA>
__device__ __forceinline__ void trav_init(const DevGeometry& G, TravState& s, float ox, float oy, float oz, float dx,
                                          float dy, float dz, float t_max, const uint32_t* aux) {
  if (ALPHA) {
    s.alpha_on = aux != nullptr && G.inst_alpha != nullptr;
    s.aux = aux ? *aux : 0u;
    s.alpha = 1.0f;
  }
  s.wox = ox; s.woy = oy; s.woz = oz; s.wdx = dx; s.wdy = dy; s.wdz = dz;
  s.closest = t_max;
  s.res.tri = -1;
  s.res.inst = -1;
  s.res.b0 = s.res.b1 = s.res.b2 = 0.0f;
  s.in_blas = false;
  s.floor_sp = 0;
  s.sp = 0;
  s.node_base = G.tlas_node_base;
  s.tri_base = s.inst_id = 0;
  s.next = kNone;
  if (G.num_instances == 0) return;
  const uint32_t root = G.tlas_root_word;
  if ((root & kLeafBit) && ((root >> 24) & 0x7Fu) == 1u) {
    // TLAS is a single-instance root leaf (qbvh.rs:615-620): go straight to it
    enter_instance<ALPHA>(G, s, __ldg(G.tlas_prims + (root & 0xFFFFFFu)));
  } else {
    s.r.ox = ox; s.r.oy = oy; s.r.oz = oz;
    ray_setup_boxes(s.r, dx, dy, dz);
    s.boxes_ready = true;
    s.next = root;
  }
}

// Processes the interior node in `next`.  The hit children end up, bottom to
// top, as interiors far-to-near then leaves near-to-far (qbvh.rs:640-671: leaves
// are handled far-to-near at once, the nearest interior is popped first); the
// would-be top becomes `next`, the rest go to the stack.
//
// A child's key orders the hit children as they will be popped: leaves first,
// far to near (the complemented distance, negative), then interiors near to
// far (the distance's bits).  On equal distances the lower lane is the nearer
// (stable order): it comes first among interiors and last among leaves, which
// the +1 of an interior's right-hand key expresses.  Ranks from the six
// comparisons place every child without branches, so the lanes of a warp stay
// together: 13.8 instead of 10.7 active lanes per instruction and 17.0 instead
// of 23.4 warp instructions per node test on incoherent rays.
template <bool STATS, class Stack>
__device__ __forceinline__ void node_step(const DevGeometry& G, TravState& s, Stack& st, TraceCounters& cnt,
                                          uint32_t* err) {
  const DevNode* n = G.nodes + min(s.node_base + s.next, G.num_nodes - 1u);
  if (STATS) cnt.nodes++;
  float tmin[4];
  uint32_t ch[4];
  const uint32_t mask = box4(n, s.r, s.closest, tmin, ch);
  const int nh = __popc(mask);
  if (nh == 0) {
    trav_pop(G, s, st);
    return;
  }
  int key[4], right[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int leaf = (int)ch[i] >> 31;  // all ones for a leaf
    const int k = (__float_as_int(tmin[i]) & 0x7fffffff) ^ leaf;
    key[i] = (mask >> i) & 1u ? k : 0x7ffffffe;  // not hit: behind every hit
    right[i] = key[i] + 1 + leaf;
  }
  const bool c01 = key[0] < right[1], c02 = key[0] < right[2], c03 = key[0] < right[3];
  const bool c12 = key[1] < right[2], c13 = key[1] < right[3], c23 = key[2] < right[3];
  const int rank[4] = {3 - c01 - c02 - c03, 2 + c01 - c12 - c13, 1 + c02 + c12 - c23, 0 + c03 + c13 + c23};
  const int top = s.sp + nh - 1;  // entries on the stack afterwards
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (rank[i] == 0) s.next = ch[i];
  if (top <= Stack::kShared) {
    uint32_t* base = st.sh + top * Stack::kStride;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (rank[i] > 0 && rank[i] < nh) base[-rank[i] * Stack::kStride] = ch[i];
  } else {
    if (top > kStackDepth) {
      atomicOr(err, kDevErrStackOverflow);
      s.sp = 0;
      s.next = kNone;
      return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (rank[i] > 0 && rank[i] < nh) st.set(top - rank[i], ch[i]);
  }
  s.sp = top;
}

// Processes the leaf, TLAS leaf or instance marker in `next`.
template <int MODE, bool STATS, bool ALPHA, class Stack>
__device__ __forceinline__ void leaf_step(const DevGeometry& G, TravState& s, Stack& st, TraceCounters& cnt,
                                          uint32_t* err) {
  const uint32_t w = s.next;
  const uint32_t count = (w >> 24) & 0x7Fu, off = w & 0xFFFFFFu;
  if (s.in_blas) {
    // BLAS leaf: triangles in leaf order, t_max shrinking on each hit
    uint32_t g = s.tri_base + off;
    const uint32_t end = min(g + count, G.num_tris);
    if (!s.r.tris_ready) ray_setup_tris(s.r);
    for (; g < end; ++g) {
      const DevTri tri = load_tri(G.tris, g);
      if (STATS) cnt.tris++;
      float t, b0, b1, b2;
      if (tri_test(s.r, s.closest, tri, t, b0, b1, b2)) {
        // any_hit of an alpha-tested material: keep the hit iff u < opacity
        if (ALPHA && s.alpha < 1.0f && !(aux_next_f32(s.aux) < s.alpha)) continue;
        s.closest = t;
        s.res.tri = __float_as_int(tri.v0.w);
        s.res.inst = (int32_t)s.inst_id;
        s.res.b0 = b0; s.res.b1 = b1; s.res.b2 = b2;
        if (MODE == 1) {
          s.sp = 0;
          s.next = kNone;
          return;
        }
      }
    }
    trav_pop(G, s, st);
  } else if (count == 0) {
    enter_instance<ALPHA>(G, s, min(off, G.num_instances - 1u));
  } else {
    // TLAS leaf: its instances in order; the first is entered now
    if (s.sp + (int)count > kStackDepth) {
      atomicOr(err, kDevErrStackOverflow);
      s.sp = 0;
      s.next = kNone;
      return;
    }
    for (int j = (int)count - 1; j >= 1; --j) st.set(s.sp++, kLeafBit | __ldg(G.tlas_prims + min(off + j, G.num_instances - 1u)));
    enter_instance<ALPHA>(G, s, __ldg(G.tlas_prims + min(off, G.num_instances - 1u)));
  }
}

// One thread traces one ray to the end (used where a thread owns its ray).
template <int MODE, bool STATS, class Stack>
__device__ __forceinline__ void trace_ray(const DevGeometry& G, Stack& st, float ox, float oy, float oz, float dx,
                                          float dy, float dz, float t_max, TraceResult& res, TraceCounters& cnt,
                                          uint32_t* err, uint32_t* aux = nullptr) {
  TravState s;
  trav_init<true>(G, s, ox, oy, oz, dx, dy, dz, t_max, aux);
  if (STATS) { cnt.nodes = 0; cnt.tris = 0; }
  while (s.next != kNone) {
    if (!(s.next & kLeafBit)) node_step<STATS>(G, s, st, cnt, err);
    else leaf_step<MODE, STATS, true>(G, s, st, cnt, err);
  }
  res = s.res;
  res.t = hit_distance(s);
  if (aux) *aux = s.aux;
}

// trace_ray for lanes that trace together: the lanes in `act` (all of which
// call this) step through interior nodes together until each faces a leaf,
// then test their leaves together ("while-while"), so the warp runs one code
// path at a time.  Each ray's own visit order is unchanged.
template <int MODE, class Stack>
__device__ __forceinline__ void trace_ray_ww(const DevGeometry& G, Stack& st, unsigned act, float ox, float oy,
                                             float oz, float dx, float dy, float dz, float t_max, TraceResult& res,
                                             uint32_t* err, uint32_t* aux = nullptr) {
  TravState s;
  TraceCounters c;
  trav_init<true>(G, s, ox, oy, oz, dx, dy, dz, t_max, aux);
  for (;;) {
    for (;;) {
      const bool want = !(s.next & kLeafBit);
      if (!__any_sync(act, want)) break;
      if (want) node_step<false>(G, s, st, c, err);
    }
    if (s.next != kNone) leaf_step<MODE, false, true>(G, s, st, c, err);
    if (!__any_sync(act, s.next != kNone)) break;
  }
  res = s.res;
  res.t = hit_distance(s);
  if (aux) *aux = s.aux;
}

}  // namespace tpt
