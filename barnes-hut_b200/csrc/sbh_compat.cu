// Reference-compatible ("compat") entry points: the softened direct sums,
// the dense Morton octree8 build and its classic and stochastic Barnes-Hut
// traversals, all on the reference's byte layouts.
//
// This translation unit is compiled with --use_fast_math, the flag the
// reference's sbh_ffi target uses (CMakeLists.txt:39), so that the Morton
// quantisation (v - min) / span runs the same division instruction and
// produces the same codes, and the opening tests round the same way.
//
// Differences from the reference that are deliberate (and invisible at the
// byte level except where noted):
//  * no cudaMalloc/cudaFree, no D2H copy and no stream synchronisation: the
//    bounding span is computed on the device and temporaries live in a
//    caller-provided workspace (the reference syncs the stream and allocates
//    4*depth+12 buffers per build, src/sbh_ffi.cu:1111-1370);
//  * leaves are ordered by a stable radix sort of (Morton code, input index),
//    so the order inside one leaf cell is the input order (the reference's
//    atomic cursor makes it nondeterministic, src/sbh_ffi.cu:1732);
//  * the upward pass sums in FP64 (prefix sums over the sorted leaves), the
//    reference accumulates FP32 atomics;
//  * parameters travel by value, not through __constant__ globals, so calls
//    on concurrent streams do not race (src/sbh_ffi.cu:2536-2561);
//  * a traversal whose stack would exceed 128 entries records
//    SBH_DEV_STACK_OVERFLOW instead of writing past the array.
#include <cuda_runtime.h>
#include <curand_kernel.h>

#include <cstdint>
#include <mutex>
#include <string>

#include "sbh_common.cuh"
#include "sbh_primitives.cuh"

namespace sbh {

// ---------------------------------------------------------------------------
// Direct potential (src/sbh_ffi.cu:399-429), shared-memory tiled, one query
// per thread, Kahan-compensated across tiles.
// ---------------------------------------------------------------------------
constexpr int kDirectThreads = 256;

__global__ void __launch_bounds__(kDirectThreads)
    bruteforce_gravity_kernel(const float* __restrict__ pts, const float* __restrict__ masses, int64_t n,
                              int dim, const float* __restrict__ queries, int64_t nq,
                              float* __restrict__ out, Periodic per) {
  __shared__ float4 tile[kDirectThreads];
  int64_t qi = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  bool active = qi < nq;
  float q0 = 0.f, q1 = 0.f, q2 = 0.f;
  if (active) {
    q0 = queries[dim * qi];
    q1 = queries[dim * qi + 1];
    q2 = dim == 3 ? queries[dim * qi + 2] : 0.f;
  }
  float s = 0.f, c = 0.f;
  for (int64_t base = 0; base < n; base += kDirectThreads) {
    int64_t j = base + threadIdx.x;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j < n) v = make_float4(pts[dim * j], pts[dim * j + 1], dim == 3 ? pts[dim * j + 2] : 0.f, masses[j]);
    tile[threadIdx.x] = v;
    __syncthreads();
    int cnt = static_cast<int>(n - base < kDirectThreads ? n - base : kDirectThreads);
    float a = 0.f;
    for (int k = 0; k < cnt; k++) {
      float4 p = tile[k];
      // src/sbh_ffi.cu:414-426: diff = p - q, wrapped with nearbyint(diff / L)
      float d0 = p.x - q0, d1 = p.y - q1, d2 = p.z - q2;
      if (per.on && per.box > 0.0f) {
        d0 -= per.box * nearbyintf(d0 / per.box);
        d1 -= per.box * nearbyintf(d1 / per.box);
        if (dim == 3) d2 -= per.box * nearbyintf(d2 / per.box);
      }
      float dsq = d0 * d0 + d1 * d1;
      if (dim == 3) dsq += d2 * d2;
      a += -p.w / (sqrtf(dsq) + 1e-1f);
    }
    kahan_add(s, c, a);
    __syncthreads();
  }
  if (active) out[qi] = s;
}

// ---------------------------------------------------------------------------
// octree8 build (src/sbh_ffi.cu:1039-1420)
// ---------------------------------------------------------------------------
struct O8Params {
  float min[3];
  float span;
  float cx, cy, cz, half;
  int valid;
};

// span = max axis extent, root centre = min + span/2 (src/sbh_ffi.cu:1128-1133,1395-1398).
__global__ void o8_setup_kernel(const float* min_corner, const float* max_corner, O8Params* prm,
                                uint32_t* status) {
  float mn0 = min_corner[0], mn1 = min_corner[1], mn2 = min_corner[2];
  float span = fmaxf(fmaxf(max_corner[0] - mn0, max_corner[1] - mn1), max_corner[2] - mn2);
  O8Params p;
  p.min[0] = mn0;
  p.min[1] = mn1;
  p.min[2] = mn2;
  p.span = span;
  p.cx = mn0 + span * 0.5f;
  p.cy = mn1 + span * 0.5f;
  p.cz = mn2 + span * 0.5f;
  p.half = span * 0.5f;
  p.valid = span > 0.0f ? 1 : 0;
  if (!p.valid) raise_status(status, SBH_DEV_BAD_BOUNDS);
  *prm = p;
}

// quantize_axis (src/sbh_ffi.cu:173-179); fast-math division like the reference.
__device__ __forceinline__ uint32_t o8_quantize(float v, float min_v, float span, int bits) {
  float t = (v - min_v) / span;
  t = fminf(fmaxf(t, 0.0f), 0.999999f);
  uint32_t max_bin = (1u << bits) - 1u;
  return static_cast<uint32_t>(t * static_cast<float>(max_bin + 1));
}

__device__ __forceinline__ uint32_t o8_morton(uint32_t x, uint32_t y, uint32_t z, int bits) {
  uint32_t code = 0;
  for (int i = 0; i < bits; i++) {
    code |= ((x >> i) & 1u) << (3 * i);
    code |= ((y >> i) & 1u) << (3 * i + 1);
    code |= ((z >> i) & 1u) << (3 * i + 2);
  }
  return code;
}

__global__ void o8_codes_kernel(const float* __restrict__ pts, int64_t n, const O8Params* __restrict__ prm,
                                int depth, uint32_t* __restrict__ codes, uint32_t* __restrict__ counts) {
  if (!prm->valid) return;
  float mn0 = prm->min[0], mn1 = prm->min[1], mn2 = prm->min[2], span = prm->span;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    uint32_t qx = o8_quantize(pts[3 * i], mn0, span, depth);
    uint32_t qy = o8_quantize(pts[3 * i + 1], mn1, span, depth);
    uint32_t qz = o8_quantize(pts[3 * i + 2], mn2, span, depth);
    uint32_t c = o8_morton(qx, qy, qz, depth);
    codes[i] = c;
    atomicAdd(&counts[c], 1u);
  }
}

// Leaf records in sorted order (src/sbh_ffi.cu:1723-1743 writes the same record).
__global__ void o8_gather_kernel(const float* __restrict__ pts, const float* __restrict__ nrm,
                                 const float* __restrict__ masses, int64_t n,
                                 const uint32_t* __restrict__ perm, const O8Params* __restrict__ prm,
                                 Leaf3* __restrict__ leaf) {
  if (prm && !prm->valid) return;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    uint32_t s = perm[i];
    float4 a = make_float4(pts[3 * s], pts[3 * s + 1], pts[3 * s + 2], nrm ? nrm[3 * s] : 0.f);
    float4 b = make_float4(nrm ? nrm[3 * s + 1] : 0.f, nrm ? nrm[3 * s + 2] : 0.f, masses[s], 1.0f);
    float4* dst = reinterpret_cast<float4*>(leaf + i);
    dst[0] = a;
    dst[1] = b;
  }
}

// FP64 moment vector of a leaf record: (m, m x, m y, m z, m nx, m ny, m nz).
struct LeafMomentLoad {
  const Leaf3* leaf;
  __device__ DVec<7> operator()(int64_t i) const {
    const float4* p = reinterpret_cast<const float4*>(leaf + i);
    float4 a = p[0], b = p[1];
    double m = b.z;
    DVec<7> r;
    r.v[0] = m;
    r.v[1] = m * a.x;
    r.v[2] = m * a.y;
    r.v[3] = m * a.z;
    r.v[4] = m * a.w;
    r.v[5] = m * b.x;
    r.v[6] = m * b.y;
    return r;
  }
};

// One thread per dense node, all levels (src/sbh_ffi.cu:1788-1876).
__global__ void o8_nodes_kernel(OctreeNode8* __restrict__ nodes, Leaf3* __restrict__ contrib,
                                const uint32_t* __restrict__ off, const DVec<7>* __restrict__ P,
                                int depth, uint64_t total, const O8Params* __restrict__ prm) {
  if (!prm->valid) return;
  float cx0 = prm->cx, cy0 = prm->cy, cz0 = prm->cz, half0 = prm->half;
  for (uint64_t node_idx = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; node_idx < total;
       node_idx += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    int level = 0;
    uint64_t level_off = 0, level_n = 1;
    while (node_idx >= level_off + level_n) {
      level_off += level_n;
      level_n <<= 3;
      level++;
    }
    uint32_t idx = static_cast<uint32_t>(node_idx - level_off);
    int shift = 3 * (depth - level);
    uint64_t first_leaf = static_cast<uint64_t>(idx) << shift;
    uint64_t last_leaf = static_cast<uint64_t>(idx + 1) << shift;
    OctreeNode8 nd;
    nd.start = off[first_leaf];
    nd.end = off[last_leaf];
    nd.depth = static_cast<uint8_t>(level);
    nd.parent = level == 0 ? static_cast<uint32_t>(node_idx)
                           : static_cast<uint32_t>(level_off - (level_n >> 3) + (idx >> 3));
    nd.is_leaf = level == depth ? 1 : 0;
    nd.first_child = 0xFFFFFFFFu;
    nd.child_mask = 0;
    nd.pad0 = 0;
    int grid = 1 << level;
    int ix = 0, iy = 0, iz = 0;
    for (int b = 0; b < level; b++) {
      ix |= ((idx >> (3 * b + 0)) & 1) << b;
      iy |= ((idx >> (3 * b + 1)) & 1) << b;
      iz |= ((idx >> (3 * b + 2)) & 1) << b;
    }
    float step = half0 * 2.0f / static_cast<float>(grid);
    nd.cx = fmaf(static_cast<float>(ix) + 0.5f, step, cx0 - half0);
    nd.cy = fmaf(static_cast<float>(iy) + 0.5f, step, cy0 - half0);
    nd.cz = fmaf(static_cast<float>(iz) + 0.5f, step, cz0 - half0);
    nd.half_size = step * 0.5f;
    nd.diameter = step * sqrtf(3.0f);
    if (level < depth) {
      uint32_t child_base = static_cast<uint32_t>(level_off + level_n) + (idx << 3);
      int cshift = 3 * (depth - level - 1);
      uint8_t mask = 0;
      for (uint32_t c = 0; c < 8; c++) {
        nd.child[c] = child_base + c;
        uint64_t cl = static_cast<uint64_t>((idx << 3) + c) << cshift;
        uint64_t ch = static_cast<uint64_t>((idx << 3) + c + 1) << cshift;
        if (off[ch] > off[cl]) {
          mask |= static_cast<uint8_t>(1u << c);
          if (nd.first_child == 0xFFFFFFFFu) nd.first_child = child_base + c;
        }
      }
      nd.child_mask = mask;
      if (mask == 0) nd.is_leaf = 1;
    } else {
      for (int c = 0; c < 8; c++) nd.child[c] = 0xFFFFFFFFu;
    }
    DVec<7> hi = P[nd.end], lo = P[nd.start];
    double M = hi.v[0] - lo.v[0];
    float mass = static_cast<float>(M);
    nd.contrib.alpha = 1.0f;
    nd.contrib.mass = mass;
    if (mass > 0.0f) {
      for (int d = 0; d < 3; d++) {
        nd.contrib.pos[d] = static_cast<float>((hi.v[1 + d] - lo.v[1 + d]) / M);
        nd.contrib.nrm[d] = static_cast<float>((hi.v[4 + d] - lo.v[4 + d]) / M);
      }
    } else {
      for (int d = 0; d < 3; d++) {
        nd.contrib.pos[d] = 0.0f;
        nd.contrib.nrm[d] = 0.0f;
      }
    }
    // 8-byte stores: node_idx * 104 is 8-byte aligned.
    const uint2* src = reinterpret_cast<const uint2*>(&nd);
    uint2* dst = reinterpret_cast<uint2*>(nodes + node_idx);
#pragma unroll
    for (int k = 0; k < 13; k++) dst[k] = src[k];
    const float4* cs = reinterpret_cast<const float4*>(&nd.contrib);
    float4* cd = reinterpret_cast<float4*>(contrib + node_idx);
    cd[0] = cs[0];
    cd[1] = cs[1];
  }
}

// ---------------------------------------------------------------------------
// octree8 classic BH traversal (src/sbh_ffi.cu:1878-2144)
// ---------------------------------------------------------------------------
constexpr int kO8Stack = 128;

struct O8Node {
  float cx, cy, cz, half, diam;
  uint32_t start, end;
  uint8_t mask, is_leaf;
};

__device__ __forceinline__ float o8_mass(const OctreeNode8* nodes, int idx) {
  return __ldg(&nodes[idx].contrib.mass);
}

template <typename Node>
__device__ __forceinline__ bool o8_far(const Node& nd, float qx, float qy, float qz, float beta,
                                       const Periodic& per) {
  if (nd.is_leaf) return true;
  float dx = min_image_floor(qx - nd.cx, per);
  float dy = min_image_floor(qy - nd.cy, per);
  float dz = min_image_floor(qz - nd.cz, per);
  float dist = sqrtf(dx * dx + dy * dy + dz * dz);
  return dist / nd.diameter >= beta;
}

__device__ __forceinline__ float axis_gap(float q, float lo, float hi) {
  if (q < lo) return lo - q;
  if (q > hi) return q - hi;
  return 0.0f;
}

template <typename Node>
__device__ __forceinline__ bool o8_prune(const Node& nd, float qx, float qy, float qz,
                                         int prune_on, float r_cut_sq, const Periodic& per) {
  if (!prune_on) return false;
  if (per.on && per.box > 0.0f) {
    float inv_l = 1.0f / per.box;
    qx -= per.box * nearbyintf((qx - nd.cx) * inv_l);
    qy -= per.box * nearbyintf((qy - nd.cy) * inv_l);
    qz -= per.box * nearbyintf((qz - nd.cz) * inv_l);
  }
  float dx = axis_gap(qx, nd.cx - nd.half_size, nd.cx + nd.half_size);
  float dy = axis_gap(qy, nd.cy - nd.half_size, nd.cy + nd.half_size);
  float dz = axis_gap(qz, nd.cz - nd.half_size, nd.cz + nd.half_size);
  return dx * dx + dy * dy + dz * dz > r_cut_sq;
}

enum O8Kernel { O8_GRAV_GRAD = 0, O8_SOFT = 1, O8_SOFT_VJP = 2, O8_GRAV_GRAD_VJP = 3 };

// Softened pair terms in one fixed order of single-rounding operations
// (flush-to-zero, as the rest of this file under fast math), written once for
// a scalar pair and once for two pairs packed into FFMA2 / FADD2 / FMUL2
// (sm_100 f32x2). Both forms round every component the same way, so the
// traversal that sums a leaf two particles at a time and the one that sums
// it one at a time add bit-identical terms. The accumulation into the
// query's sum stays scalar and in the leaf's order.
struct F2 {
  unsigned long long v;
};

__device__ __forceinline__ F2 f2_pack(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_unpack(F2 x, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ float o8_add(float a, float b) {
  float d;
  asm("add.rn.ftz.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float o8_sub(float a, float b) {
  float d;
  asm("sub.rn.ftz.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float o8_mul(float a, float b) {
  float d;
  asm("mul.rn.ftz.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float o8_fma(float a, float b, float c) {
  float d;
  asm("fma.rn.ftz.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ F2 o8_add(F2 a, F2 b) {
  F2 d;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F2 o8_sub(F2 a, F2 b) {
  F2 d;
  asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F2 o8_mul(F2 a, F2 b) {
  F2 d;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F2 o8_fma(F2 a, F2 b, F2 c) {
  F2 d;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}
__device__ __forceinline__ float o8_splat_like(float, float s) { return s; }
__device__ __forceinline__ F2 o8_splat_like(F2, float s) { return f2_pack(s, s); }
__device__ __forceinline__ float o8_rsqrt(float a) { return rsqrtf(a); }
__device__ __forceinline__ F2 o8_rsqrt(F2 a) {
  float x, y;
  f2_unpack(a, x, y);
  return f2_pack(rsqrtf(x), rsqrtf(y));
}

// Shared first steps of the softened pair: r^2 = (rx rx + ry ry) + rz rz as
// two fused steps, h = (r^2 + eps^2) + 1e-12 and 1 / sqrt(h).
template <typename V>
__device__ __forceinline__ void o8_soft_head(V rx, V ry, V rz, V eps2, V& r2, V& ir) {
  r2 = o8_fma(rz, rz, o8_fma(ry, ry, o8_mul(rx, rx)));
  ir = o8_rsqrt(o8_add(o8_add(r2, eps2), o8_splat_like(eps2, 1e-12f)));
}

// Whether a pair lies in the att = 1 range (no cutoff, or r^2 + 1e-12 under
// the unity radius): then its terms skip the erfc attenuation.
__device__ __forceinline__ bool o8_unity(float r2, const Soft& s) {
  return !(s.cutoff > 0.0f && o8_add(r2, 1e-12f) >= s.unity_r2);
}

// erfc attenuation of one pair outside the att = 1 range (soft_coeff's slow
// path): att, and the VJP's radial term cc. Within that range cc stays below
// 1e-4 (r^2 + eps^2) / cutoff^2 of the 3 att ir^5 term it joins and is left out.
__device__ __forceinline__ void o8_soft_att(float r2, float ir3, const Soft& s, float& att, float& cc) {
  float dist = sqrtf(o8_add(r2, 1e-12f));
  float u = dist / (2.0f * s.cutoff);
  float e = 1.0f;
  att = 1.0f;
  if (u >= kAttUnityU) {
    e = expf(-(u * u));
    att = erfcf(u) + (2.0f / 1.772453850905516f) * u * e;
  }
  cc = ir3 * dist * e / (2.0f * 1.772453850905516f * s.cutoff * s.cutoff * s.cutoff);
}

// Softened force of one pair, nm = -m: acc += c r with c = nm / h^{3/2}
// (times att outside the att = 1 range).
__device__ __forceinline__ void o8_soft_force(float rx, float ry, float rz, float nm, float eps2, const Soft& s,
                                              float& ax, float& ay, float& az) {
  float r2, ir;
  o8_soft_head(rx, ry, rz, eps2, r2, ir);
  const float ir3 = o8_mul(o8_mul(ir, ir), ir);
  float c;
  if (o8_unity(r2, s)) {
    c = o8_mul(nm, ir3);
  } else {
    float att, cc;
    o8_soft_att(r2, ir3, s, att, cc);
    c = o8_mul(o8_mul(nm, att), ir3);
  }
  ax = o8_fma(c, rx, ax);
  ay = o8_fma(c, ry, ay);
  az = o8_fma(c, rz, az);
}

// Query-side VJP of one softened pair, nm = -m: acc += nm (lin g - rad r),
// with lin = att / h^{3/2} and rad = (r . g) (3 att / h^{5/2} + cc); the
// negated radial term is formed directly (rounding is symmetric in sign).
__device__ __forceinline__ void o8_soft_vjp(float rx, float ry, float rz, float nm, float gx, float gy, float gz,
                                            float eps2, const Soft& s, float& ax, float& ay, float& az) {
  float r2, ir;
  o8_soft_head(rx, ry, rz, eps2, r2, ir);
  const float ir3 = o8_mul(o8_mul(ir, ir), ir);
  const float ir5 = o8_mul(o8_mul(ir3, ir), ir);
  const float rg = o8_fma(rz, gz, o8_fma(ry, gy, o8_mul(rx, gx)));
  float lin, nrad;
  if (o8_unity(r2, s)) {
    lin = ir3;
    nrad = o8_mul(rg, o8_mul(-3.0f, ir5));
  } else {
    float att, cc;
    o8_soft_att(r2, ir3, s, att, cc);
    lin = o8_mul(att, ir3);
    nrad = o8_mul(rg, o8_sub(o8_mul(o8_mul(-3.0f, att), ir5), cc));
  }
  ax = o8_fma(nm, o8_fma(nrad, rx, o8_mul(lin, gx)), ax);
  ay = o8_fma(nm, o8_fma(nrad, ry, o8_mul(lin, gy)), ay);
  az = o8_fma(nm, o8_fma(nrad, rz, o8_mul(lin, gz)), az);
}

template <int KERNEL>
__device__ __forceinline__ void o8_pair(float qx, float qy, float qz, float px, float py, float pz, float m,
                                        float gx, float gy, float gz, const Soft& s, const Periodic& per,
                                        float& ax, float& ay, float& az) {
  if (KERNEL == O8_SOFT || KERNEL == O8_SOFT_VJP) {
    const float rx = min_image_floor(o8_sub(qx, px), per);
    const float ry = min_image_floor(o8_sub(qy, py), per);
    const float rz = min_image_floor(o8_sub(qz, pz), per);
    const float eps2 = o8_mul(s.eps, s.eps);
    if (KERNEL == O8_SOFT)
      o8_soft_force(rx, ry, rz, -m, eps2, s, ax, ay, az);
    else
      o8_soft_vjp(rx, ry, rz, -m, gx, gy, gz, eps2, s, ax, ay, az);
    return;
  }
  float rx = min_image_floor(qx - px, per);
  float ry = min_image_floor(qy - py, per);
  float rz = min_image_floor(qz - pz, per);
  if (KERNEL == O8_GRAV_GRAD) {
    float c = grav_grad_coeff(rx * rx + ry * ry + rz * rz, m);
    ax += c * rx;
    ay += c * ry;
    az += c * rz;
  } else {
    grav_grad_vjp_accum(rx, ry, rz, m, gx, gy, gz, ax, ay, az);
  }
}

// Two softened pairs without a periodic box, particles a then b: positions
// X, Y, Z and negated masses NM packed (a, b). The pair terms are packed, and
// each pair adds into the sums in order. With CHECK, a pair outside the
// att = 1 range sends both through the scalar form; without it the caller
// has shown that both pairs lie inside that range.
template <int KERNEL, bool CHECK>
__device__ __forceinline__ void o8_pair2(const F2& QX, const F2& QY, const F2& QZ, F2 X, F2 Y, F2 Z, F2 NM,
                                         const F2& GX, const F2& GY, const F2& GZ, float eps2, const Soft& s,
                                         float& ax, float& ay, float& az) {
  const F2 rx = o8_sub(QX, X), ry = o8_sub(QY, Y), rz = o8_sub(QZ, Z);
  F2 r2, ir;
  o8_soft_head(rx, ry, rz, f2_pack(eps2, eps2), r2, ir);
  float xa, xb, ya, yb, za, zb, ma, mb;
  f2_unpack(rx, xa, xb);
  f2_unpack(ry, ya, yb);
  f2_unpack(rz, za, zb);
  f2_unpack(NM, ma, mb);
  if (CHECK) {
    float r2a, r2b;
    f2_unpack(r2, r2a, r2b);
    if (!(o8_unity(r2a, s) && o8_unity(r2b, s))) {
      float gx, gy, gz, dummy;
      f2_unpack(GX, gx, dummy);
      f2_unpack(GY, gy, dummy);
      f2_unpack(GZ, gz, dummy);
      if (KERNEL == O8_SOFT) {
        o8_soft_force(xa, ya, za, ma, eps2, s, ax, ay, az);
        o8_soft_force(xb, yb, zb, mb, eps2, s, ax, ay, az);
      } else {
        o8_soft_vjp(xa, ya, za, ma, gx, gy, gz, eps2, s, ax, ay, az);
        o8_soft_vjp(xb, yb, zb, mb, gx, gy, gz, eps2, s, ax, ay, az);
      }
      return;
    }
  }
  const F2 ir3 = o8_mul(o8_mul(ir, ir), ir);
  if (KERNEL == O8_SOFT) {
    float ca, cb;
    f2_unpack(o8_mul(NM, ir3), ca, cb);
    ax = o8_fma(ca, xa, ax);
    ay = o8_fma(ca, ya, ay);
    az = o8_fma(ca, za, az);
    ax = o8_fma(cb, xb, ax);
    ay = o8_fma(cb, yb, ay);
    az = o8_fma(cb, zb, az);
  } else {
    const F2 ir5 = o8_mul(o8_mul(ir3, ir), ir);
    const F2 rg = o8_fma(rz, GZ, o8_fma(ry, GY, o8_mul(rx, GX)));
    const F2 nrad = o8_mul(rg, o8_mul(f2_pack(-3.0f, -3.0f), ir5));
    float ta, tb;
    f2_unpack(o8_fma(nrad, rx, o8_mul(ir3, GX)), ta, tb);
    ax = o8_fma(ma, ta, ax);
    ax = o8_fma(mb, tb, ax);
    f2_unpack(o8_fma(nrad, ry, o8_mul(ir3, GY)), ta, tb);
    ay = o8_fma(ma, ta, ay);
    ay = o8_fma(mb, tb, ay);
    f2_unpack(o8_fma(nrad, rz, o8_mul(ir3, GZ)), ta, tb);
    az = o8_fma(ma, ta, az);
    az = o8_fma(mb, tb, az);
  }
}

// One warp's staging buffer for a leaf's particles: 32 positions and
// negated masses, component by component, so that two or four consecutive
// particles load into packed register pairs with one shared-memory read.
constexpr int kO8LeafChunk = 32;

struct __align__(16) O8Chunk {
  float x[kO8LeafChunk], y[kO8LeafChunk], z[kO8LeafChunk], nm[kO8LeafChunk];
};

__device__ __forceinline__ F2 o8_ld2(const float* p) {
  F2 r;
  r.v = *reinterpret_cast<const unsigned long long*>(p);
  return r;
}

// The softened terms of cnt staged particles for one query, in order.
template <int KERNEL, bool CHECK>
__device__ __forceinline__ void o8_chunk_sum(const O8Chunk& ch, int cnt, float qx, float qy, float qz, float gx,
                                             float gy, float gz, const Soft& s, float& ax, float& ay, float& az) {
  const F2 QX = f2_pack(qx, qx), QY = f2_pack(qy, qy), QZ = f2_pack(qz, qz);
  const F2 GX = f2_pack(gx, gx), GY = f2_pack(gy, gy), GZ = f2_pack(gz, gz);
  const float eps2 = o8_mul(s.eps, s.eps);
  int j = 0;
  for (; j + 3 < cnt; j += 4) {
    const ulonglong2 X = *reinterpret_cast<const ulonglong2*>(&ch.x[j]);
    const ulonglong2 Y = *reinterpret_cast<const ulonglong2*>(&ch.y[j]);
    const ulonglong2 Z = *reinterpret_cast<const ulonglong2*>(&ch.z[j]);
    const ulonglong2 M = *reinterpret_cast<const ulonglong2*>(&ch.nm[j]);
    o8_pair2<KERNEL, CHECK>(QX, QY, QZ, F2{X.x}, F2{Y.x}, F2{Z.x}, F2{M.x}, GX, GY, GZ, eps2, s, ax, ay, az);
    o8_pair2<KERNEL, CHECK>(QX, QY, QZ, F2{X.y}, F2{Y.y}, F2{Z.y}, F2{M.y}, GX, GY, GZ, eps2, s, ax, ay, az);
  }
  if (j + 1 < cnt) {
    o8_pair2<KERNEL, CHECK>(QX, QY, QZ, o8_ld2(&ch.x[j]), o8_ld2(&ch.y[j]), o8_ld2(&ch.z[j]), o8_ld2(&ch.nm[j]),
                            GX, GY, GZ, eps2, s, ax, ay, az);
    j += 2;
  }
  if (j < cnt) {
    const float rx = o8_sub(qx, ch.x[j]), ry = o8_sub(qy, ch.y[j]), rz = o8_sub(qz, ch.z[j]);
    if (KERNEL == O8_SOFT)
      o8_soft_force(rx, ry, rz, ch.nm[j], eps2, s, ax, ay, az);
    else
      o8_soft_vjp(rx, ry, rz, ch.nm[j], gx, gy, gz, eps2, s, ax, ay, az);
  }
}

// Whether every pair of the query with a particle inside the cell (centre
// c, half size h, as o8_in_cell tests it) lies in the att = 1 range: the
// farthest corner's squared distance stays under the unity radius, with an
// absolute slack per axis (1e-6 of the magnitudes involved) and a relative
// margin (1e-4) far above the rounding of the differences and of r^2.
template <typename Node>
__device__ __forceinline__ bool o8_cell_unity(float qx, float qy, float qz, const Node& nd, const Soft& s) {
  if (!(s.cutoff > 0.0f)) return true;
  const float h = nd.half_size;
  const float mx = fabsf(qx - nd.cx) + h + 1e-6f * (fabsf(qx) + fabsf(nd.cx) + h);
  const float my = fabsf(qy - nd.cy) + h + 1e-6f * (fabsf(qy) + fabsf(nd.cy) + h);
  const float mz = fabsf(qz - nd.cz) + h + 1e-6f * (fabsf(qz) + fabsf(nd.cz) + h);
  const float R2 = mx * mx + my * my + mz * mz;
  return R2 * 1.0001f + 1e-12f < s.unity_r2;
}

template <typename Node>
__device__ __forceinline__ bool o8_in_cell(float px, float py, float pz, const Node& nd) {
  const float h = nd.half_size;
  return fabsf(px - nd.cx) <= h && fabsf(py - nd.cy) <= h && fabsf(pz - nd.cz) <= h;
}

// Direct softened sums (src/sbh_ffi.cu:431-546). A block of 16 warps stages
// tiles of 512 sources component by component, and each warp sums its 32
// queries (one per lane) over a 1 / SPLIT share of every tile; the SPLIT warps of
// the same queries then add their sums in order. With one query per lane the
// packed arithmetic takes two consecutive sources per FFMA2 / FADD2 / FMUL2. A
// chunk of 32 sources whose pairs with the warp's queries all lie in the
// att = 1 range (the farthest corners of the two bounding boxes, with margins,
// inside the unity radius: always so under the "no cutoff" convention) is
// summed without a per-pair test; otherwise it takes the scalar form pair by
// pair. Both round every component the same way (o8_soft_force, o8_soft_vjp).
// Each tile's sum joins the query's Kahan-compensated total.
constexpr int kDirectWarps = 16;
constexpr int kDirectTile = 32 * kDirectWarps;

struct __align__(16) DirectTile {
  float x[kDirectTile], y[kDirectTile], z[kDirectTile], nm[kDirectTile];
  float box[kDirectWarps][8];  // per chunk of 32: minima, maxima
};

template <bool PER>
__device__ __forceinline__ float direct_image(float d, float inv_l, const Periodic& per) {
  return PER ? min_image_rint(d, inv_l, per) : d;
}
template <bool PER>
__device__ __forceinline__ F2 direct_image(F2 d, float inv_l, const Periodic& per) {
  if (!PER) return d;
  float a, b;
  f2_unpack(d, a, b);
  return f2_pack(min_image_rint(a, inv_l, per), min_image_rint(b, inv_l, per));
}

template <int SPLIT, bool VJP, bool PER>
__global__ void __launch_bounds__(32 * kDirectWarps, 2)
    direct_soft_kernel(const float* __restrict__ pts, const float* __restrict__ masses, int64_t n,
                       const float* __restrict__ queries, const float* __restrict__ cot, int64_t nq,
                       float* __restrict__ out, Soft s, Periodic per) {
  __shared__ DirectTile T;
  __shared__ float part[SPLIT > 1 ? kDirectWarps : 1][3][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kChunks = kDirectWarps / SPLIT;  // chunks of 32 sources per warp and tile
  const int slice = warp % SPLIT;  // chunks slice, slice + SPLIT, ...: a short tile is shared too
  const int64_t qi = (static_cast<int64_t>(blockIdx.x) * (kDirectWarps / SPLIT) + warp / SPLIT) * 32 + lane;
  const bool active = qi < nq;
  const int64_t ql = active ? qi : nq - 1;
  const float qx = queries[3 * ql], qy = queries[3 * ql + 1], qz = queries[3 * ql + 2];
  float gx = 0.f, gy = 0.f, gz = 0.f;
  if (VJP) {
    gx = cot[3 * ql];
    gy = cot[3 * ql + 1];
    gz = cot[3 * ql + 2];
  }
  const float qbox[6] = {warp_min(qx), warp_min(qy), warp_min(qz), warp_max(qx), warp_max(qy), warp_max(qz)};
  const float inv_l = PER ? 1.0f / per.box : 0.0f;
  const F2 QX = f2_pack(qx, qx), QY = f2_pack(qy, qy), QZ = f2_pack(qz, qz);
  const F2 GX = f2_pack(gx, gx), GY = f2_pack(gy, gy), GZ = f2_pack(gz, gz);
  const float eps2 = o8_mul(s.eps, s.eps);
  const F2 EPS2 = f2_pack(eps2, eps2), M3 = f2_pack(-3.0f, -3.0f);
  float sx = 0.f, sy = 0.f, sz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
  float px = 0.f, py = 0.f, pz = 0.f, pm = 0.f;  // the thread's source of the next tile
  auto load = [&](int64_t j) {
    const bool in = j < n;
    px = in ? pts[3 * j] : 0.f;
    py = in ? pts[3 * j + 1] : 0.f;
    pz = in ? pts[3 * j + 2] : 0.f;
    pm = in ? masses[j] : 0.f;
  };
  load(threadIdx.x);
  for (int64_t base = 0; base < n; base += kDirectTile) {
    T.x[threadIdx.x] = px;
    T.y[threadIdx.x] = py;
    T.z[threadIdx.x] = pz;
    T.nm[threadIdx.x] = -pm;
    if (s.cutoff > 0.0f) {
      const bool in = base + threadIdx.x < n;
      const float b[6] = {warp_min(in ? px : INFINITY),  warp_min(in ? py : INFINITY),  warp_min(in ? pz : INFINITY),
                          warp_max(in ? px : -INFINITY), warp_max(in ? py : -INFINITY), warp_max(in ? pz : -INFINITY)};
      if (lane == 0)
        for (int d = 0; d < 6; d++) T.box[warp][d] = b[d];
    }
    __syncthreads();
    load(base + kDirectTile + threadIdx.x);  // in flight during this tile's sums
    const int left = static_cast<int>(n - base < kDirectTile ? n - base : kDirectTile);
    uint32_t unity = 0xffffffffu;  // bit c: chunk c * SPLIT + slice lies in the att = 1 range
    if (s.cutoff > 0.0f) {
      bool u = false;
      if (lane < kChunks) {
        const float* tb = T.box[lane * SPLIT + slice];
        float R2 = 0.0f;
        for (int d = 0; d < 3; d++) {
          const float span = fmaxf(fabsf(qbox[3 + d] - tb[d]), fabsf(tb[3 + d] - qbox[d]));
          const float mag = fmaxf(fmaxf(fabsf(qbox[d]), fabsf(qbox[3 + d])), fmaxf(fabsf(tb[d]), fabsf(tb[3 + d])));
          const float m = span + 1e-6f * mag;
          R2 += m * m;
        }
        u = R2 * 1.0001f + 1e-12f < s.unity_r2;
      }
      unity = __ballot_sync(0xffffffffu, u);
    }
    float ax = 0.f, ay = 0.f, az = 0.f;
    F2 AX = f2_pack(0.f, 0.f), AY = AX, AZ = AX;
    for (int c = 0; c < kChunks; c++) {
      const int j0 = (c * SPLIT + slice) * 32;
      const int cnt = left - j0 < 32 ? left - j0 : 32;
      if (cnt <= 0) break;
      if ((unity >> c) & 1u) {  // sources past the last one carry mass zero
#pragma unroll 2
        for (int j = j0; j < j0 + cnt; j += 4) {
          const ulonglong2 X = *reinterpret_cast<const ulonglong2*>(&T.x[j]);
          const ulonglong2 Y = *reinterpret_cast<const ulonglong2*>(&T.y[j]);
          const ulonglong2 Z = *reinterpret_cast<const ulonglong2*>(&T.z[j]);
          const ulonglong2 M = *reinterpret_cast<const ulonglong2*>(&T.nm[j]);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const F2 nm{h ? M.y : M.x};
            const F2 rx = direct_image<PER>(o8_sub(QX, F2{h ? X.y : X.x}), inv_l, per);
            const F2 ry = direct_image<PER>(o8_sub(QY, F2{h ? Y.y : Y.x}), inv_l, per);
            const F2 rz = direct_image<PER>(o8_sub(QZ, F2{h ? Z.y : Z.x}), inv_l, per);
            F2 r2, ir;
            o8_soft_head(rx, ry, rz, EPS2, r2, ir);
            const F2 ir3 = o8_mul(o8_mul(ir, ir), ir);
            if (!VJP) {
              const F2 k = o8_mul(nm, ir3);
              AX = o8_fma(k, rx, AX);
              AY = o8_fma(k, ry, AY);
              AZ = o8_fma(k, rz, AZ);
            } else {
              const F2 ir5 = o8_mul(o8_mul(ir3, ir), ir);
              const F2 rg = o8_fma(rz, GZ, o8_fma(ry, GY, o8_mul(rx, GX)));
              const F2 nrad = o8_mul(rg, o8_mul(M3, ir5));
              AX = o8_fma(nm, o8_fma(nrad, rx, o8_mul(ir3, GX)), AX);
              AY = o8_fma(nm, o8_fma(nrad, ry, o8_mul(ir3, GY)), AY);
              AZ = o8_fma(nm, o8_fma(nrad, rz, o8_mul(ir3, GZ)), AZ);
            }
          }
        }
      } else {
#pragma unroll 4
        for (int j = j0; j < j0 + cnt; j++) {
          const float rx = direct_image<PER>(o8_sub(qx, T.x[j]), inv_l, per);
          const float ry = direct_image<PER>(o8_sub(qy, T.y[j]), inv_l, per);
          const float rz = direct_image<PER>(o8_sub(qz, T.z[j]), inv_l, per);
          if (VJP)
            o8_soft_vjp(rx, ry, rz, T.nm[j], gx, gy, gz, eps2, s, ax, ay, az);
          else
            o8_soft_force(rx, ry, rz, T.nm[j], eps2, s, ax, ay, az);
        }
      }
    }
    float a, b;
    f2_unpack(AX, a, b);
    kahan_add(sx, cx, ax + (a + b));
    f2_unpack(AY, a, b);
    kahan_add(sy, cy, ay + (a + b));
    f2_unpack(AZ, a, b);
    kahan_add(sz, cz, az + (a + b));
    __syncthreads();
  }
  if (SPLIT > 1) {
    part[warp][0][lane] = sx;
    part[warp][1][lane] = sy;
    part[warp][2][lane] = sz;
    __syncthreads();
    if (slice == 0) {
#pragma unroll
      for (int w = 1; w < SPLIT; w++) {
        sx += part[warp + w][0][lane];
        sy += part[warp + w][1][lane];
        sz += part[warp + w][2][lane];
      }
    }
  }
  if (active && slice == 0) {
    out[3 * qi] = sx;
    out[3 * qi + 1] = sy;
    out[3 * qi + 2] = sz;
  }
}

// One query's terms from leaf particles [start, end), in order; softened
// pairs without a periodic box go two at a time through o8_pair2. AHEAD: the
// unsoftened VJP, whose pair is a long chain, loads four particles before their
// terms (stochastic estimate, 20,000 queries of 2^20 Plummer particles: 18.9 ms one
// by one, 13.1 by two, 9.8 by four, at 99 registers).
template <int KERNEL, bool AHEAD = false>
__device__ __forceinline__ void o8_leaf_sum(const Leaf3* __restrict__ leaf, uint32_t start, uint32_t end,
                                            float qx, float qy, float qz, float gx, float gy, float gz,
                                            const Soft& s, const Periodic& per, float& ax, float& ay,
                                            float& az) {
  uint32_t i = start;
  if ((KERNEL == O8_SOFT || KERNEL == O8_SOFT_VJP) && !per.on) {
    const F2 QX = f2_pack(qx, qx), QY = f2_pack(qy, qy), QZ = f2_pack(qz, qz);
    const F2 GX = f2_pack(gx, gx), GY = f2_pack(gy, gy), GZ = f2_pack(gz, gz);
    const float eps2 = o8_mul(s.eps, s.eps);
    for (; i + 1 < end; i += 2) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(leaf + i));
      const float4 b = __ldg(reinterpret_cast<const float4*>(leaf + i + 1));
      const float ma = __ldg(&leaf[i].mass), mb = __ldg(&leaf[i + 1].mass);
      o8_pair2<KERNEL, true>(QX, QY, QZ, f2_pack(a.x, b.x), f2_pack(a.y, b.y), f2_pack(a.z, b.z), f2_pack(-ma, -mb),
                             GX, GY, GZ, eps2, s, ax, ay, az);
    }
  }
  if (AHEAD && KERNEL == O8_GRAV_GRAD_VJP) {
    for (; i < end && end - i >= 4; i += 4) {
      float4 a[4];
      float m[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        a[j] = __ldg(reinterpret_cast<const float4*>(leaf + i + j));
        m[j] = __ldg(&leaf[i + j].mass);
      }
#pragma unroll
      for (int j = 0; j < 4; j++)
        o8_pair<KERNEL>(qx, qy, qz, a[j].x, a[j].y, a[j].z, m[j], gx, gy, gz, s, per, ax, ay, az);
    }
  }
  for (; i < end; i++) {
    const float4* p = reinterpret_cast<const float4*>(leaf + i);
    float4 a = __ldg(p);
    float m = __ldg(&leaf[i].mass);
    o8_pair<KERNEL>(qx, qy, qz, a.x, a.y, a.z, m, gx, gy, gz, s, per, ax, ay, az);
  }
}

// Buffers come from the caller: child indices and leaf ranges are checked
// against the buffer sizes and a violation sets SBH_DEV_BAD_BOUNDS instead of
// reading out of bounds.
struct O8Bounds {
  uint32_t num_nodes;
  uint32_t num_leaves;
};

__device__ __forceinline__ bool o8_node_ok(uint32_t idx, const O8Bounds& bd, uint32_t* status) {
  if (idx < bd.num_nodes) return true;
  raise_status(status, SBH_DEV_BAD_BOUNDS);
  return false;
}

__device__ __forceinline__ uint32_t o8_leaf_end(uint32_t start, uint32_t end, const O8Bounds& bd,
                                                uint32_t* status) {
  if (end <= bd.num_leaves && start <= end) return end;
  raise_status(status, SBH_DEV_BAD_BOUNDS);
  return start <= bd.num_leaves ? (end < bd.num_leaves ? end : bd.num_leaves) : start;
}

// For trees of up to kO8UnitLeaves particles a query's sum is taken in units: the
// root, each of its children and each of their children with its whole subtree, in
// the order of the DFS. Every unit is summed from zero and the units are added in
// order, so warps may share a query's units without changing a bit of its row.
// (Larger trees keep the single running sum of the reference's traversal: its
// rounding grows with the tree, and the units' smaller one, though nearer the 64-bit
// sum, would leave the reference's rows by 2e-5 at 2^18 particles against 2e-6
// here.) Which entry starts a unit follows from the stack's heights: the level-1
// entries lie below h1, the level-2 entries of the current level-1 node between h1
// and h2.
struct O8Units {
  int h1 = 0, h2 = 0;
  bool started = false;
  // The level (0 root, 1, 2, or 3 for any deeper) of the entry popped from index i.
  __device__ __forceinline__ int pop(int i) {
    if (!started) {
      started = true;
      return 0;
    }
    if (i < h1) {
      h1 = h2 = i;
      return 1;
    }
    if (i < h2) {
      h2 = i;
      return 2;
    }
    return 3;
  }
  // After the children of a node of that level were pushed up to `top`.
  __device__ __forceinline__ void pushed(int level, int top) {
    if (level == 0) h1 = h2 = top;
    if (level == 1) h2 = top;
  }
};
constexpr int kO8MaxUnits = 1 + 8 + 64;
constexpr uint32_t kO8UnitLeaves = 16384;

template <int KERNEL>
__global__ void __launch_bounds__(256)
    o8_bh_kernel(const Leaf3* __restrict__ leaf, const OctreeNode8* __restrict__ nodes,
                 const float* __restrict__ queries, const float* __restrict__ cot, int64_t nq, float beta,
                 Soft s, int prune_on, float r_cut_sq, Periodic per, float* __restrict__ out,
                 uint32_t* status, O8Bounds bd, const uint32_t* __restrict__ order) {
  int64_t ti = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (ti >= nq) return;
  const int64_t qi = order ? static_cast<int64_t>(order[ti]) : ti;
  float qx = queries[3 * qi], qy = queries[3 * qi + 1], qz = queries[3 * qi + 2];
  float gx = 0.f, gy = 0.f, gz = 0.f;
  if (KERNEL == O8_SOFT_VJP || KERNEL == O8_GRAV_GRAD_VJP) {
    gx = cot[3 * qi];
    gy = cot[3 * qi + 1];
    gz = cot[3 * qi + 2];
  }
  float ax = 0.f, ay = 0.f, az = 0.f, tx = 0.f, ty = 0.f, tz = 0.f;
  int stack[kO8Stack];
  int top = 0;
  stack[top++] = 0;
  bool overflow = false;
  O8Units units;
  // A well-formed tree reaches each node from the root exactly once, so one
  // query pops at most num_nodes nodes. More pops mean that the caller's
  // child indices form a cycle: stop, flag it and keep the partial sum.
  uint32_t visits = 0;
  while (top > 0) {
    if (++visits > bd.num_nodes) {
      raise_status(status, SBH_DEV_ITER_LIMIT);
      break;
    }
    int idx = stack[--top];
    const int level = units.pop(top);
    if (level < 3 && bd.num_leaves <= kO8UnitLeaves) {  // a new unit: the last one's sum joins the query's total
      tx += ax, ty += ay, tz += az;
      ax = ay = az = 0.f;
    }
    if (o8_mass(nodes, idx) == 0.0f) continue;
    const OctreeNode8& nd = nodes[idx];
    if (KERNEL != O8_GRAV_GRAD && KERNEL != O8_GRAV_GRAD_VJP &&
        o8_prune(nd, qx, qy, qz, prune_on, r_cut_sq, per))
      continue;
    if (o8_far(nd, qx, qy, qz, beta, per)) {
      if (nd.is_leaf) {
        o8_leaf_sum<KERNEL>(leaf, nd.start, o8_leaf_end(nd.start, nd.end, bd, status), qx, qy, qz, gx, gy, gz, s,
                            per, ax, ay, az);
      } else {
        o8_pair<KERNEL>(qx, qy, qz, nd.contrib.pos[0], nd.contrib.pos[1], nd.contrib.pos[2], nd.contrib.mass,
                        gx, gy, gz, s, per, ax, ay, az);
      }
    } else {
      uint8_t mask = nd.child_mask;
      for (int c = 0; c < 8; c++) {
        if (mask & (1u << c)) {
          if (!o8_node_ok(nd.child[c], bd, status)) continue;
          if (top < kO8Stack) {
            stack[top++] = static_cast<int>(nd.child[c]);
          } else {
            overflow = true;
          }
        }
      }
      units.pushed(level, top);
    }
  }
  if (overflow) raise_status(status, SBH_DEV_STACK_OVERFLOW);
  out[3 * qi] = tx + ax;
  out[3 * qi + 1] = ty + ay;
  out[3 * qi + 2] = tz + az;
}

// Warp-cooperative form of o8_bh_kernel, for queries taken in Morton order
// (32 neighbouring queries per warp). The warp walks one DFS stack in shared
// memory whose entries carry the lanes that still descend at that node, and
// each lane takes its own prune and opening decisions, exactly as its thread
// does in o8_bh_kernel: a node is pushed (children in the same order) when
// some lane opens it, with that set of lanes. A lane's nodes thus come off
// the stack in the order of its own per-thread DFS, so it adds the same terms
// in the same order and every output row equals o8_bh_kernel's bit for bit;
// node records are read once per warp instead of once per thread. The next
// entry's record loads while the current node's terms are summed. At a leaf
// the warp copies the particles in chunks of 32 (one coalesced load per lane)
// into a per-warp buffer in shared memory, and the summing lanes read them
// from there in the leaf's order.
//
// WQ = 8: the block's eight warps share one set of 32 queries. Every warp walks
// the tree's top two levels and takes units (O8Units) off a counter; the units'
// sums meet in shared memory and are added in order. WQ = 1: each warp of the
// block has its own `per_set` queries (the lanes past them idle).
// The block's dynamic shared memory holds each warp's leaf buffer (32 x 16 B),
// then each warp's stack of STACK entries (64 for a dense octree8 of depth <= 9:
// a DFS of depth d holds at most 7 d + 1 entries; otherwise the reference's
// 128), then for WQ = 8 the units' sums.
struct O8StackEntry {
  int node;
  uint32_t lanes;
};

__host__ __device__ constexpr size_t o8_warp_smem(int warps, int stack) {
  return static_cast<size_t>(warps) * (sizeof(O8Chunk) + stack * sizeof(O8StackEntry));
}

// What a visit reads of a node record.
struct O8Visit {
  float mass, cx, cy, cz, half_size, diameter, px, py, pz;
  uint32_t start, end;
  uint8_t child_mask, is_leaf;
};

__device__ __forceinline__ O8Visit o8_visit(const OctreeNode8* __restrict__ nodes, int idx) {
  const char* p = reinterpret_cast<const char*>(nodes + idx);
  const uint2 range = __ldg(reinterpret_cast<const uint2*>(p));
  const uint2 fl = __ldg(reinterpret_cast<const uint2*>(p + 48));
  const float2 yz = __ldg(reinterpret_cast<const float2*>(p + 56)), hd = __ldg(reinterpret_cast<const float2*>(p + 64));
  const float2 xy = __ldg(reinterpret_cast<const float2*>(p + 72));
  O8Visit v;
  v.start = range.x;
  v.end = range.y;
  v.child_mask = static_cast<uint8_t>(fl.x);
  v.is_leaf = static_cast<uint8_t>(fl.x >> 16);
  v.cx = __uint_as_float(fl.y);
  v.cy = yz.x;
  v.cz = yz.y;
  v.half_size = hd.x;
  v.diameter = hd.y;
  v.px = xy.x;
  v.py = xy.y;
  v.pz = __ldg(reinterpret_cast<const float*>(p + 80));
  v.mass = __ldg(reinterpret_cast<const float*>(p + 96));
  return v;
}
static_assert(offsetof(OctreeNode8, child_mask) == 48 && offsetof(OctreeNode8, is_leaf) == 50 &&
                  offsetof(OctreeNode8, cx) == 52 && offsetof(OctreeNode8, half_size) == 64,
              "OctreeNode8 offsets read by o8_visit");

struct O8UnitSums {
  float v[kO8MaxUnits][3][32];
  int next;
};

// Blocks of 128 threads per SM with own query sets: 6 (80 registers) for the
// forces; the VJPs 7 (72), in a periodic box 8 (64), so that trees of 10^6
// particles, where more warps hide more of the visits' latency, are not slower
// than without the prefetch: Plummer 218 ms against 225 at 6 blocks (222 without
// prefetch), periodic 8.06 against 8.34 (8.00). It costs a VJP 4% at 60,000 to
// 100,000 particles (6.8 and 8.6 ms; 8.4 and 10.6 without prefetch). Forces at 7
// blocks: 153 ms against 149 at 10^6.
template <int KERNEL, bool STAGED>
constexpr int kO8OwnBlocks = KERNEL == O8_SOFT_VJP || KERNEL == O8_GRAV_GRAD_VJP ? (STAGED ? 7 : 8) : 6;

template <int KERNEL, int STACK, bool STAGED, int WQ>
__global__ void __launch_bounds__(WQ > 1 ? 256 : 128, WQ > 1 ? 3 : kO8OwnBlocks<KERNEL, STAGED>)
    o8_bh_warp_kernel(const Leaf3* __restrict__ leaf, const OctreeNode8* __restrict__ nodes,
                      const float* __restrict__ queries, const float* __restrict__ cot, int64_t nq, float beta,
                      Soft s, int prune_on, float r_cut_sq, Periodic per, float* __restrict__ out, uint32_t* status,
                      O8Bounds bd, const uint32_t* __restrict__ order, int per_set) {
  extern __shared__ float4 o8_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  O8Chunk& chunk = reinterpret_cast<O8Chunk*>(o8_smem)[warp];
  O8StackEntry* stack = reinterpret_cast<O8StackEntry*>(reinterpret_cast<O8Chunk*>(o8_smem) + (blockDim.x >> 5)) +
                        warp * STACK;
  O8UnitSums& sums = *reinterpret_cast<O8UnitSums*>(reinterpret_cast<char*>(o8_smem) +
                                                    o8_warp_smem(static_cast<int>(blockDim.x >> 5), STACK));
  const int64_t set = WQ > 1 ? static_cast<int64_t>(blockIdx.x)
                             : static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + warp;
  const int64_t ti = WQ > 1 ? set * 32 + lane : set * per_set + lane;
  const bool valid = (WQ > 1 || lane < per_set) && ti < nq;
  const uint32_t live = __ballot_sync(0xffffffffu, valid);
  if (live == 0) return;  // uniform over the warps of a set
  int mine = 0;           // WQ > 1: the unit this warp takes next
  if (WQ > 1) {
    if (threadIdx.x == 0) sums.next = WQ;
    for (int i = threadIdx.x; i < kO8MaxUnits * 96; i += 32 * WQ) (&sums.v[0][0][0])[i] = 0.0f;
    mine = warp;
    __syncthreads();
  }
  const int64_t qi = valid ? static_cast<int64_t>(order[ti]) : 0;
  float qx = 0.f, qy = 0.f, qz = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
  if (valid) {
    qx = queries[3 * qi];
    qy = queries[3 * qi + 1];
    qz = queries[3 * qi + 2];
    if (KERNEL == O8_SOFT_VJP || KERNEL == O8_GRAV_GRAD_VJP) {
      gx = cot[3 * qi];
      gy = cot[3 * qi + 1];
      gz = cot[3 * qi + 2];
    }
  }
  float ax = 0.f, ay = 0.f, az = 0.f, tx = 0.f, ty = 0.f, tz = 0.f;
  const bool in_units = bd.num_leaves <= kO8UnitLeaves;
  int unit = -1;  // units begun so far, less one
  auto end_unit = [&] {  // the current unit's sum joins the total
    if (WQ == 1) {
      if (!in_units) return;
      tx += ax, ty += ay, tz += az;
    } else if (unit == mine) {
      sums.v[unit][0][lane] = ax;
      sums.v[unit][1][lane] = ay;
      sums.v[unit][2][lane] = az;
      if (lane == 0) mine = atomicAdd(&sums.next, 1);
      mine = __shfl_sync(0xffffffffu, mine, 0);
    }
    ax = ay = az = 0.f;
  };
  if (lane == 0) stack[0] = O8StackEntry{0, live};
  __syncwarp();
  int top = 1;  // warp-uniform
  bool overflow = false;
  uint32_t visits = 0;  // bounded as in o8_bh_kernel
  O8Units units;
  O8StackEntry en{0, live};
  O8Visit nx = o8_visit(nodes, 0);
  while (top > 0) {
    if (++visits > bd.num_nodes) {
      if (lane == 0) raise_status(status, SBH_DEV_ITER_LIMIT);
      break;
    }
    const O8Visit nd = nx;
    const int idx = en.node;
    const uint32_t lanes = en.lanes;
    top--;
    const int level = units.pop(top);
    if (level < 3) {
      end_unit();
      unit++;
    }
    const bool own = WQ == 1 || unit == mine;
    bool act = ((lanes >> lane) & 1u) && nd.mass != 0.0f && (own || level < 2);
    if (KERNEL != O8_GRAV_GRAD && KERNEL != O8_GRAV_GRAD_VJP)
      act = act && !o8_prune(nd, qx, qy, qz, prune_on, r_cut_sq, per);
    const bool far = act && o8_far(nd, qx, qy, qz, beta, per);
    const uint32_t open = __ballot_sync(0xffffffffu, act && !far);
    if (open) {
      // slot c's child index in lane c; the pushes keep the slots' order
      const uint32_t ch = lane < 8 ? __ldg(&nodes[idx].child[lane]) : 0u;
      bool push = lane < 8 && ((nd.child_mask >> lane) & 1u);
      if (push && !o8_node_ok(ch, bd, status)) push = false;
      const uint32_t pm = __ballot_sync(0xffffffffu, push);
      const int at = top + __popc(pm & ((1u << lane) - 1u));
      if (push && at < STACK) stack[at] = O8StackEntry{static_cast<int>(ch), open};
      top += __popc(pm);
      if (top > STACK) {
        top = STACK;
        overflow = true;
      }
      units.pushed(level, top);
    }
    __syncwarp();
    if (top > 0) {
      en = stack[top - 1];
      nx = o8_visit(nodes, en.node);
    }
    if (!own || !__any_sync(0xffffffffu, far)) {
      __syncwarp();  // every lane has read the entry before it is overwritten
      continue;
    }
    if (nd.is_leaf && !STAGED) {  // nd is warp-uniform: every lane reads the same node
      if (far)
        o8_leaf_sum<KERNEL>(leaf, nd.start, o8_leaf_end(nd.start, nd.end, bd, status), qx, qy, qz, gx, gy, gz, s,
                            per, ax, ay, az);
    } else if (nd.is_leaf) {
      const uint32_t start = nd.start, end = o8_leaf_end(start, nd.end, bd, status);
      constexpr bool kSoft = KERNEL == O8_SOFT || KERNEL == O8_SOFT_VJP;
      const bool q_unity = !far || o8_cell_unity(qx, qy, qz, nd, s);
      // chunks of 32 particles, one per lane, the next one loaded while
      // the current one is summed
      float4 nxt = make_float4(0.f, 0.f, 0.f, 0.f);
      float nxt_m = 0.f;
      if (start + lane < end) {
        nxt = __ldg(reinterpret_cast<const float4*>(leaf + start + lane));
        nxt_m = __ldg(&leaf[start + lane].mass);
      }
      for (uint32_t c = start; c < end; c += kO8LeafChunk) {
        const uint32_t i = c + lane;
        bool in_cell = true;
        if (i < end) {
          chunk.x[lane] = nxt.x;
          chunk.y[lane] = nxt.y;
          chunk.z[lane] = nxt.z;
          chunk.nm[lane] = -nxt_m;
          in_cell = o8_in_cell(nxt.x, nxt.y, nxt.z, nd);
        }
        if (i + kO8LeafChunk < end) {
          nxt = __ldg(reinterpret_cast<const float4*>(leaf + i + kO8LeafChunk));
          nxt_m = __ldg(&leaf[i + kO8LeafChunk].mass);
        }
        const bool unity = __all_sync(0xffffffffu, in_cell && q_unity);
        __syncwarp();
        const int cnt = end - c < kO8LeafChunk ? static_cast<int>(end - c) : kO8LeafChunk;
        if (far) {
          if (kSoft && !per.on) {
            if (unity)
              o8_chunk_sum<KERNEL, false>(chunk, cnt, qx, qy, qz, gx, gy, gz, s, ax, ay, az);
            else
              o8_chunk_sum<KERNEL, true>(chunk, cnt, qx, qy, qz, gx, gy, gz, s, ax, ay, az);
          } else {
            for (int j = 0; j < cnt; j++)
              o8_pair<KERNEL>(qx, qy, qz, chunk.x[j], chunk.y[j], chunk.z[j], -chunk.nm[j], gx, gy, gz, s, per, ax,
                              ay, az);
          }
        }
        __syncwarp();  // the chunk is read before the next one overwrites it
      }
    } else if (far) {
      o8_pair<KERNEL>(qx, qy, qz, nd.px, nd.py, nd.pz, nd.mass, gx, gy, gz, s, per, ax, ay, az);
    }
    __syncwarp();
  }
  if (overflow && lane == 0) raise_status(status, SBH_DEV_STACK_OVERFLOW);
  if (WQ == 1) {
    if (valid) {
      out[3 * qi] = tx + ax;
      out[3 * qi + 1] = ty + ay;
      out[3 * qi + 2] = tz + az;
    }
  } else {
    end_unit();
    __syncthreads();
    for (int c = warp; c < 3; c += WQ) {
      float t = 0.f;
      for (int u = 0; u < kO8MaxUnits; u++) t += sums.v[u][c][lane];
      if (valid) out[3 * qi + c] = t;
    }
  }
}

// ---------------------------------------------------------------------------
// octree8 stochastic BH, the multi-level prefix control variate
// (src/sbh_ffi.cu:2146-2442). Same curand calls as the reference, so a
// fixed seed gives the reference's sample paths.
// ---------------------------------------------------------------------------
constexpr int kControlDepth = 3;
constexpr int kMaxSubdomains = 512;
constexpr int kO8MaxDescent = 64;

template <int KERNEL>
__device__ __forceinline__ void o8_contrib_pair(const OctreeNode8& nd, float qx, float qy, float qz, float gx,
                                                float gy, float gz, const Soft& s, const Periodic& per,
                                                float& ax, float& ay, float& az) {
  o8_pair<KERNEL>(qx, qy, qz, nd.contrib.pos[0], nd.contrib.pos[1], nd.contrib.pos[2], nd.contrib.mass, gx,
                  gy, gz, s, per, ax, ay, az);
}

__device__ __forceinline__ uint32_t o8_child_slot(const OctreeNode8& nd, float px, float py, float pz) {
  uint32_t ix = px >= nd.cx ? 1u : 0u;
  uint32_t iy = py >= nd.cy ? 1u : 0u;
  uint32_t iz = pz >= nd.cz ? 1u : 0u;
  return ix | (iy << 1) | (iz << 2);
}

// The subdomains of the estimator (the reference's DFS from the root down to
// leaves and nodes of depth 3) do not depend on the query, so a block lists them
// once in shared memory, level by level: every round replaces each node that
// is neither by its children, slot 7 first, which keeps the order of a DFS that
// pops the last child pushed. Per thread this search was a chain of some 600
// dependent visits and 2.5 KB of local memory. A well-formed tree ends after
// three rounds with at most 512 entries; more nodes seen than the buffer has
// (a cycle in the caller's child indices) or a longer list sets the status bits
// of the per-thread search.
constexpr int kStochThreads = 128;

struct O8Subdomains {
  uint32_t list[2][kMaxSubdomains];
  int warp_sum[kStochThreads / 32];
  int cur;
};

__device__ __forceinline__ int o8_subdomains(const OctreeNode8* __restrict__ nodes, const O8Bounds& bd,
                                             uint32_t* status, O8Subdomains& S) {
  constexpr int kPer = kMaxSubdomains / kStochThreads;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) S.list[0][0] = 0;
  __syncthreads();
  int n = 1, cur = 0;
  for (uint64_t seen = 1;;) {
    int cnt[kPer], sum = 0;
    uint32_t id[kPer];
    uint8_t mask[kPer];  // children that replace the entry; 0 with cnt 1: the entry itself
    bool open = false;  // a later round is needed
#pragma unroll
    for (int e = 0; e < kPer; e++) {
      const int i = static_cast<int>(threadIdx.x) * kPer + e;
      cnt[e] = 0;
      mask[e] = 0;
      if (i < n) {
        id[e] = S.list[cur][i];
        const OctreeNode8& nd = nodes[id[e]];
        if (nd.contrib.mass != 0.0f) {
          if (nd.is_leaf || nd.depth >= kControlDepth) {
            cnt[e] = 1;
          } else {
            for (int c = 0; c < 8; c++)
              if (((nd.child_mask >> c) & 1u) && o8_node_ok(nd.child[c], bd, status))
                mask[e] |= static_cast<uint8_t>(1u << c);
            cnt[e] = __popc(mask[e]);
            open = true;
          }
        }
      }
      sum += cnt[e] + (mask[e] ? cnt[e] << 16 : 0);  // entries; above, the new ones
    }
    int inc = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) S.warp_sum[warp] = inc;
    open = __syncthreads_or(open);
    int at = inc - sum, total = 0;
    for (int w = 0; w < kStochThreads / 32; w++) {
      if (w < warp) at += S.warp_sum[w];
      total += S.warp_sum[w];
    }
    seen += static_cast<uint64_t>(total >> 16);
    at &= 0xFFFF;
    total &= 0xFFFF;
#pragma unroll
    for (int e = 0; e < kPer; e++) {
      if (cnt[e] == 0) continue;
      if (mask[e] == 0) {
        if (at < kMaxSubdomains) S.list[cur ^ 1][at] = id[e];
        at++;
      } else {
        for (int c = 7; c >= 0; c--) {
          if (!((mask[e] >> c) & 1u)) continue;
          if (at < kMaxSubdomains) S.list[cur ^ 1][at] = nodes[id[e]].child[c];
          at++;
        }
      }
    }
    if (total > kMaxSubdomains) {
      if (threadIdx.x == 0) raise_status(status, SBH_DEV_STACK_OVERFLOW);
      total = kMaxSubdomains;
    }
    cur ^= 1;
    n = total;
    __syncthreads();
    if (!open || n == 0) break;
    if (seen > bd.num_nodes) {
      if (threadIdx.x == 0) raise_status(status, SBH_DEV_ITER_LIMIT);
      break;
    }
  }
  if (threadIdx.x == 0) S.cur = cur;
  __syncthreads();
  return n;
}

// (Bounded by 256 threads the softened force takes 80 registers, by its 128 72: with
// attenuation 13.5 ms against 12.7, 20,000 queries of 2^20 Plummer particles.)
template <int KERNEL, bool SOFTENED>
__global__ void __launch_bounds__(2 * kStochThreads)
    o8_stochastic_kernel(const Leaf3* __restrict__ leaf, const OctreeNode8* __restrict__ nodes,
                         const float* __restrict__ queries, const float* __restrict__ cot, int64_t nq,
                         int samples, int seed, float beta, Soft s, int prune_on, float r_cut_sq,
                         Periodic per, float* __restrict__ out, uint32_t* status, O8Bounds bd,
                         const uint32_t* __restrict__ order) {
  __shared__ O8Subdomains S;
  const int nsub = o8_subdomains(nodes, bd, status, S);
  const uint32_t* subs = S.list[S.cur];
  int64_t ti = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (ti >= nq) return;
  const int64_t qi = order ? static_cast<int64_t>(order[ti]) : ti;
  float qx = queries[3 * qi], qy = queries[3 * qi + 1], qz = queries[3 * qi + 2];
  float gx = 0.f, gy = 0.f, gz = 0.f;
  if (KERNEL == O8_SOFT_VJP || KERNEL == O8_GRAV_GRAD_VJP) {
    gx = cot[3 * qi];
    gy = cot[3 * qi + 1];
    gz = cot[3 * qi + 2];
  }
  // curand_init(seed + q, 0, 0) and curand_init(seed + q + 0x9e3779b9, 0, 0):
  // int addition, then sign extension (first) or u32 wraparound (second).
  int sq = seed + static_cast<int>(qi);
  curandState st, st2;
  curand_init(static_cast<unsigned long long>(static_cast<long long>(sq)), 0, 0, &st);
  curand_init(static_cast<unsigned long long>(static_cast<unsigned>(sq) + 0x9e3779b9u), 0, 0, &st2);

  float tx = 0.f, ty = 0.f, tz = 0.f;
  for (int sd = 0; sd < nsub; sd++) {
    const OctreeNode8& sub = nodes[subs[sd]];
    if (SOFTENED && o8_prune(sub, qx, qy, qz, prune_on, r_cut_sq, per)) continue;
    uint32_t sub_end = o8_leaf_end(sub.start, sub.end, bd, status);
    if (sub.is_leaf) {
      o8_leaf_sum<KERNEL, true>(leaf, sub.start, sub_end, qx, qy, qz, gx, gy, gz, s, per, tx, ty, tz);
    } else {
      o8_contrib_pair<KERNEL>(sub, qx, qy, qz, gx, gy, gz, s, per, tx, ty, tz);
    }
    if (sub_end <= sub.start) continue;
    uint32_t num_el = sub.end - sub.start;
    float sx = 0.f, sy = 0.f, sz = 0.f;
    for (int ss = 0; ss < samples; ss++) {
      uint32_t pick = min(static_cast<uint32_t>(num_el * curand_uniform(&st2)) + sub.start, sub_end - 1);
      float spx = leaf[pick].pos[0], spy = leaf[pick].pos[1], spz = leaf[pick].pos[2];
      const OctreeNode8* prev = &sub;
      const OctreeNode8* cur = &sub;
      float event_prob = 1.0f;
      float wx = 0.f, wy = 0.f, wz = 0.f;
      float dx = min_image_floor(qx - cur->cx, per);
      float dy = min_image_floor(qy - cur->cy, per);
      float dz = min_image_floor(qz - cur->cz, per);
      float cur_beta = fmaxf(beta, sqrtf(dx * dx + dy * dy + dz * dz) / cur->diameter);
      // Each step goes one level down a tree of depth <= 10; a longer descent
      // follows a cycle in the caller's child indices.
      int steps = 0;
      while (!cur->is_leaf) {
        if (++steps > kO8MaxDescent) {
          raise_status(status, SBH_DEV_ITER_LIMIT);
          break;
        }
        if (SOFTENED && o8_prune(*cur, qx, qy, qz, prune_on, r_cut_sq, per)) break;
        float ex = min_image_floor(qx - cur->cx, per);
        float ey = min_image_floor(qy - cur->cy, per);
        float ez = min_image_floor(qz - cur->cz, per);
        float dist = sqrtf(ex * ex + ey * ey + ez * ez);
        float ffr = dist / cur->diameter;
        float tp = fminf(cur_beta / ffr, 1.0f);
        float p = curand_uniform(&st);
        if (p > tp) {
          event_prob *= 1.0f - tp;
          break;
        }
        event_prob *= tp;
        prev = cur;
        uint32_t slot = o8_child_slot(*cur, spx, spy, spz);
        if (!(cur->child_mask & (1u << slot))) break;
        if (!o8_node_ok(cur->child[slot], bd, status)) break;
        cur = &nodes[cur->child[slot]];
        cur_beta = fmaxf(cur_beta, ffr);
        float px_ = 0.f, py_ = 0.f, pz_ = 0.f;
        o8_contrib_pair<KERNEL>(*prev, qx, qy, qz, gx, gy, gz, s, per, px_, py_, pz_);
        float cx_ = 0.f, cy_ = 0.f, cz_ = 0.f;
        uint8_t mask = prev->child_mask;
        for (int cc = 0; cc < 8; cc++) {
          if (!(mask & (1u << cc))) continue;
          if (!o8_node_ok(prev->child[cc], bd, status)) continue;
          const OctreeNode8& ch = nodes[prev->child[cc]];
          if (SOFTENED && o8_prune(ch, qx, qy, qz, prune_on, r_cut_sq, per)) continue;
          if (ch.is_leaf) {
            o8_leaf_sum<KERNEL, true>(leaf, ch.start, o8_leaf_end(ch.start, ch.end, bd, status), qx, qy, qz, gx, gy,
                                      gz, s, per, cx_, cy_, cz_);
          } else {
            o8_contrib_pair<KERNEL>(ch, qx, qy, qz, gx, gy, gz, s, per, cx_, cy_, cz_);
          }
        }
        float pinv = static_cast<float>(num_el) / (event_prob * static_cast<float>(prev->end - prev->start));
        wx += pinv * (cx_ - px_);
        wy += pinv * (cy_ - py_);
        wz += pinv * (cz_ - pz_);
      }
      sx += wx;
      sy += wy;
      sz += wz;
    }
    if (samples > 0) {
      float inv = static_cast<float>(samples);
      tx += sx / inv;
      ty += sy / inv;
      tz += sz / inv;
    }
  }
  out[3 * qi] = tx;
  out[3 * qi + 1] = ty;
  out[3 * qi + 2] = tz;
}

// ---------------------------------------------------------------------------
// host helpers
// ---------------------------------------------------------------------------
static int check_threads(int threads) {
  if (threads <= 0 || threads > 1024) return invalid("threads must be in [1, 1024]");
  return SBH_OK;
}

static unsigned grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  return static_cast<unsigned>(b < 1 ? 1 : b);
}

// Warps per 32 queries of a direct sum: 16 while two blocks per SM hold all of
// them, then 16, 4 or 1, the one with the least
// estimated time: waves of two blocks per SM (a last wave of at most one block per
// SM counts half), times the chunks of 32 sources that a warp sums and a quarter
// for the block itself, times what a split costs in tile loads and shorter loops, by
// measurement 1.15, 1.1 and 1 (1.03 in a periodic box, where images and erfc
// dominate). Force / VJP, ms on a B200,
// against one warp per 64 queries over every source: 4,096 x 4,096 with erfc on
// nearly every pair 1.46 / 1.61 -> 0.10 / 0.09, 60,000 x 60,000 21.0 / 23.4 -> 10.6 /
// 13.0 (12.9 / 16.0 with 4 warps). Fixed lines at 37,888 and 151,552 queries left nearly empty last
// waves, and idle warps on few sources: 5,000 sources x 151,553 queries,
// periodic, 3.58 / 4.25 with one warp, 2.55 / 3.07 with 16 (3.13 / 3.65 by one query per
// thread); 100 x 151,552 periodic 0.137 / 0.157 with 4, 0.069 / 0.080 with one.
static int direct_split(int64_t n, int64_t nq, bool per) {
  if (nq <= 2 * 148 * 32) return 16;  // all blocks resident at once
  const int64_t tail = (n % kDirectTile + 31) / 32;  // chunks of the last tile
  int best = 1;
  double least = 0.0;
  for (int split = 1; split <= 16; split *= 4) {
    const int64_t blocks = (nq * split + kDirectTile - 1) / kDirectTile, rest = blocks % (2 * 148);
    const double waves = blocks / (2 * 148) + (rest == 0 ? 0.0 : rest <= 148 ? 0.5 : 1.0);
    const double chunks = n / kDirectTile * (kDirectWarps / split) + (tail + split - 1) / split;
    const double cost = waves * (chunks + 0.25) * (split == 1 ? 1.0 : per ? 1.03 : split == 4 ? 1.1 : 1.15);
    if (split == 1 || cost < least) {
      best = split;
      least = cost;
    }
  }
  return best;
}

template <bool VJP, bool PER>
static void direct_launch(cudaStream_t stream, const float* pts, const float* masses, int64_t n, const float* queries,
                          const float* cot, int64_t nq, float* out, Soft s, Periodic per) {
  constexpr int kThreads = 32 * kDirectWarps;
  const int split = direct_split(n, nq, PER);
  if (split == 16) {
    direct_soft_kernel<16, VJP, PER>
        <<<grid_for(nq, kThreads / 16), kThreads, 0, stream>>>(pts, masses, n, queries, cot, nq, out, s, per);
  } else if (split == 4) {
    direct_soft_kernel<4, VJP, PER>
        <<<grid_for(nq, kThreads / 4), kThreads, 0, stream>>>(pts, masses, n, queries, cot, nq, out, s, per);
  } else {
    direct_soft_kernel<1, VJP, PER>
        <<<grid_for(nq, kThreads), kThreads, 0, stream>>>(pts, masses, n, queries, cot, nq, out, s, per);
  }
}

static unsigned grid_stride(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  if (b > 148 * 64) b = 148 * 64;
  return static_cast<unsigned>(b < 1 ? 1 : b);
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <typename Body>
static int o8_layout_checks(const void* leaf, size_t leaf_bytes, const void* nodes, size_t node_bytes,
                            const float* queries, int64_t nq, Body) {
  if (leaf_bytes % sizeof(Leaf3) != 0) return invalid("leaf_bytes size mismatch");
  if (node_bytes % sizeof(OctreeNode8) != 0) return invalid("node_bytes size mismatch");
  if (node_bytes == 0) return invalid("node_bytes must hold at least the root");
  if (nq < 0) return invalid("num_queries must be >= 0");
  if (nq > 0 && !queries) return invalid("queries must be non-null");
  if ((leaf_bytes > 0 && !aligned16(leaf)) || !aligned16(nodes)) return invalid("leaf/node buffers must be 16-byte aligned");
  return SBH_OK;
}

template <typename C>
static void o8_carve(C& c, int64_t n, int depth, O8Params** prm, uint32_t** k0, uint32_t** v0,
                     uint32_t** k1, uint32_t** v1, uint32_t** counts, uint32_t** hist, uint32_t** scan_tmp,
                     DVec<7>** P, DVec<7>** ptmp) {
  uint64_t cells = 1ull << (3 * depth);
  int64_t nn = n > 0 ? n : 1;
  *prm = c.template take<O8Params>(1);
  *k0 = c.template take<uint32_t>(nn);
  *v0 = c.template take<uint32_t>(nn);
  *k1 = c.template take<uint32_t>(nn);
  *v1 = c.template take<uint32_t>(nn);
  *counts = c.template take<uint32_t>(cells + 1);
  int64_t hist_n = radix_hist_elems(nn);
  *hist = c.template take<uint32_t>(hist_n);
  int64_t st = scan_tiles(static_cast<int64_t>(cells) + 1);
  int64_t st2 = scan_tiles(hist_n);
  *scan_tmp = c.template take<uint32_t>(st > st2 ? st : st2);
  *P = c.template take<DVec<7>>(nn + 1);
  *ptmp = c.template take<DVec<7>>(scan_tiles<DVec<7>>(nn));
}

}  // namespace sbh

using namespace sbh;

// Query order of the per-query octree8 traversals. Each query walks the
// tree on its own (the deterministic kernels) or with curand streams seeded
// by its own index (the stochastic ones), so the order in which threads take
// queries changes no result; it only decides which queries share a warp.
// With a large enough workspace the queries are sorted by the 30-bit Morton
// code of their position in the root cell, so a warp's threads walk nearby
// paths and the per-thread traversal diverges far less than for queries in
// random order.
constexpr int64_t kOrderMinQueries = 64;

template <typename C>
static void order_carve(C& c, int64_t nq, uint32_t** k0, uint32_t** v0, uint32_t** k1, uint32_t** v1,
                        uint32_t** hist, uint32_t** tmp) {
  *k0 = c.template take<uint32_t>(static_cast<size_t>(nq));
  *v0 = c.template take<uint32_t>(static_cast<size_t>(nq));
  *k1 = c.template take<uint32_t>(static_cast<size_t>(nq));
  *v1 = c.template take<uint32_t>(static_cast<size_t>(nq));
  int64_t h = radix_hist_elems(nq);
  *hist = c.template take<uint32_t>(static_cast<size_t>(h));
  *tmp = c.template take<uint32_t>(static_cast<size_t>(scan_tiles<uint32_t>(h)));
}

// 10 bits per axis of the query's position in the root cell (clamped; NaN
// goes to 0), interleaved x, y, z from bit 0.
__global__ void o8_query_codes_kernel(const OctreeNode8* __restrict__ nodes, const float* __restrict__ q,
                                      int64_t nq, uint32_t* __restrict__ codes) {
  const float h = nodes[0].half_size;
  const float lo[3] = {nodes[0].cx - h, nodes[0].cy - h, nodes[0].cz - h};
  const float scale = h > 0.0f ? 512.0f / h : 0.0f;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nq;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    uint32_t c = 0;
    for (int d = 0; d < 3; d++) {
      float t = (q[3 * i + d] - lo[d]) * scale;
      uint32_t v = t > 0.0f ? (t < 1023.0f ? static_cast<uint32_t>(t) : 1023u) : 0u;
      for (int b = 0; b < 10; b++) c |= ((v >> b) & 1u) << (3 * b + d);
    }
    codes[i] = c;
  }
}

// The sorted query order, or null (input order) when nq is small or the
// workspace has no room for the sort.
static const uint32_t* o8_query_order(cudaStream_t stream, const OctreeNode8* nodes, const float* queries,
                                      int64_t nq, void* workspace, size_t workspace_bytes, int* rc) {
  *rc = SBH_OK;
  if (nq < kOrderMinQueries || workspace_bytes < sbh_traversal_ordered_workspace_bytes(nq)) return nullptr;
  Carver c(workspace, workspace_bytes);
  uint32_t *k0, *v0, *k1, *v1, *hist, *tmp;
  order_carve(c, nq, &k0, &v0, &k1, &v1, &hist, &tmp);
  o8_query_codes_kernel<<<grid_stride(nq, 256), 256, 0, stream>>>(nodes, queries, nq, k0);
  int which = 0;
  cudaError_t e = radix_sort<uint32_t>(stream, k0, v0, k1, v1, nq, 30, false, hist, tmp, &which);
  if (e != cudaSuccess) {
    *rc = fail(SBH_ERR_CUDA, cudaGetErrorString(e));
    return nullptr;
  }
  return which == 0 ? v0 : v1;
}

// Whether the buffer is a dense octree8 of depth <= 9 ((8^(d+1) - 1) / 7
// nodes), whose DFS never holds more than 64 stack entries.
static bool o8_small_stack(uint32_t num_nodes) {
  uint64_t total = 1, level = 1;
  for (int d = 0; d <= 9; d++) {
    if (total == num_nodes) return true;
    level *= 8;
    total += level;
  }
  return false;
}

// With a periodic box the pairs take the scalar minimum-image form, which
// gains little from staged particles, so that kernel sums each leaf per lane
// straight from global memory and holds fewer registers (TreePM short range,
// 2^21 particles: 16.6 ms against 17.7 ms staged).
template <int KERNEL, int STACK, int WQ>
static void o8_launch_warp_kind(int warps, int per_set, cudaStream_t stream, const Leaf3* L, const OctreeNode8* N,
                                const float* queries, const float* cot, int64_t nq, float beta, Soft s, int prune_on,
                                float r_cut_sq, Periodic per, float* out, uint32_t* status, O8Bounds bd,
                                const uint32_t* order) {
  const unsigned block = 32u * static_cast<unsigned>(warps);
  const unsigned grid = grid_for(nq, WQ > 1 ? per_set : per_set * warps);
  const size_t smem = o8_warp_smem(warps, STACK) + (WQ > 1 ? sizeof(O8UnitSums) : 0);
  if (per.on)
    o8_bh_warp_kernel<KERNEL, STACK, false, WQ><<<grid, block, smem, stream>>>(
        L, N, queries, cot, nq, beta, s, prune_on, r_cut_sq, per, out, status, bd, order, per_set);
  else
    o8_bh_warp_kernel<KERNEL, STACK, true, WQ><<<grid, block, smem, stream>>>(
        L, N, queries, cot, nq, beta, s, prune_on, r_cut_sq, per, out, status, bd, order, per_set);
}

// Eight warps share 32 queries while the query sets alone give the SMs fewer
// than 16 warps each (75,776 queries) and the sums are taken in units; else each
// warp has its own queries and the caller's `threads` gives the warps per block
// (at most 4, so that a block's slowest warp holds up few others: 10^5 queries 7.7
// / 8.5 ms against 8.2 / 9.5 with 8; the result does not depend on it). Softened force / VJP of the
// particles themselves, ms on a B200, shared against own: 5,000 particles 0.55 /
// 0.56 and 2.5 / 2.6 (3.1 / 3.1 before the next node's prefetch), 20,000 1.6 / 1.6
// and 4.2 / 4.3, 60,000 in a uniform cube 5.6 / 5.8 and 6.7 / 6.9, in a Plummer
// sphere 7.2 / 7.5 and 6.3 / 6.8; 10^5 12.5 / 13.2 and 8.5 / 9.7 (9.6 / 10.7 before).
static bool o8_shared_sets(int64_t nq, uint32_t leaves) { return nq <= 148 * 16 * 32 && leaves <= kO8UnitLeaves; }

// Queries per warp that walks them down one stack. The 32 of a warp share visits
// when they are near each other; few queries in a large tree are far apart, and a
// warp then visits up to 32 queries' nodes one after the other while most of the
// chip idles. So below 4,096 queries a warp takes one (up to 16 warps per SM), then
// four. Force, ms on a B200, with 32 per warp / now / one thread per query: 64
// queries of 2^20 uniform particles 56 / 3.6 / 10, 1,000 41 / 4.0 / 15, 4,095 30 /
// 9.7 / 15; of a Plummer sphere 48 / 15 / 270, 36 / 16 / 297, 30 / 19 / 315; 64
// queries of 17,000 uniform particles 11 / 1.9 / 5.0.
static int o8_queries_per_warp(int64_t nq) { return nq >= 4096 ? 32 : nq > 148 * 16 ? 4 : 1; }

template <int KERNEL, int STACK, typename... A>
static void o8_launch_warp_sets(int threads, int64_t nq, uint32_t leaves, cudaStream_t stream, A... args) {
  if (o8_shared_sets(nq, leaves)) {
    o8_launch_warp_kind<KERNEL, STACK, 8>(8, 32, stream, args...);
  } else {
    const int per_warp = o8_queries_per_warp(nq);
    const int warps = threads >= 64 && per_warp == 32 ? (threads < 128 ? threads / 32 : 4) : 1;
    o8_launch_warp_kind<KERNEL, STACK, 1>(warps, per_warp, stream, args...);
  }
}

template <int STACK>
static void o8_launch_warp(int kernel, int threads, cudaStream_t stream, const Leaf3* L, const OctreeNode8* N,
                           const float* queries, const float* cot, int64_t nq, float beta, Soft s, int prune_on,
                           float r_cut_sq, Periodic per, float* out, uint32_t* status, O8Bounds bd,
                           const uint32_t* order) {
  switch (kernel) {
    case O8_GRAV_GRAD:
      o8_launch_warp_sets<O8_GRAV_GRAD, STACK>(threads, nq, bd.num_leaves, stream, L, N, queries, cot, nq, beta, s,
          0, 0.f, per, out, status, bd, order);
      break;
    case O8_SOFT:
      o8_launch_warp_sets<O8_SOFT, STACK>(threads, nq, bd.num_leaves, stream, L, N, queries, cot, nq, beta, s,
          prune_on, r_cut_sq, per, out, status, bd, order);
      break;
    case O8_GRAV_GRAD_VJP:
      o8_launch_warp_sets<O8_GRAV_GRAD_VJP, STACK>(threads, nq, bd.num_leaves, stream, L, N, queries, cot, nq, beta, s,
          0, 0.f, per, out, status, bd, order);
      break;
    default:
      o8_launch_warp_sets<O8_SOFT_VJP, STACK>(threads, nq, bd.num_leaves, stream, L, N, queries, cot, nq, beta, s,
          prune_on, r_cut_sq, per, out, status, bd, order);
      break;
  }
}

extern "C" {

int sbh_bruteforce_gravity(cudaStream_t stream, const float* points, const float* masses, int64_t n, int dim,
                           const float* queries, int64_t nq, float* out, int periodic, float box_length,
                           int threads) {
  if (n < 0 || nq < 0) return invalid("sizes must be >= 0");
  if (dim != 2 && dim != 3) return invalid("only dim=2 or dim=3 supported");
  if (int rc = check_threads(threads)) return rc;
  if (nq == 0) return SBH_OK;
  bruteforce_gravity_kernel<<<grid_for(nq, kDirectThreads), kDirectThreads, 0, stream>>>(
      points, masses, n, dim, queries, nq, out, Periodic{periodic, box_length});
  return check_launch("bruteforce_gravity");
}

int sbh_direct_force_soft(cudaStream_t stream, const float* points, const float* masses, int64_t n,
                          const float* queries, int64_t nq, float* out, float softening_scale,
                          float cutoff_scale, int periodic, float box_length, int threads) {
  if (n < 0 || nq < 0) return invalid("sizes must be >= 0");
  if (softening_scale < 0.0f) return invalid("softening_scale must be >= 0");
  if (!(cutoff_scale > 0.0f)) return invalid("cutoff_scale must be > 0");
  if (int rc = check_threads(threads)) return rc;
  if (nq == 0) return SBH_OK;
  const Soft soft{fmaxf(softening_scale, 0.0f), cutoff_scale};
  if (periodic && box_length > 0.0f)
    direct_launch<false, true>(stream, points, masses, n, queries, nullptr, nq, out, soft,
                               Periodic{periodic, box_length});
  else
    direct_launch<false, false>(stream, points, masses, n, queries, nullptr, nq, out, soft, Periodic{0, 0.0f});
  return check_launch("direct_force_soft");
}

int sbh_direct_force_soft_vjp(cudaStream_t stream, const float* points, const float* masses, int64_t n,
                              const float* queries, int64_t nq, const float* cotangent, float* out,
                              float softening_scale, float cutoff_scale, int periodic, float box_length,
                              int threads) {
  if (n < 0 || nq < 0) return invalid("sizes must be >= 0");
  if (softening_scale < 0.0f) return invalid("softening_scale must be >= 0");
  if (!(cutoff_scale > 0.0f)) return invalid("cutoff_scale must be > 0");
  if (int rc = check_threads(threads)) return rc;
  if (nq == 0) return SBH_OK;
  const Soft soft{fmaxf(softening_scale, 0.0f), cutoff_scale};
  if (periodic && box_length > 0.0f)
    direct_launch<true, true>(stream, points, masses, n, queries, cotangent, nq, out, soft,
                              Periodic{periodic, box_length});
  else
    direct_launch<true, false>(stream, points, masses, n, queries, cotangent, nq, out, soft, Periodic{0, 0.0f});
  return check_launch("direct_force_soft_vjp");
}

size_t sbh_build_octree8_workspace_bytes(int64_t n, int max_depth) {
  if (max_depth < 1 || max_depth > 10 || n < 0) return 0;
  Sizer s;
  O8Params* prm;
  uint32_t *k0, *v0, *k1, *v1, *counts, *hist, *scan_tmp;
  DVec<7>*P, *ptmp;
  o8_carve(s, n, max_depth, &prm, &k0, &v0, &k1, &v1, &counts, &hist, &scan_tmp, &P, &ptmp);
  return s.off;
}

int sbh_build_octree8(cudaStream_t stream, const float* points, const float* normals, const float* masses,
                      int64_t n, const float* min_corner, const float* max_corner, int max_depth, void* leaf_out,
                      size_t leaf_bytes, void* node_out, size_t node_bytes, void* contrib_out,
                      size_t contrib_bytes, void* workspace, size_t workspace_bytes) {
  if (max_depth < 1 || max_depth > 10) return invalid("max_depth must be in [1, 10]");
  if (n < 0 || n > 0xFFFFFFFFll) return invalid("number of points must be in [0, 2^32)");
  uint64_t total = sbh_octree8_total_nodes(max_depth);
  if (leaf_bytes != static_cast<size_t>(n) * sizeof(Leaf3)) return invalid("leaf_out size mismatch");
  if (node_bytes != total * sizeof(OctreeNode8)) return invalid("node_out size mismatch");
  if (contrib_bytes != total * sizeof(Leaf3)) return invalid("contrib_out size mismatch");
  if (!min_corner || !max_corner) return invalid("min_corner/max_corner must be non-null");
  if ((n > 0 && !aligned16(leaf_out)) || !aligned16(node_out) || !aligned16(contrib_out))
    return invalid("output buffers must be 16-byte aligned");
  size_t need = sbh_build_octree8_workspace_bytes(n, max_depth);
  if (!workspace || workspace_bytes < need)
    return fail(SBH_ERR_WORKSPACE, "workspace too small: need " + std::to_string(need) + " bytes");
  Carver c(workspace, workspace_bytes);
  O8Params* prm;
  uint32_t *k0, *v0, *k1, *v1, *counts, *hist, *scan_tmp;
  DVec<7>*P, *ptmp;
  o8_carve(c, n, max_depth, &prm, &k0, &v0, &k1, &v1, &counts, &hist, &scan_tmp, &P, &ptmp);
  uint32_t* status = static_cast<uint32_t*>(workspace);
  uint64_t cells = 1ull << (3 * max_depth);
  cudaError_t e = cudaMemsetAsync(status, 0, sizeof(uint32_t), stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(counts, 0, (cells + 1) * sizeof(uint32_t), stream);
  if (e != cudaSuccess) return fail(SBH_ERR_CUDA, cudaGetErrorString(e));
  o8_setup_kernel<<<1, 1, 0, stream>>>(min_corner, max_corner, prm, status);
  if (n > 0) {
    o8_codes_kernel<<<grid_stride(n, 256), 256, 0, stream>>>(points, n, prm, max_depth, k0, counts);
    int which = 0;
    e = radix_sort<uint32_t>(stream, k0, v0, k1, v1, n, 3 * max_depth, false, hist, scan_tmp, &which);
    if (e != cudaSuccess) return fail(SBH_ERR_CUDA, cudaGetErrorString(e));
    const uint32_t* perm = which == 0 ? v0 : v1;
    o8_gather_kernel<<<grid_stride(n, 256), 256, 0, stream>>>(points, normals, masses, n, perm, prm,
                                                              static_cast<Leaf3*>(leaf_out));
  }
  e = exclusive_scan<uint32_t>(stream, ArrayLoad<uint32_t>{counts}, static_cast<int64_t>(cells), counts, scan_tmp,
                               true);
  if (e != cudaSuccess) return fail(SBH_ERR_CUDA, cudaGetErrorString(e));
  e = exclusive_scan<DVec<7>>(stream, LeafMomentLoad{static_cast<const Leaf3*>(leaf_out)}, n, P, ptmp, true);
  if (e != cudaSuccess) return fail(SBH_ERR_CUDA, cudaGetErrorString(e));
  o8_nodes_kernel<<<grid_stride(static_cast<int64_t>(total), 256), 256, 0, stream>>>(
      static_cast<OctreeNode8*>(node_out), static_cast<Leaf3*>(contrib_out), counts, P, max_depth, total, prm);
  return check_launch("build_octree8");
}

// --------------------------- octree8 traversals -----------------------------
static int o8_launch_bh(int kernel, cudaStream_t stream, const void* leaf, size_t leaf_bytes, const void* nodes,
                        size_t node_bytes, const float* queries, int64_t nq, const float* cot, float* out,
                        float beta, Soft s, int prune_on, float r_cut_sq, Periodic per, int threads,
                        void* workspace, size_t workspace_bytes) {
  if (int rc = o8_layout_checks(leaf, leaf_bytes, nodes, node_bytes, queries, nq, 0)) return rc;
  if (int rc = check_threads(threads)) return rc;
  if (!workspace || workspace_bytes < kStatusBytes) return fail(SBH_ERR_WORKSPACE, "workspace too small");
  uint32_t* status = static_cast<uint32_t*>(workspace);
  cudaError_t e = cudaMemsetAsync(status, 0, sizeof(uint32_t), stream);
  if (e != cudaSuccess) return fail(SBH_ERR_CUDA, cudaGetErrorString(e));
  if (nq == 0) return SBH_OK;
  const Leaf3* L = static_cast<const Leaf3*>(leaf);
  const OctreeNode8* N = static_cast<const OctreeNode8*>(nodes);
  O8Bounds bd{static_cast<uint32_t>(node_bytes / sizeof(OctreeNode8)), static_cast<uint32_t>(leaf_bytes / sizeof(Leaf3))};
  int orc = SBH_OK;
  const uint32_t* order = o8_query_order(stream, N, queries, nq, workspace, workspace_bytes, &orc);
  if (orc != SBH_OK) return orc;
  if (order) {  // Morton-ordered queries: a warp walks 32 neighbours together
    if (o8_small_stack(bd.num_nodes))
      o8_launch_warp<64>(kernel, threads, stream, L, N, queries, cot, nq, beta, s, prune_on, r_cut_sq, per, out, status,
                         bd, order);
    else
      o8_launch_warp<kO8Stack>(kernel, threads, stream, L, N, queries, cot, nq, beta, s, prune_on, r_cut_sq, per, out,
                               status, bd, order);
    return check_launch("barnes_hut_force_octree8");
  }
  unsigned g = grid_for(nq, 256);
  switch (kernel) {
    case O8_GRAV_GRAD:
      o8_bh_kernel<O8_GRAV_GRAD><<<g, 256, 0, stream>>>(L, N, queries, cot, nq, beta, s, 0, 0.f, per, out, status, bd,
                                                        order);
      break;
    case O8_SOFT:
      o8_bh_kernel<O8_SOFT><<<g, 256, 0, stream>>>(L, N, queries, cot, nq, beta, s, prune_on, r_cut_sq, per, out,
                                                   status, bd, order);
      break;
    case O8_GRAV_GRAD_VJP:
      o8_bh_kernel<O8_GRAV_GRAD_VJP><<<g, 256, 0, stream>>>(L, N, queries, cot, nq, beta, s, 0, 0.f, per, out, status,
                                                            bd, order);
      break;
    default:
      o8_bh_kernel<O8_SOFT_VJP><<<g, 256, 0, stream>>>(L, N, queries, cot, nq, beta, s, prune_on, r_cut_sq, per,
                                                       out, status, bd, order);
      break;
  }
  return check_launch("barnes_hut_force_octree8");
}

// prune_on / r_cut exactly as the reference handler derives them (src/sbh_ffi.cu:3235-3237).
static void o8_prune_params(int prune_enabled, float prune_r_cut_mult, float cutoff_scale, int* on, float* rsq) {
  *on = (prune_enabled != 0 && cutoff_scale > 0.0f) ? 1 : 0;
  float r_cut = *on ? prune_r_cut_mult * cutoff_scale : 0.0f;
  *rsq = r_cut * r_cut;
}

int sbh_barnes_hut_force_octree8(cudaStream_t stream, const void* leaf, size_t leaf_bytes, const void* nodes,
                                 size_t node_bytes, const float* queries, int64_t nq, float* out, float beta,
                                 int periodic, float box_length, int threads, void* workspace,
                                 size_t workspace_bytes) {
  return o8_launch_bh(O8_GRAV_GRAD, stream, leaf, leaf_bytes, nodes, node_bytes, queries, nq, nullptr, out, beta,
                      Soft{0.f, 0.f}, 0, 0.f, Periodic{periodic, box_length}, threads, workspace, workspace_bytes);
}

int sbh_barnes_hut_force_octree8_vjp(cudaStream_t stream, const void* leaf, size_t leaf_bytes, const void* nodes,
                                     size_t node_bytes, const float* queries, int64_t nq, const float* cotangent,
                                     float* out, float beta, int periodic, float box_length, int threads,
                                     void* workspace, size_t workspace_bytes) {
  if (nq > 0 && !cotangent) return invalid("cotangent must be non-null");
  return o8_launch_bh(O8_GRAV_GRAD_VJP, stream, leaf, leaf_bytes, nodes, node_bytes, queries, nq, cotangent, out, beta,
                      Soft{0.f, 0.f}, 0, 0.f, Periodic{periodic, box_length}, threads, workspace, workspace_bytes);
}

int sbh_barnes_hut_force_octree8_soft(cudaStream_t stream, const void* leaf, size_t leaf_bytes, const void* nodes,
                                      size_t node_bytes, const float* queries, int64_t nq, float* out, float beta,
                                      float softening_scale, float cutoff_scale, int prune_enabled,
                                      float prune_r_cut_mult, int periodic, float box_length, int threads,
                                      void* workspace, size_t workspace_bytes) {
  if (prune_enabled != 0 && prune_r_cut_mult <= 0.0f)
    return invalid("prune_r_cut_mult must be > 0 when prune_enabled is set");
  int on;
  float rsq;
  o8_prune_params(prune_enabled, prune_r_cut_mult, cutoff_scale, &on, &rsq);
  return o8_launch_bh(O8_SOFT, stream, leaf, leaf_bytes, nodes, node_bytes, queries, nq, nullptr, out, beta,
                      Soft{fmaxf(softening_scale, 0.0f), cutoff_scale}, on, rsq, Periodic{periodic, box_length},
                      threads, workspace, workspace_bytes);
}

int sbh_barnes_hut_force_octree8_soft_vjp(cudaStream_t stream, const void* leaf, size_t leaf_bytes,
                                          const void* nodes, size_t node_bytes, const float* queries, int64_t nq,
                                          const float* cotangent, float* out, float beta, float softening_scale,
                                          float cutoff_scale, int prune_enabled, float prune_r_cut_mult,
                                          int periodic, float box_length, int threads, void* workspace,
                                          size_t workspace_bytes) {
  if (prune_enabled != 0 && prune_r_cut_mult <= 0.0f)
    return invalid("prune_r_cut_mult must be > 0 when prune_enabled is set");
  if (nq > 0 && !cotangent) return invalid("cotangent must be non-null");
  int on;
  float rsq;
  o8_prune_params(prune_enabled, prune_r_cut_mult, cutoff_scale, &on, &rsq);
  return o8_launch_bh(O8_SOFT_VJP, stream, leaf, leaf_bytes, nodes, node_bytes, queries, nq, cotangent, out, beta,
                      Soft{fmaxf(softening_scale, 0.0f), cutoff_scale}, on, rsq, Periodic{periodic, box_length},
                      threads, workspace, workspace_bytes);
}

static int o8_launch_stochastic(bool vjp, int softened, cudaStream_t stream, const void* leaf, size_t leaf_bytes,
                                const void* nodes, size_t node_bytes, const float* queries, int64_t nq,
                                const float* cot, float* out, int samples, int seed, float beta,
                                float softening_scale, float cutoff_scale, int prune_enabled,
                                float prune_r_cut_mult, int periodic, float box_length, int threads,
                                void* workspace, size_t workspace_bytes) {
  if (int rc = o8_layout_checks(leaf, leaf_bytes, nodes, node_bytes, queries, nq, 0)) return rc;
  if (int rc = check_threads(threads)) return rc;
  if (softened && prune_enabled != 0 && prune_r_cut_mult <= 0.0f)
    return invalid("prune_r_cut_mult must be > 0 when prune_enabled is set");
  if (vjp && nq > 0 && !cot) return invalid("cotangent must be non-null");
  if (!workspace || workspace_bytes < kStatusBytes) return fail(SBH_ERR_WORKSPACE, "workspace too small");
  uint32_t* status = static_cast<uint32_t*>(workspace);
  cudaError_t e = cudaMemsetAsync(status, 0, sizeof(uint32_t), stream);
  if (e != cudaSuccess) return fail(SBH_ERR_CUDA, cudaGetErrorString(e));
  if (nq == 0) return SBH_OK;
  int on = 0;
  float rsq = 0.f;
  if (softened) o8_prune_params(prune_enabled, prune_r_cut_mult, cutoff_scale, &on, &rsq);
  Soft s{fmaxf(softening_scale, 0.0f), cutoff_scale};
  Periodic per{periodic, box_length};
  const Leaf3* L = static_cast<const Leaf3*>(leaf);
  const OctreeNode8* N = static_cast<const OctreeNode8*>(nodes);
  O8Bounds bd{static_cast<uint32_t>(node_bytes / sizeof(OctreeNode8)), static_cast<uint32_t>(leaf_bytes / sizeof(Leaf3))};
  // The reference's kernel reads a curand state per query, independent of
  // the block size and of which thread takes the query, so any launch shape
  // and query order give the same numbers.
  int orc = SBH_OK;
  const uint32_t* order = o8_query_order(stream, N, queries, nq, workspace, workspace_bytes, &orc);
  if (orc != SBH_OK) return orc;
  unsigned g = grid_for(nq, kStochThreads);
  if (!vjp) {
    if (softened)
      o8_stochastic_kernel<O8_SOFT, true><<<g, kStochThreads, 0, stream>>>(
          L, N, queries, cot, nq, samples, seed, beta, s, on, rsq, per, out, status, bd, order);
    else
      o8_stochastic_kernel<O8_GRAV_GRAD, false><<<g, kStochThreads, 0, stream>>>(
          L, N, queries, cot, nq, samples, seed, beta, s, 0, 0.f, per, out, status, bd, order);
  } else {
    if (softened)
      o8_stochastic_kernel<O8_SOFT_VJP, true><<<g, kStochThreads, 0, stream>>>(
          L, N, queries, cot, nq, samples, seed, beta, s, on, rsq, per, out, status, bd, order);
    else
      o8_stochastic_kernel<O8_GRAV_GRAD_VJP, false><<<g, kStochThreads, 0, stream>>>(
          L, N, queries, cot, nq, samples, seed, beta, s, 0, 0.f, per, out, status, bd, order);
  }
  return check_launch("stochastic_bh_force_octree8");
}

size_t sbh_traversal_ordered_workspace_bytes(int64_t nq) {
  if (nq < 0) return 0;
  Sizer z;
  uint32_t *k0, *v0, *k1, *v1, *hist, *tmp;
  order_carve(z, nq, &k0, &v0, &k1, &v1, &hist, &tmp);
  return z.off;
}

int sbh_stochastic_bh_force_octree8(cudaStream_t stream, int softened, const void* leaf, size_t leaf_bytes,
                                    const void* nodes, size_t node_bytes, const float* queries, int64_t nq,
                                    float* out, int samples_per_subdomain, int seed, float beta,
                                    float softening_scale, float cutoff_scale, int prune_enabled,
                                    float prune_r_cut_mult, int periodic, float box_length, int threads,
                                    void* workspace, size_t workspace_bytes) {
  return o8_launch_stochastic(false, softened, stream, leaf, leaf_bytes, nodes, node_bytes, queries, nq, nullptr,
                              out, samples_per_subdomain, seed, beta, softening_scale, cutoff_scale, prune_enabled,
                              prune_r_cut_mult, periodic, box_length, threads, workspace, workspace_bytes);
}

int sbh_stochastic_bh_force_octree8_vjp(cudaStream_t stream, int softened, const void* leaf, size_t leaf_bytes,
                                        const void* nodes, size_t node_bytes, const float* queries, int64_t nq,
                                        const float* cotangent, float* out, int samples_per_subdomain, int seed,
                                        float beta, float softening_scale, float cutoff_scale, int prune_enabled,
                                        float prune_r_cut_mult, int periodic, float box_length, int threads,
                                        void* workspace, size_t workspace_bytes) {
  return o8_launch_stochastic(true, softened, stream, leaf, leaf_bytes, nodes, node_bytes, queries, nq, cotangent,
                              out, samples_per_subdomain, seed, beta, softening_scale, cutoff_scale, prune_enabled,
                              prune_r_cut_mult, periodic, box_length, threads, workspace, workspace_bytes);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// octree8 build with library-owned scratch (no allocation by the caller or
// by the library at call time)
// ---------------------------------------------------------------------------
// Some callers cannot allocate device memory when they need a tree: an XLA
// custom call running under JAX's default preallocation (the framework holds
// most of the GPU, so a cudaMalloc from inside the handler can fail), code
// that runs with a fixed, pre-reserved memory budget, or a caller that must
// not trigger the implicit device synchronisation a cudaMalloc may cause.
// For them this variant of sbh_build_octree8 takes its temporaries from one
// fixed array that is part of the library image. Every GPU that loads the
// library holds these bytes until the process exits. The build clears what
// must start at zero (status word, cell counters) on every call, so what an
// earlier call left in the array does not matter. Calls that may overlap on
// the GPU (two streams, or two host threads) share the array and race: the
// caller serialises them.
namespace {

constexpr size_t kStaticScratchBytes = size_t(16) << 20;  // 16 MiB
__device__ __align__(256) unsigned char g_o8_static_scratch[kStaticScratchBytes];

std::mutex g_static_mu;
void* g_static_addr[128] = {};  // device address of the array, per device ordinal

// Device address of the scratch on the current device. On the host the
// array's name only stands for the device symbol; the address a kernel can
// use comes from cudaGetSymbolAddress with that device current.
int static_scratch(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(SBH_ERR_CUDA, cudaGetErrorString(e));
  if (dev < 0 || dev >= 128) return fail(SBH_ERR_CUDA, "device ordinal out of range");
  std::lock_guard<std::mutex> lk(g_static_mu);
  if (!g_static_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_o8_static_scratch);
    if (e != cudaSuccess || !p) return fail(SBH_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    g_static_addr[dev] = p;
  }
  *out = g_static_addr[dev];
  return SBH_OK;
}

}  // namespace

extern "C" {

size_t sbh_build_octree8_static_scratch_bytes(void) { return kStaticScratchBytes; }

int sbh_build_octree8_static(cudaStream_t stream, const float* points, const float* normals, const float* masses,
                             int64_t n, const float* min_corner, const float* max_corner, int max_depth,
                             void* leaf_out, size_t leaf_bytes, void* node_out, size_t node_bytes, void* contrib_out,
                             size_t contrib_bytes) {
  if (max_depth < 1 || max_depth > 10) return invalid("max_depth must be in [1, 10]");
  if (n < 0) return invalid("number of points must be >= 0");
  size_t need = sbh_build_octree8_workspace_bytes(n, max_depth);
  if (need > kStaticScratchBytes)
    return invalid("n = " + std::to_string(n) + " at max_depth = " + std::to_string(max_depth) + " needs " +
                   std::to_string(need) + " bytes of scratch; the built-in scratch holds " +
                   std::to_string(kStaticScratchBytes) + " (use sbh_build_octree8 with a workspace)");
  void* ws = nullptr;
  if (int rc = static_scratch(&ws)) return rc;
  return sbh_build_octree8(stream, points, normals, masses, n, min_corner, max_corner, max_depth, leaf_out, leaf_bytes,
                           node_out, node_bytes, contrib_out, contrib_bytes, ws, kStaticScratchBytes);
}

}  // extern "C"
