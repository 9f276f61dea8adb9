// gr_diff.cu -- differentiable shading on top of the exact visibility pass.
//
// This is an extension with no counterpart in the reference renderer.  The
// frame pipeline (gr_kernels.cu) resolves visibility exactly as
// FrameBuffer.Triangle does (rasterizer.go:90-183) and, for views flagged
// kViewFaceIds, writes the winning face per pixel instead of a colour.  The
// kernels here add a smooth shading model over that fixed visibility:
//
//   screen position of corner i   s_i = S * (clip_i / W_i)          clip_i = MVP * p_i
//   edge functions at pixel (x,y) e_0 = (x1-x)(y2-y) - (x2-x)(y1-y)  (and cyclic)
//   perspective barycentrics      b_i = (e_i / W_i) / sum_j (e_j / W_j)
//   clipped to the triangle       l_i = max(b_i, 0) / sum_j max(b_j, 0)
//
// The barycentrics are evaluated in the 2D homogeneous form (Olano and Greer,
// "Triangle scan conversion using 2D homogeneous coordinates", 1997), which
// needs no perspective divide: with Q = S * MVP,
//   u_i = (Q_0 - x Q_3) . p_i,  v_i = (Q_1 - y Q_3) . p_i       (= (s_i - pixel) * W_i)
//   D_0 = u_1 v_2 - u_2 v_1 (and cyclic),  b_i = D_i / (D_0 + D_1 + D_2)
// u and v cancel screen positions of hundreds of pixels down to a few, and on
// thin faces D amplifies what is left, so float32 would leave relative errors
// up to ~1e-3: hx = Q_0.p, hy = Q_1.p and W = Q_3.p are computed once per
// (view, vertex) in double and kept as float-float pairs, and u, v and D are
// formed per pixel in float-float arithmetic (error-free sums and products,
// Dekker 1971; Knuth, TAOCP vol. 2) on the float32 pipes, which on this GPU
// run about 64 times as many operations as the double-precision ones.
// The barycentrics are homogeneous of degree 0 in D, so the clip and the
// normalisation run in float32 on D's correctly signed values:
//   l_i = max(s D_i, 0) / sum_j max(s D_j, 0),  s = sign(D_0 + D_1 + D_2).
// The backward chain runs in float32 from those values and from per-column
// and per-row tables of Q_0 - x Q_3 and Q_1 - y Q_3 (exact in double, then
// rounded).
//   colour                        c   = sum_i l_i c_i               (vertex RGB)
//   intensity                     I   = sum_i l_i (0.5 + 0.5 nhat_i . L)
//   texel                         t   = tex[floor(v th) mod th][floor(u tw) mod tw],  (u,v) = sum_i l_i uv_i
//   pixel                         out = (I c_r t_r, I c_g t_g, I c_b t_b, t_a)
//   loss                          sum over pixels and channels of (out - target)^2
//
// nhat_i is the renderer's Gouraud normal, xyz of Vec4.Normalize(world * n)
// (renderer.go:328-331); vertex normals are fixed inputs.  The forward pass
// stores per pixel the face, the texel and (l0, l1); the backward pass reads
// them back, recomputes the shading and accumulates the gradients of the loss
// with respect to vertex colours, texels, the light direction and vertex
// positions.  Position gradients flow through the barycentrics only (the
// interior term): visibility and texel choices are held fixed.

#include <cuda_runtime.h>

#include <algorithm>

#include "gr_internal.h"

namespace gr {

namespace {

constexpr int kThreads = kDiffThreads;
static_assert(kDiffSlots == kThreads, "sum_slots takes a slot a thread");

// Waits for the kernel ahead on the stream (launch_after); a no-op after a
// plain launch.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Go's min and max of floats (NaN wins, -0 below +0) as those of unsigned
// keys, so that a warp reduces with one instruction.
template <bool MAX>
__device__ __forceinline__ uint32_t go_key(float a) {
  const uint32_t u = __float_as_uint(a);
  if (a != a) return MAX ? ~0u : 0u;
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float go_value(uint32_t k) {
  if (k == 0u || k == ~0u) return __int_as_float(0x7fc00000);
  return __uint_as_float(k & 0x80000000u ? k & 0x7FFFFFFFu : ~k);
}

// Mesh.BoundingBox (mesh.go:28-51) of pos; min and max are order-free, so a
// tree reduction gives the sequential loop's result.  Each CTA reduces a
// grid-strided share into partial[6 * block]; the last CTA to finish (an
// atomic counter, no waiting) reduces the partials and writes the corners and
// each item's visibility.  Bound by the latency of those steps one after the
// other: a warp an item, a lane a corner of its box (one thread doing the eight
// corners of an item took as long as the rest), and the items' tables are
// waited for only there, so the positions are read while k_stage copies them.
// 642 vertices, 3 views: 11.5 -> 4.4 us; 40,962 vertices, 64 views: 13.9 -> 6.9.
__global__ void __launch_bounds__(1024) k_diff_bbox(const float* __restrict__ pos, int nv, DevItem* items,
                                                    int num_items, uint32_t* partial, unsigned* done) {
  __shared__ uint32_t s_v[6][32];
  __shared__ float s_b[32];
  __shared__ unsigned s_last;
  const int tid = threadIdx.x;
  uint32_t m[6] = {~0u, ~0u, ~0u, 0u, 0u, 0u};  // min x, y, z, max x, y, z
  for (int i = blockIdx.x * blockDim.x + tid; i < nv; i += gridDim.x * blockDim.x) {
    const float4 p = reinterpret_cast<const float4*>(pos)[i];
    const float c[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      m[k] = min(m[k], go_key<false>(c[k]));
      m[3 + k] = max(m[3 + k], go_key<true>(c[k]));
    }
  }
  auto reduce = [&]() {  // over the warp
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      m[k] = __reduce_min_sync(0xffffffffu, m[k]);
      m[3 + k] = __reduce_max_sync(0xffffffffu, m[3 + k]);
    }
  };
  reduce();
  const int warp = tid >> 5, lane = tid & 31;
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < 6; ++k) s_v[k][warp] = m[k];
  }
  __syncthreads();
  if (warp == 0) {  // 32 warps
#pragma unroll
    for (int k = 0; k < 6; ++k) m[k] = s_v[k][lane];
    reduce();
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < 6; ++k) partial[6 * blockIdx.x + k] = m[k];
      __threadfence();
      s_last = atomicAdd(done, 1u) == gridDim.x - 1u ? 1u : 0u;
    }
  }
  griddep_wait();  // the items' matrices; no CTA ends before the kernels ahead have
  __syncthreads();
  if (!s_last) return;
  if (warp == 0) {
    __threadfence();
    const volatile uint32_t* pv = partial;
    for (unsigned b = (unsigned)lane; b < gridDim.x; b += 32) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        m[k] = min(m[k], pv[6 * b + k]);
        m[3 + k] = max(m[3 + k], pv[6 * b + 3 + k]);
      }
    }
    reduce();
    if (lane == 0) *done = 0u;  // ready for the next forward pass
    // corners in mesh.go's order: x outermost, then y, then z; w = 1
    const int c = lane >> 2, k = lane & 3;
    const uint32_t key = k == 0 ? m[c & 4 ? 3 : 0] : k == 1 ? m[c & 2 ? 4 : 1] : m[c & 1 ? 5 : 2];
    s_b[lane] = k == 3 ? 1.0f : go_value(key);
  }
  __syncthreads();
  // and each view's BoxVisibility of this box, which k_vertex and k_cull read
  for (int i = warp; i < num_items; i += (int)blockDim.x / 32) {
    items[i].bbox[lane] = s_b[lane];
    const unsigned out = box_corner_outside(items[i].mvp, s_b + 4 * (lane & 7));
    unsigned some = out, all = out;
    for (int o = 4; o > 0; o >>= 1) {
      some |= __shfl_xor_sync(0xffffffffu, some, o);
      all &= __shfl_xor_sync(0xffffffffu, all, o);
    }
    if (lane == 0) items[i].vis = box_visibility(some, all);
  }
}

__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

__device__ __forceinline__ float4 mvp_apply(const float* m, float4 v) {
  float4 r;
  r.x = m[0] * v.x + m[1] * v.y + m[2] * v.z + m[3] * v.w;
  r.y = m[4] * v.x + m[5] * v.y + m[6] * v.z + m[7] * v.w;
  r.z = m[8] * v.x + m[9] * v.y + m[10] * v.z + m[11] * v.w;
  r.w = m[12] * v.x + m[13] * v.y + m[14] * v.z + m[15] * v.w;
  return r;
}

__global__ void __launch_bounds__(kThreads) k_diff_normals(const float* __restrict__ world,
                                                           const float* __restrict__ vnrm, int nn, float* nhat) {
  const int n = blockIdx.x * kThreads + threadIdx.x;
  if (n >= nn) return;
  const float4 v = mvp_apply(world, ldg4(vnrm + 4 * (size_t)n));
  const float len = __fsqrt_rn(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
  reinterpret_cast<float4*>(nhat)[n] = make_float4(v.x / len, v.y / len, v.z / len, 0.0f);
}

// Float-float arithmetic: a value is hi + lo with |lo| <= ulp(hi) / 2.
struct FF {
  float hi, lo;
};
__device__ __forceinline__ FF two_sum(float a, float b) {  // exact: s + e = a + b
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return FF{s, e};
}
__device__ __forceinline__ FF fast_two_sum(float a, float b) {  // exact when |a| >= |b|
  const float s = __fadd_rn(a, b);
  return FF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FF ff_sub(FF a, FF b) {
  FF s = two_sum(a.hi, -b.hi);
  s.lo = __fadd_rn(s.lo, __fsub_rn(a.lo, b.lo));
  return fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ FF ff_add(FF a, FF b) {
  FF s = two_sum(a.hi, b.hi);
  s.lo = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
  return fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ FF ff_mul(FF a, FF b) {  // the product of the his is exact with an FMA
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fadd_rn(e, __fadd_rn(__fmul_rn(a.hi, b.lo), __fmul_rn(a.lo, b.hi)));
  return fast_two_sum(p, e);
}

// A sum of floats as three: the additions' errors go to the next part, so it holds
// some 70 bits (a double's sum rounds at each addition to 53), on the float32 pipes.
struct Sum3 {
  float hi = 0.0f, mid = 0.0f, lo = 0.0f;
  __device__ __forceinline__ void add(float x) {
    const FF t = two_sum(hi, x), u = two_sum(mid, t.lo);
    hi = t.hi;
    mid = u.hi;
    lo = __fadd_rn(lo, u.lo);
  }
  __device__ __forceinline__ void add_lanes() {  // over the warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const FF t = two_sum(hi, __shfl_xor_sync(0xffffffffu, hi, o)), u = two_sum(mid, __shfl_xor_sync(0xffffffffu, mid, o)),
               v = two_sum(u.hi, t.lo);
      lo = __fadd_rn(__fadd_rn(lo, __shfl_xor_sync(0xffffffffu, lo, o)), __fadd_rn(u.lo, v.lo));
      hi = t.hi;
      mid = v.hi;
    }
  }
  __device__ __forceinline__ double value() const { return (double)hi + ((double)mid + (double)lo); }
};

__device__ __forceinline__ FF ff_mul_f(FF a, float b) {
  const float p = __fmul_rn(a.hi, b);
  float e = __fmaf_rn(a.hi, b, -p);
  e = __fadd_rn(e, __fmul_rn(a.lo, b));
  return fast_two_sum(p, e);
}

// Per face, once for the mesh: its vertex and normal indices and corner UVs
// side by side (64 bytes, the indices and the first UV in 32), so that a pixel
// reads two words instead of twelve.  *apart: some normal index differs from
// its vertex index.
__global__ void __launch_bounds__(kThreads) k_diff_faces(const int* __restrict__ vidx, const int* __restrict__ nidx,
                                                         const float* __restrict__ uv, int nf, int4* out, int* apart) {
  const int f = blockIdx.x * kThreads + threadIdx.x;
  if (f >= nf) return;
  const int* v = vidx + 3 * (size_t)f;
  const int* n = nidx + 3 * (size_t)f;
  int t[6] = {0, 0, 0, 0, 0, 0};
  if (uv)
    for (int k = 0; k < 6; ++k) t[k] = __float_as_int(uv[6 * (size_t)f + k]);
  int4* o = out + 4 * (size_t)f;
  o[0] = make_int4(v[0], v[1], v[2], n[0]);
  o[1] = make_int4(n[1], n[2], t[0], t[1]);
  o[2] = make_int4(t[2], t[3], t[4], t[5]);
  o[3] = make_int4(0, 0, 0, 0);
  if (v[0] != n[0] || v[1] != n[1] || v[2] != n[2]) *apart = 1;
}

// 32 bytes (one sector), p 32-byte aligned.
struct Word8 {
  uint32_t x[8];
};
__device__ __forceinline__ Word8 ldg8(const void* p) {
  const uint4 a = __ldg(reinterpret_cast<const uint4*>(p)), b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
  return Word8{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}

// Gouraud intensity of normal i.
__device__ __forceinline__ float lit_of(const DiffArgs& a, int i) {
  const float4 n = ldg4(a.nhat + 4 * (size_t)i);
  return 0.5f + 0.5f * (n.x * a.L[0] + n.y * a.L[1] + n.z * a.L[2]);
}

// What the pixels of a pass gather, in one launch.  Blocks [0, a.vert_blocks)
// of a view: per vertex homogeneous screen x and y and clip W as float pairs,
// Q.p formed in float-float from Q's float pairs (the products of Q's hi and
// the float coordinates are exact with an FMA; ~48-bit significands, more
// than the geometry needs, with no FP64 instruction), in one 32-byte sector;
// for the first view also the vertex's colour as one word, with its intensity
// where the mesh's normals have the vertices' indices.  Blocks up to
// a.vert_blocks + a.norm_blocks of the first view: the Gouraud intensity of
// every normal.  The others: Q_0 - x Q_3 for every column x and Q_1 - y Q_3 for every
// row y (d u / d p and d v / d p), evaluated in double and rounded to float.
__global__ void __launch_bounds__(kThreads) k_diff_prepare(const DiffArgs a) {
  const DiffView& vw = a.views[blockIdx.y];
  if ((int)blockIdx.x < a.vert_blocks) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= a.nv) return;
    const float4 p = ldg4(a.pos + 4 * (size_t)i);
    const float c[3] = {p.x, p.y, p.z};
    float h[6];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const float* q = vw.Qf + 8 * r;
      FF d{q[6], q[7]};
#pragma unroll
      for (int j = 0; j < 3; ++j) d = ff_add(d, ff_mul_f(FF{q[2 * j], q[2 * j + 1]}, c[j]));
      h[2 * r] = d.hi;
      h[2 * r + 1] = d.lo;
    }
    float4* o = a.vh + 2 * ((size_t)blockIdx.y * (size_t)a.nv + (size_t)i);
    o[0] = make_float4(h[0], h[1], h[2], h[3]);
    o[1] = make_float4(h[4], h[5], 0.0f, 0.0f);
    if (blockIdx.y == 0) {
      const float* cp = a.vcol + 3 * (size_t)i;
      a.col4[i] = make_float4(__ldg(cp), __ldg(cp + 1), __ldg(cp + 2), !a.apart && i < a.nn ? lit_of(a, i) : 0.0f);
    }
    return;
  }
  int i = ((int)blockIdx.x - a.vert_blocks) * kThreads + threadIdx.x;
  if ((int)blockIdx.x < a.vert_blocks + a.norm_blocks) {
    if (blockIdx.y == 0 && i < a.nn) a.lit[i] = lit_of(a, i);
    return;
  }
  i -= a.norm_blocks * kThreads;
  if (i < vw.W) {
    float4 r;
    r.x = (float)__fma_rn(-(double)i, vw.Q[8], vw.Q[0]);
    r.y = (float)__fma_rn(-(double)i, vw.Q[9], vw.Q[1]);
    r.z = (float)__fma_rn(-(double)i, vw.Q[10], vw.Q[2]);
    r.w = 0.0f;
    a.col_tab[vw.col_base + i] = r;
  }
  if (i < vw.H) {
    float4 r;
    r.x = (float)__fma_rn(-(double)i, vw.Q[8], vw.Q[4]);
    r.y = (float)__fma_rn(-(double)i, vw.Q[9], vw.Q[5]);
    r.z = (float)__fma_rn(-(double)i, vw.Q[10], vw.Q[6]);
    r.w = 0.0f;
    a.row_tab[vw.row_base + i] = r;
  }
}

// Geometry of one face at one pixel, shared by the forward and backward passes
// so that both compute bit-identical values.
struct FaceGeom {
  int vi[3];
  float u[3], v[3];   // (s_i - pixel) * W_i, rounded from double
  float d[3];         // s * D_i, rounded from double (s = sign of the sum)
  float m[3], M;      // max(d_i, 0) and their sum
  float sg;           // s
  bool ok;
};

__device__ __forceinline__ void face_geom(const DiffArgs& a, int view, const Word8& face, int px, int py,
                                          FaceGeom& g) {
  const float X = (float)px, Y = (float)py;  // exact (< 2^24)
  FF u[3], v[3];
  g.ok = true;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    g.vi[k] = (int)face.x[k];
    const Word8 h = ldg8(a.vh + 2 * ((size_t)view * (size_t)a.nv + (size_t)g.vi[k]));
    const float2 hx = make_float2(__uint_as_float(h.x[0]), __uint_as_float(h.x[1]));
    const float2 hy = make_float2(__uint_as_float(h.x[2]), __uint_as_float(h.x[3]));
    const float2 w = make_float2(__uint_as_float(h.x[4]), __uint_as_float(h.x[5]));
    const FF W{w.x, w.y};
    g.ok = g.ok && W.hi < 0.0f;  // in front of the camera (W is negative there)
    u[k] = ff_sub(FF{hx.x, hx.y}, ff_mul_f(W, X));
    v[k] = ff_sub(FF{hy.x, hy.y}, ff_mul_f(W, Y));
    g.u[k] = __fadd_rn(u[k].hi, u[k].lo);
    g.v[k] = __fadd_rn(v[k].hi, v[k].lo);
  }
  const FF D0 = ff_sub(ff_mul(u[1], v[2]), ff_mul(u[2], v[1]));
  const FF D1 = ff_sub(ff_mul(u[2], v[0]), ff_mul(u[0], v[2]));
  const FF D2 = ff_sub(ff_mul(u[0], v[1]), ff_mul(u[1], v[0]));
  const FF T = ff_add(ff_add(D0, D1), D2);
  g.sg = T.hi < 0.0f ? -1.0f : 1.0f;
  g.d[0] = g.sg * __fadd_rn(D0.hi, D0.lo);
  g.d[1] = g.sg * __fadd_rn(D1.hi, D1.lo);
  g.d[2] = g.sg * __fadd_rn(D2.hi, D2.lo);
#pragma unroll
  for (int k = 0; k < 3; ++k) g.m[k] = fmaxf(g.d[k], 0.0f);
  g.M = g.m[0] + g.m[1] + g.m[2];
  g.ok = g.ok && T.hi != 0.0f && g.M > 0.0f && isfinite(g.M);
}

struct Shade {
  float l[3];
  float c[3][3];    // vertex colours
  float Ii[3];      // corner intensities
  float col[3];     // interpolated colour
  float I;
  float4 t;         // texel
  float4 out;
};

__device__ __forceinline__ void shade(const DiffArgs& a, const FaceGeom& g, float l0, float l1, uint32_t texel,
                                      const int* ni, Shade& s) {
  s.l[0] = l0;
  s.l[1] = l1;
  s.l[2] = 1.0f - l0 - l1;
  s.I = 0.0f;
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) s.col[ch] = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float4 c = __ldg(a.col4 + g.vi[k]);
    s.Ii[k] = a.apart ? __ldg(a.lit + ni[k]) : c.w;
    s.I += s.l[k] * s.Ii[k];
    s.c[k][0] = c.x; s.c[k][1] = c.y; s.c[k][2] = c.z;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) s.col[ch] += s.l[k] * s.c[k][ch];
  }
  s.t = texel != kNoFace ? ldg4(a.tex + 4 * (size_t)texel) : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
  s.out = make_float4(s.I * s.col[0] * s.t.x, s.I * s.col[1] * s.t.y, s.I * s.col[2] * s.t.z, s.t.w);
}

__device__ __forceinline__ int wrap_index(float u, int n) {
  const float f = floorf(u * (float)n);
  if (!(f > -2.0e9f && f < 2.0e9f)) return 0;
  int i = (int)f;
  if ((unsigned)i < (unsigned)n) return i;
  i %= n;
  return i < 0 ? i + n : i;
}

// The pixels of a thread: column x of its view, rows y, y + rows, ..., a.blocks_down
// of them.  A CTA's warps take an 8 x 4 block each (blocks share more faces, and so more
// gathered lines, than rows of 32 do), side by side first (diff_block_shift).
struct Pixels {
  int view, x, y, rows;
};

// The CTAs of all views stand in one list, so that each view has those that its own
// size asks for (a grid of the largest width by the largest height made 2048 x 64
// views beside 64 x 2048 ones three times as slow, and numbers of CTAs beyond 32 bits).
// Views of as many CTAs each, the usual case, need a division; others a search, 32
// views a round and the same in every warp.
__device__ __forceinline__ Pixels block_pixels(const DiffArgs& a) {
  int view = 0;
  if (a.view_blocks) {
    view = (int)(blockIdx.x / a.view_blocks);
  } else {
    const int lane = (int)(threadIdx.x & 31u);
    int hi = a.num_views - 1;  // the last view whose first CTA is at most this one lies in [view, hi]
    while (view < hi) {
      const int step = (hi - view + 31) >> 5, p = view + 1 + lane * step;
      const unsigned got = __ballot_sync(0xffffffffu, p <= hi && a.views[p].block_base <= blockIdx.x);
      if (!got) break;
      view += 1 + (31 - __clz((int)got)) * step;
      hi = min(hi, view + step - 1);
    }
  }
  const DiffView& vw = a.views[view];
  const int local = (int)(blockIdx.x - vw.block_base);
  const int by = local / vw.blocks_x, bx = local - by * vw.blocks_x;
  const int sh = diff_block_shift(vw.W), rows = kThreads >> sh, warp = (int)(threadIdx.x >> 5);
  const int wy = warp >> (sh - 3), wx = warp & ((1 << (sh - 3)) - 1);
  return Pixels{view, (bx << sh) + wx * 8 + (int)(threadIdx.x & 7u),
                by * a.blocks_down * rows + wy * 4 + (int)((threadIdx.x >> 3) & 3u), rows};
}

// The calling warp's slot of DiffArgs::partials (warps spread over the slots
// so that their atomics rarely meet).
__device__ __forceinline__ int diff_slot() {
  return (int)((blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) & (kDiffSlots - 1));
}

// The last of a grid's CTAs to get here (an atomic counter, no waiting) writes
// the sums of components [c0, c0 + N) of the slots to dst (page-locked host
// memory, through its device address: no copy follows) and returns the slots and
// the counter to zero.  Called by every thread.
template <int N>
__device__ __forceinline__ void sum_slots(const DiffArgs& a, int c0, double* dst) {
  __shared__ double s_w[N][kThreads / 32];
  __shared__ bool s_last;
  if ((threadIdx.x & 31) == 0) __threadfence();  // the warp's slot sums before the count
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(a.done, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double* p = a.partials + 4 * threadIdx.x + c0;  // kDiffSlots = kThreads
  double t[N];
#pragma unroll
  for (int j = 0; j < N; ++j) t[j] = __ldcg(p + j);
#pragma unroll
  for (int j = 0; j < N; ++j) p[j] = 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int j = 0; j < N; ++j) t[j] += __shfl_xor_sync(0xffffffffu, t[j], o);
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int j = 0; j < N; ++j) s_w[j][threadIdx.x >> 5] = t[j];
  }
  __syncthreads();
  if (threadIdx.x < N) {
    double sum = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) sum += s_w[threadIdx.x][w];
    dst[threadIdx.x] = sum;
  }
  if (threadIdx.x == 0) *a.done = 0u;
}

// Forward: per pixel record, shaded pixel and the loss.  Bound by the latency of
// its gathers (face, then corners, then texel: 46 % of the issue slots, 38 % of
// the memory rate).  64 views of 512 x 512 pixels of an 81,920-face mesh: 394 -> 233
// us with the gathered data packed (36 loads a covered pixel before, 13 now),
// blocks instead of rows of pixels a warp, and the loss out of the FP64 pipe as
// two floats; 245 with three, which hold all of its bits.
__global__ void __launch_bounds__(kThreads, 4) k_diff_shade(const DiffArgs a) {
  griddep_wait();
  const Pixels at = block_pixels(a);
  const DiffView& vw = a.views[at.view];
  const int px = at.x;
  // the pixels' losses, summed as three floats, no less exact than in FP64 (the warp's
  // sum goes to FP64), since FP64 additions, one a pixel or five for each warp's
  // tree, held this kernel at the FP64 pipe's rate.  (Two floats round to about
  // 46 bits.)  Losses near float32's end, and infinities and NaN, are summed
  // apart, scaled by 2^-80, as two floats: multiples of 2^16 up to 2^48 then, 256 at
  // most, so the low part is a multiple of 2^16 up to 2^39 and exact too.
  Sum3 sum;
  float bhi = 0.0f, blo = 0.0f;
  for (int k = 0; k < a.blocks_down; ++k) {
    const int py = at.y + k * at.rows;
    if (px >= vw.W || py >= vw.H) break;
    const size_t gp = (size_t)vw.pix_base + (size_t)py * (size_t)vw.W + (size_t)px;
    const uint32_t gf = a.ids[gp];
    const float4 tg = __ldcs(reinterpret_cast<const float4*>(a.target) + gp);
    DiffRecord rec{kNoFace, kNoFace, 0.0f, 0.0f};
    float4 out = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (gf != kNoFace) {
      const int4* fr = a.faces + 4 * (size_t)(gf - vw.face_base);
      const Word8 face = ldg8(fr);
      FaceGeom g;
      face_geom(a, at.view, face, px, py, g);
      if (g.ok) {
        // the visibility pass snaps corners to whole pixels, so a pixel may lie
        // just outside the unsnapped face: its barycentrics are clipped to it
        const float l0 = g.m[0] / g.M, l1 = g.m[1] / g.M;
        uint32_t texel = kNoFace;
        if (a.tex && a.uv) {
          const float l2 = 1.0f - l0 - l1;
          const int4 r2 = __ldg(fr + 2);
          const float u = l0 * __uint_as_float(face.x[6]) + l1 * __int_as_float(r2.x) + l2 * __int_as_float(r2.z);
          const float v = l0 * __uint_as_float(face.x[7]) + l1 * __int_as_float(r2.y) + l2 * __int_as_float(r2.w);
          texel = (uint32_t)(wrap_index(v, a.th) * a.tw + wrap_index(u, a.tw));
        }
        Shade s;
        const int ni[3] = {(int)face.x[3], (int)face.x[4], (int)face.x[5]};
        shade(a, g, l0, l1, texel, ni, s);
        out = s.out;
        rec = DiffRecord{gf, texel, l0, l1};
      }
    }
    reinterpret_cast<uint4*>(a.rec)[gp] =
        make_uint4(rec.face, rec.texel, __float_as_uint(rec.l0), __float_as_uint(rec.l1));
    if (a.image) reinterpret_cast<float4*>(a.image)[gp] = out;
    const float dx = out.x - tg.x, dy = out.y - tg.y, dz = out.z - tg.z, dw = out.w - tg.w;
    const float lp = dx * dx + dy * dy + dz * dz + dw * dw;
    if (lp < 1e36f) {
      sum.add(lp);
    } else {
      const FF t = two_sum(bhi, lp * 0x1p-80f);
      bhi = t.hi;
      blo = __fadd_rn(blo, t.lo);
    }
  }
  sum.add_lanes();
  double loss = sum.value();
  if (__any_sync(0xffffffffu, bhi != 0.0f)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const FF t = two_sum(bhi, __shfl_xor_sync(0xffffffffu, bhi, o));
      blo = __fadd_rn(__fadd_rn(blo, __shfl_xor_sync(0xffffffffu, blo, o)), t.lo);
      bhi = t.hi;
    }
    loss += (isfinite(bhi) ? (double)bhi + (double)blo : (double)bhi) * 0x1p80;
  }
  // one atomic into the warp's slot, so that warps never wait for each other
  if ((threadIdx.x & 31) == 0 && loss != 0.0) atomicAdd(a.partials + 4 * diff_slot(), loss);
  sum_slots<1>(a, 0, a.loss);
}

// Backward: gradients of the loss of the last forward pass.  Bound by the
// reductions' way through L1 (78 % of its data pipe on the busiest SMs before
// pixels were paired).  64 views of 512 x 512 pixels of an 81,920-face mesh: 400 ->
// 254 us with the gathered data packed, the normals and the light's sums left
// to k_diff_scatter (303 us), neighbouring pixels of a face paired (263; side
// by side alone 272) and the face ids read a step ahead (254); records and
// targets, read once, evict-first here and in k_diff_shade: the step 1184 -> 1179.
// The light's weights in FP64: 288.
__global__ void __launch_bounds__(kThreads) k_diff_grad(const DiffArgs a) {
  const Pixels at = block_pixels(a);
  const DiffView& vw = a.views[at.view];
  // the vertices' gradients, which only k_diff_scatter adds to, start at zero
  for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < 4 * (size_t)a.nv; i += (size_t)gridDim.x * kThreads) {
    a.g_pos[i] = 0.0f;
    if (i < 3 * (size_t)a.nv) a.g_vcol[i] = 0.0f;
  }
  const int px = at.x;
  const size_t down = (size_t)at.rows * (size_t)vw.W;
  size_t gp = (size_t)vw.pix_base + (size_t)at.y * (size_t)vw.W + (size_t)px;
  // the face ids first, a step ahead: most pixels of a view are background, and
  // their records (four times the bytes) are not read
  uint32_t next = px < vw.W && at.y < vw.H ? a.ids[gp] : kNoFace;
  for (int step = 0; step < a.blocks_down; ++step, gp += down) {
    const int py = at.y + step * at.rows;
    bool on = next != kNoFace;
    next = step + 1 < a.blocks_down && px < vw.W && py + at.rows < vw.H ? a.ids[gp + down] : kNoFace;
    if (!__any_sync(0xffffffffu, on)) continue;
    DiffRecord rec{kNoFace, kNoFace, 0.0f, 0.0f};
    if (on) {
      const uint4 rw = __ldcs(reinterpret_cast<const uint4*>(a.rec) + gp);
      rec = DiffRecord{rw.x, rw.y, __uint_as_float(rw.z), __uint_as_float(rw.w)};
    }
    const int f = (int)(rec.face - vw.face_base);
    float gc[3][7];  // the corners' sums: colour, position, light weight
    if (rec.face != kNoFace) {
      const Word8 face = ldg8(a.faces + 4 * (size_t)f);
      FaceGeom g;
      face_geom(a, at.view, face, px, py, g);
      Shade s;
      const int ni[3] = {(int)face.x[3], (int)face.x[4], (int)face.x[5]};
      shade(a, g, rec.l0, rec.l1, rec.texel, ni, s);
      const float4 tg = __ldcs(reinterpret_cast<const float4*>(a.target) + gp);  // read once, like the records
      const float go[4] = {2.0f * (s.out.x - tg.x), 2.0f * (s.out.y - tg.y), 2.0f * (s.out.z - tg.z),
                           2.0f * (s.out.w - tg.w)};
      const float t3[3] = {s.t.x, s.t.y, s.t.z};
      // texels
      if (rec.texel != kNoFace)
        atomicAdd(reinterpret_cast<float4*>(a.g_tex) + rec.texel,
                  make_float4(go[0] * s.I * s.col[0], go[1] * s.I * s.col[1], go[2] * s.I * s.col[2], go[3]));
      // vertex colours, and d loss / d intensity
      float dI = 0.0f;
#pragma unroll
      for (int ch = 0; ch < 3; ++ch) dI += go[ch] * s.col[ch] * t3[ch];
      // positions through the barycentrics: G_k = d loss / d l_k
      float G[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        float gk = dI * s.Ii[k];
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) gk += go[ch] * s.I * t3[ch] * s.c[k][ch];
        G[k] = gk;
      }
      // l_k = m_k / M, m_k = max(s D_k, 0): d l / d D_j = s [m_j > 0] (G_j - G.l) / M
      const float Gl = G[0] * s.l[0] + G[1] * s.l[1] + G[2] * s.l[2];
      float dD[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) dD[k] = g.m[k] > 0.0f ? g.sg * (G[k] - Gl) / g.M : 0.0f;
      // D_0 = u1 v2 - u2 v1, D_1 = u2 v0 - u0 v2, D_2 = u0 v1 - u1 v0
      const float gu[3] = {dD[2] * g.v[1] - dD[1] * g.v[2], dD[0] * g.v[2] - dD[2] * g.v[0],
                           dD[1] * g.v[0] - dD[0] * g.v[1]};
      const float gv[3] = {dD[1] * g.u[2] - dD[2] * g.u[1], dD[2] * g.u[0] - dD[0] * g.u[2],
                           dD[0] * g.u[1] - dD[1] * g.u[0]};
      // u_k = (Q_0 - x Q_3) . p_k, v_k = (Q_1 - y Q_3) . p_k
      const float4 A = __ldg(a.col_tab + vw.col_base + px);
      const float4 B = __ldg(a.row_tab + vw.row_base + py);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        gc[k][0] = go[0] * s.I * t3[0] * s.l[k];
        gc[k][1] = go[1] * s.I * t3[1] * s.l[k];
        gc[k][2] = go[2] * s.I * t3[2] * s.l[k];
        gc[k][3] = gu[k] * A.x + gv[k] * B.x;
        gc[k][4] = gu[k] * A.y + gv[k] * B.y;
        gc[k][5] = gu[k] * A.z + gv[k] * B.z;
        gc[k][6] = dI * 0.5f * s.l[k];
      }
    }
    // Colour and position gradients go to the face's corners first
    // (k_diff_scatter adds them to the vertices): a vertex is shared by about
    // six faces, so per-face sums meet far fewer atomics at one address
    // (measured: the backward pass 20 % faster).  Each corner's six sums are a
    // float4 and a float2, the texel's four a float4.  Beside them stands, as a
    // double, the corner's weight in the light's gradient, dI/dL = sum_k l_k 0.5
    // nhat_k, which k_diff_scatter multiplies with its normal: no normal is read
    // here, and from these doubles on the light is summed in FP64 up to its end (in
    // float32 it was 35 us faster at 64 views and its error, 1.3e-8 to 1.1e-7 over seven
    // cases, up to three times as large in one).  The reductions' way out of
    // the SM bounds this kernel, so pixels of one face side by side or one
    // above the other, up to four, are added up first, in float32 like all that
    // is a pixel's own.
    on = rec.face != kNoFace;
#pragma unroll
    for (int o = 1; o <= 8; o <<= 3) {
      const uint32_t other = __shfl_xor_sync(0xffffffffu, on ? rec.face : kNoFace, o);
      const bool same = on && other == rec.face;
      if (!__any_sync(0xffffffffu, same)) continue;
      const bool take = same && !(threadIdx.x & o);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int j = 0; j < 7; ++j) {
          const float x = __shfl_xor_sync(0xffffffffu, gc[k][j], o);
          if (take) gc[k][j] += x;
        }
      }
      if (same && (threadIdx.x & o)) on = false;
    }
    if (on) {
      float4* gf = reinterpret_cast<float4*>(a.g_face + 24 * (size_t)f);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        atomicAdd(gf + 2 * k, make_float4(gc[k][0], gc[k][1], gc[k][2], gc[k][3]));
        atomicAdd(reinterpret_cast<float2*>(gf + 2 * k + 1), make_float2(gc[k][4], gc[k][5]));
        atomicAdd(reinterpret_cast<double*>(gf + 2 * k + 1) + 1, (double)gc[k][6]);
      }
    }
  }
}

// Adds every face's corner sums (k_diff_grad) to its vertices' colour and
// position gradients and, weighted with its normals, to the light's, and
// returns the sums to zero.  One thread per face; position gradients as one
// vector reduction where the caller's buffer is aligned for it.  Bound by
// latency: a face's sums and normals are all read before the first addition
// (no load passes one): 22.1 -> 21.3 us for 81,920 faces, 10.9 -> 10.0 for 1,280.
__global__ void __launch_bounds__(kThreads) k_diff_scatter(const DiffArgs a) {
  griddep_wait();
  const int f = blockIdx.x * kThreads + threadIdx.x;
  double gl[3] = {0.0, 0.0, 0.0};
  if (f < a.nf) {
    float4* gf = reinterpret_cast<float4*>(a.g_face + 24 * (size_t)f);
    const Word8 face = ldg8(a.faces + 4 * (size_t)f);
    const bool vec = !((uintptr_t)a.g_pos & 15u);
    float4 ps[3], qs[3], ns[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      ps[k] = gf[2 * k];
      qs[k] = gf[2 * k + 1];
      ns[k] = ldg4(a.nhat + 4 * (size_t)face.x[3 + k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float4 p = ps[k], q = qs[k], n = ns[k];
      const float x[6] = {p.x, p.y, p.z, p.w, q.x, q.y};
      const int v = (int)face.x[k];
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (x[j] != 0.0f) atomicAdd(a.g_vcol + 3 * (size_t)v + j, x[j]);
      if (x[3] != 0.0f || x[4] != 0.0f || x[5] != 0.0f) {
        if (vec) {
          atomicAdd(reinterpret_cast<float4*>(a.g_pos) + v, make_float4(x[3], x[4], x[5], 0.0f));
        } else {
#pragma unroll
          for (int j = 3; j < 6; ++j) atomicAdd(a.g_pos + 4 * (size_t)v + (j - 3), x[j]);
        }
      }
      const double w = __hiloint2double(__float_as_int(q.w), __float_as_int(q.z));
      if (w != 0.0) {
        gl[0] += w * (double)n.x;
        gl[1] += w * (double)n.y;
        gl[2] += w * (double)n.z;
      }
      if (p.x != 0.0f || p.y != 0.0f || p.z != 0.0f || p.w != 0.0f) gf[2 * k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (q.x != 0.0f || q.y != 0.0f || w != 0.0) gf[2 * k + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int j = 0; j < 3; ++j) gl[j] += __shfl_xor_sync(0xffffffffu, gl[j], o);
  }
  if ((threadIdx.x & 31) == 0) {
    double* p = a.partials + 4 * diff_slot();
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (gl[j] != 0.0) atomicAdd(p + 1 + j, gl[j]);
  }
  sum_slots<3>(a, 1, a.g_light);
}

}  // namespace

// Launches kern behind a kernel on the same stream with programmatic stream
// serialization (it waits in griddep_wait).
template <typename... P, typename... A>
static void launch_after(void (*kern)(P...), dim3 grid, unsigned block, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, args...);
}

int launch_diff_bbox(const float* pos, int nv, DevItem* items, int num_items, uint32_t* partial, unsigned* done,
                     void* stream) {
  if (nv <= 0 || num_items <= 0) return 0;
  const int blocks = std::min(kBBoxBlocks, (nv + 1023) / 1024);
  launch_after(k_diff_bbox, dim3((unsigned)blocks), 1024, (cudaStream_t)stream, pos, nv, items, num_items, partial, done);
  return (int)cudaGetLastError();
}

int launch_diff_normals(const float* world, const float* vnrm, int nn, float* nhat, void* stream) {
  if (nn <= 0) return 0;
  k_diff_normals<<<(nn + kThreads - 1) / kThreads, kThreads, 0, (cudaStream_t)stream>>>(world, vnrm, nn, nhat);
  return (int)cudaGetLastError();
}

int launch_diff_faces(const int* vidx, const int* nidx, const float* uv, int nf, int4* faces, int* apart,
                      void* stream) {
  if (nf <= 0) return 0;
  k_diff_faces<<<(nf + kThreads - 1) / kThreads, kThreads, 0, (cudaStream_t)stream>>>(vidx, nidx, uv, nf, faces, apart);
  return (int)cudaGetLastError();
}

int launch_diff_forward(const DiffArgs& a, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const int sides = (a.max_side + kThreads - 1) / kThreads;
  k_diff_prepare<<<dim3((unsigned)(a.vert_blocks + a.norm_blocks + sides), (unsigned)a.num_views), kThreads, 0, s>>>(a);
  launch_after(k_diff_shade, dim3(a.blocks), kThreads, s, a);
  return (int)cudaGetLastError();
}

int launch_diff_backward(const DiffArgs& a, void* stream) {
  k_diff_grad<<<a.blocks, kThreads, 0, (cudaStream_t)stream>>>(a);
  launch_after(k_diff_scatter, dim3((unsigned)((a.nf + kThreads - 1) / kThreads)), kThreads, (cudaStream_t)stream, a);
  return (int)cudaGetLastError();
}

}  // namespace gr
