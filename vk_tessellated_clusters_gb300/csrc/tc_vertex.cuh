// tc_vertex.cuh — displaced vertex of a part triangle in per-part affine form.
//
// The reference (triangle_tess_template_instantiate.comp.glsl:343-371) maps
// each table vertex w of the config through the part's sub-triangle corners
// bb_k into base-triangle barycentrics, interpolates position, normalised
// normal and uv with them, samples the displacement map and displaces along
// the renormalised normal. Both interpolations are linear, so for a table
// vertex w = (1 - a - b, a, b) every attribute is
//
//     A(w) = A_0 + a (A_1 - A_0) + b (A_2 - A_0),   A_k = sum_j C_k[j] attr_j
//
// with C_k the sub-triangle corners (a flipped config swaps C_0 and C_1, the
// same as swapping w.x and w.y). A_k are evaluated once per part; a vertex then
// costs three fused multiply-adds per component. The result equals the
// reference's two-level evaluation up to rounding (a few ulps of the
// coordinates), inside the |dp| <= 1e-5 x bounding-box-diagonal tolerance the
// positions are held to; integer outputs are unaffected.
//
// Bilinear displacement: mip 0, REPEAT, texel centres at (i + 0.5) / size,
// fp32 weights, texels through read-only loads (one path for fp32, fp16 and
// unorm16 maps).
#pragma once

#include "tc_device.cuh"

namespace tc {

// Nine 16-byte words read with vector loads from shared memory; the 144-byte
// stride puts consecutive records of an array in different bank groups.
struct __align__(16) PartAffine
{
  float4 q[9];
  // q[0] = P0.xyz, E1.x       P0 = position at corner 0, E1 = P1 - P0, E2 = P2 - P0
  // q[1] = E1.yz, E2.xy
  // q[2] = E2.z, N0.xyz       N = interpolated normalised base normals
  // q[3] = F1.xyz, F2.x       F1 = N1 - N0, F2 = N2 - N0
  // q[4] = F2.yz, T0.xy       T = uv
  // q[5] = G1.xy, G2.xy       G1 = T1 - T0, G2 = T2 - T0
  // q[6] = scale, offset, firstVertex (bits), kind (bits; see affine_kind)
  // q[7] = texels lo, texels hi, width, height (bits; width 0 = no displacement)
  // q[8] = width, height (as floats), width - 1, height - 1 (bits; the wrap
  //        masks of power-of-two sizes)
};

// Record kinds (q[6].w): what the vertex needs beyond the interpolated position.
enum : u32
{
  kAffineFlat     = 0,  // no displacement map
  kAffineZeroMap  = 1,  // map of height 0: displaced by the offsets only
  kAffineTextured = 2,  // 2 + 2 * format + (1 if both sizes are powers of two)
  kAffineLarge    = 8,  // 8 + format: 2^32 texels and more (no walk is specialised for these)
};

__host__ __device__ constexpr u32 affine_kind(u32 format, bool pow2) { return kAffineTextured + 2 * format + (pow2 ? 1 : 0); }

// A displacement map as the vertex code reads it: q7 = texels lo, texels hi,
// width, height (bits); q8 = width, height (floats), width - 1, height - 1
// (bits; the wrap masks of power-of-two sizes); kind = affine_kind(format, pow2)
// or kAffineLarge + format, kAffineFlat without a map, kAffineZeroMap for a map
// of height 0.
struct MapDesc
{
  float4 q7, q8;
  u32    kind;
};

__device__ __forceinline__ MapDesc make_map_desc(const tc_DisplacementTexture& tx)
{
  MapDesc   m;
  const u32 w = tx.width, h = tx.height;
  m.q7 = w ? make_float4(__uint_as_float((u32)tx.texels), __uint_as_float((u32)(tx.texels >> 32)), __uint_as_float(w),
                         __uint_as_float(h))
           : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  m.q8 = make_float4(__uint2float_rn(w), __uint2float_rn(h), __uint_as_float(w - 1), __uint_as_float(h - 1));
  const bool pow2 = w != 0 && h != 0 && (w & (w - 1)) == 0 && (h & (h - 1)) == 0;
  // formats other than fp16 / unorm16 read as fp32, as in every other sampling path
  const u32 fmt = tx.format == TC_TEXEL_F16 || tx.format == TC_TEXEL_UNORM16 ? tx.format : TC_TEXEL_F32;
  const u32 textured = __umulhi(w, h) ? kAffineLarge + fmt : affine_kind(fmt, pow2);
  m.kind             = w == 0 ? kAffineFlat : (h == 0 ? kAffineZeroMap : textured);
  return m;
}

__device__ __forceinline__ f3 fma3(float s, f3 a, f3 b)
{
  return {__fmaf_rn(s, a.x, b.x), __fmaf_rn(s, a.y, b.y), __fmaf_rn(s, a.z, b.z)};
}

// sum_j c[j] v_j
__device__ __forceinline__ f3 bary3(f3 c, f3 v0, f3 v1, f3 v2) { return fma3(c.z, v2, fma3(c.y, v1, {c.x * v0.x, c.x * v0.y, c.x * v0.z})); }
__device__ __forceinline__ f2 bary2(f3 c, f2 v0, f2 v1, f2 v2)
{
  return {__fmaf_rn(c.z, v2.x, __fmaf_rn(c.y, v1.x, c.x * v0.x)), __fmaf_rn(c.z, v2.y, __fmaf_rn(c.y, v1.y, c.x * v0.y))};
}

// normalize(v) as v * rsqrt(dot(v, v)) (hardware reciprocal square root)
__device__ __forceinline__ f3 normalize_fast(f3 v)
{
  const float k = rsqrtf(__fmaf_rn(v.z, v.z, __fmaf_rn(v.y, v.y, v.x * v.x)));
  return {v.x * k, v.y * k, v.z * k};
}

// Per-part set-up, written straight into `r` (normally shared memory) word by
// word. `corner` are the sub-triangle's encoded corners
// (TessTriangleInfo.vtxEncoded), p / n / uv the base triangle's positions,
// normals (normalised here, triangle_tess_template_instantiate.comp.glsl:329)
// and uvs; `scale` / `offset` the combined displacement scale (instance x
// view) and offset (instance + view).
__device__ __forceinline__ void write_part_affine(PartAffine& r, const u32 corner[3], bool flipped, const f3 p[3],
                                                  const f3 n[3], const f2 uv[3], u32 firstVertex,
                                                  const tc_DisplacementTexture& tx, float scale, float offset)
{
  f3 c0 = decode_bary(corner[0]), c1 = decode_bary(corner[1]), c2 = decode_bary(corner[2]);
  if(flipped)
  {
    const f3 t = c0;
    c0         = c1;
    c1         = t;
  }
  const u32     w = tx.width;
  const MapDesc m = make_map_desc(tx);
  r.q[6]          = make_float4(scale, offset, __uint_as_float(firstVertex), __uint_as_float(m.kind));
  r.q[7]          = m.q7;
  r.q[8]          = m.q8;
  {
    const f3 P0 = bary3(c0, p[0], p[1], p[2]);
    const f3 E1 = sub3(bary3(c1, p[0], p[1], p[2]), P0);
    r.q[0]      = make_float4(P0.x, P0.y, P0.z, E1.x);
    const f3 E2 = sub3(bary3(c2, p[0], p[1], p[2]), P0);
    r.q[1]      = make_float4(E1.y, E1.z, E2.x, E2.y);
    r.q[2].x    = E2.z;
  }
  if(w == 0)
    return;
  const f3 nh[3] = {normalize_fast(n[0]), normalize_fast(n[1]), normalize_fast(n[2])};
  const f3 N0    = bary3(c0, nh[0], nh[1], nh[2]);
  r.q[2]      = make_float4(r.q[2].x, N0.x, N0.y, N0.z);
  const f3 F1 = sub3(bary3(c1, nh[0], nh[1], nh[2]), N0);
  const f3 F2 = sub3(bary3(c2, nh[0], nh[1], nh[2]), N0);
  r.q[3]      = make_float4(F1.x, F1.y, F1.z, F2.x);
  const f2 T0 = bary2(c0, uv[0], uv[1], uv[2]), T1 = bary2(c1, uv[0], uv[1], uv[2]), T2 = bary2(c2, uv[0], uv[1], uv[2]);
  r.q[4]      = make_float4(F2.y, F2.z, T0.x, T0.y);
  r.q[5]      = make_float4(T1.x - T0.x, T1.y - T0.y, T2.x - T0.x, T2.y - T0.y);
}

// Encoded unit barycentrics: (1,0,0) -> 0, (0,1,0) -> 1, (0,0,1) -> 2, anything else -> 3.
__device__ __forceinline__ u32 unit_corner(u32 e)
{
  return e == 0u ? 0u : (e == TC_TESSTABLE_COORD_MAX ? 1u : (e == (TC_TESSTABLE_COORD_MAX << 16) ? 2u : 3u));
}

// Every part classify writes is a whole base triangle: its three corners are
// the base triangle's own corners, in the order get_config rotated them. Then
// each corner's composed attribute (the barycentric composition of
// write_part_affine) is exactly one base vertex's attribute, so the affine
// form is the base attributes themselves, taken in corner order. Returns true
// for such a part, with order[k] = the base vertex of corner k (a flipped
// config swaps corners 0 and 1); otherwise order = {0, 1, 2}.
__device__ __forceinline__ bool whole_triangle_order(const u32 corner[3], bool flipped, u32 order[3])
{
  u32        m0 = unit_corner(corner[0]), m1 = unit_corner(corner[1]), m2 = unit_corner(corner[2]);
  const bool whole = max(m0, max(m1, m2)) < 3u && m0 != m1 && m1 != m2 && m0 != m2;
  if(!whole)
    m0 = 0, m1 = 1, m2 = 2;
  else if(flipped)
  {
    const u32 t = m0;
    m0          = m1;
    m1          = t;
  }
  order[0] = m0, order[1] = m1, order[2] = m2;
  return whole;
}

// write_part_affine for a whole-triangle part whose base attributes p / n /
// uv are given in corner order: no compositions (the same values up to the
// sign of exact zeros).
__device__ __forceinline__ void write_part_affine_whole(PartAffine& r, const f3 p[3], const f3 n[3], const f2 uv[3],
                                                        u32 firstVertex, const tc_DisplacementTexture& tx, float scale,
                                                        float offset)
{
  const u32     w = tx.width;
  const MapDesc m = make_map_desc(tx);
  r.q[6]          = make_float4(scale, offset, __uint_as_float(firstVertex), __uint_as_float(m.kind));
  r.q[7]          = m.q7;
  r.q[8]          = m.q8;
  const f3 E1     = sub3(p[1], p[0]), E2 = sub3(p[2], p[0]);
  r.q[0]          = make_float4(p[0].x, p[0].y, p[0].z, E1.x);
  r.q[1]          = make_float4(E1.y, E1.z, E2.x, E2.y);
  r.q[2].x        = E2.z;
  if(w == 0)
    return;
  const f3 N0 = normalize_fast(n[0]), N1 = normalize_fast(n[1]), N2 = normalize_fast(n[2]);
  const f3 F1 = sub3(N1, N0), F2 = sub3(N2, N0);
  r.q[2]      = make_float4(E2.z, N0.x, N0.y, N0.z);
  r.q[3]      = make_float4(F1.x, F1.y, F1.z, F2.x);
  r.q[4]      = make_float4(F2.y, F2.z, uv[0].x, uv[0].y);
  r.q[5]      = make_float4(uv[1].x - uv[0].x, uv[1].y - uv[0].y, uv[2].x - uv[0].x, uv[2].y - uv[0].y);
}

// The affine form of part triangle `pt` (cluster / instance resolved by the
// caller): base attributes loaded in corner order for a whole-triangle part,
// else in base order and composed with the corners.
__device__ __forceinline__ void part_affine(PartAffine& r, const u32 corner[3], bool flipped, const float* pos,
                                            const float* nrm, const float* uvs, u32 firstLocalVertex,
                                            const uint8_t* triIndices, u32 firstVertex, const tc_DisplacementTexture& tx,
                                            float scale, float offset)
{
  u32        order[3];
  const bool whole = whole_triangle_order(corner, flipped, order);
  f3         bp[3], bn[3];
  f2         bt[3];
#pragma unroll
  for(int v = 0; v < 3; v++)
  {
    const u32 vi = firstLocalVertex + triIndices[order[v]];
    bp[v]        = ldg3(pos, vi);
    bn[v]        = ldg3(nrm, vi);  // normalised in write_part_affine* (triangle_tess_template_instantiate.comp.glsl:329)
    bt[v]        = ldg2(uvs, vi);
  }
  if(whole)
    write_part_affine_whole(r, bp, bn, bt, firstVertex, tx, scale, offset);
  else
    write_part_affine(r, corner, flipped, bp, bn, bt, firstVertex, tx, scale, offset);
}

template <u32 Format>
__device__ __forceinline__ float texel_at(u64 texels, u64 i)
{
  if(Format == TC_TEXEL_F16)
    return __half2float(__ushort_as_half(__ldg(reinterpret_cast<const unsigned short*>(texels) + i)));
  if(Format == TC_TEXEL_F32)
    return __ldg(reinterpret_cast<const float*>(texels) + i);
  return __uint2float_rn(__ldg(reinterpret_cast<const unsigned short*>(texels) + i)) * (1.0f / 65535.0f);
}

// bilinear sample at (u, v) of the map described by q7 and q8 (Index: of its texels)
template <u32 Format, bool Pow2, class Index = u32>
__device__ __forceinline__ float affine_sample(float4 q7, float4 q8, float u, float v)
{
  const u32   w = __float_as_uint(q7.z), h = __float_as_uint(q7.w);
  const float x = __fmaf_rn(u, q8.x, -0.5f), y = __fmaf_rn(v, q8.y, -0.5f);
  const float xf = floorf(x), yf = floorf(y);
  const float fx = x - xf, fy = y - yf;
  const int   ix = __float2int_rz(xf), iy = __float2int_rz(yf);
  int         x0, x1, y0, y1;
  if(Pow2)
  {
    const int mx = (int)__float_as_uint(q8.z), my = (int)__float_as_uint(q8.w);
    x0 = ix & mx, x1 = (ix + 1) & mx, y0 = iy & my, y1 = (iy + 1) & my;
  }
  else
  {
    x0 = wrapi(ix, (int)w), x1 = wrapi(ix + 1, (int)w), y0 = wrapi(iy, (int)h), y1 = wrapi(iy + 1, (int)h);
  }
  const u64   texels = (u64)__float_as_uint(q7.x) | ((u64)__float_as_uint(q7.y) << 32);
  const Index r0 = (Index)(u32)y0 * w, r1 = (Index)(u32)y1 * w;
  const float t00 = texel_at<Format>(texels, r0 + (u32)x0), t10 = texel_at<Format>(texels, r0 + (u32)x1);
  const float t01 = texel_at<Format>(texels, r1 + (u32)x0), t11 = texel_at<Format>(texels, r1 + (u32)x1);
  const float top = __fmaf_rn(fx, t10 - t00, t00), bot = __fmaf_rn(fx, t11 - t01, t01);
  return __fmaf_rn(fy, bot - top, top);
}

__device__ __forceinline__ u32 affine_kind_of(const PartAffine& r) { return __float_as_uint(r.q[6].w); }

// bilinear sample of a textured kind (0 for kAffineZeroMap)
__device__ __forceinline__ float sample_kind(u32 kind, float4 q7, float4 q8, float u, float v)
{
  switch(kind)
  {
    case affine_kind(TC_TEXEL_F32, true): return affine_sample<TC_TEXEL_F32, true>(q7, q8, u, v);
    case affine_kind(TC_TEXEL_F32, false): return affine_sample<TC_TEXEL_F32, false>(q7, q8, u, v);
    case affine_kind(TC_TEXEL_F16, true): return affine_sample<TC_TEXEL_F16, true>(q7, q8, u, v);
    case affine_kind(TC_TEXEL_F16, false): return affine_sample<TC_TEXEL_F16, false>(q7, q8, u, v);
    case affine_kind(TC_TEXEL_UNORM16, true): return affine_sample<TC_TEXEL_UNORM16, true>(q7, q8, u, v);
    case affine_kind(TC_TEXEL_UNORM16, false): return affine_sample<TC_TEXEL_UNORM16, false>(q7, q8, u, v);
    case kAffineLarge + TC_TEXEL_F32: return affine_sample<TC_TEXEL_F32, false, u64>(q7, q8, u, v);
    case kAffineLarge + TC_TEXEL_F16: return affine_sample<TC_TEXEL_F16, false, u64>(q7, q8, u, v);
    case kAffineLarge + TC_TEXEL_UNORM16: return affine_sample<TC_TEXEL_UNORM16, false, u64>(q7, q8, u, v);
    default: return 0.0f;
  }
}

// Displaced vertex of a full cluster (cluster_classify.comp.glsl:457-482):
// p + normalize(n) * (bilinear(uv) * scale + offset), sampled and
// renormalised like the part vertices (Kind ~0u: resolved at run time).
template <u32 Kind>
__device__ __forceinline__ f3 full_vertex_k(f3 p, f3 n, f2 uv, const MapDesc& m, float scale, float offset)
{
  const u32 kind = Kind == ~0u ? m.kind : Kind;
  if(kind == kAffineFlat)
    return p;
  const float hraw   = sample_kind(kind, m.q7, m.q8, uv.x, uv.y);
  const float height = __fmaf_rn(hraw, scale, offset);
  const float k      = height * rsqrtf(__fmaf_rn(n.z, n.z, __fmaf_rn(n.y, n.y, n.x * n.x)));
  return fma3(k, n, p);
}

// Vertex `tableVertex` (an encoded table barycentric) of the part in `r`, for
// a record of kind Kind (~0u: any kind, resolved at run time).
template <u32 Kind>
__device__ __forceinline__ f3 affine_vertex_k(const PartAffine& r, u32 tableVertex)
{
  const float  a  = __uint2float_rn(tableVertex & 0xFFFFu) * (1.0f / 32768.0f);
  const float  b  = __uint2float_rn(tableVertex >> 16) * (1.0f / 32768.0f);
  const float4 q0 = r.q[0], q1 = r.q[1], q2 = r.q[2];
  f3           P  = {__fmaf_rn(b, q1.z, __fmaf_rn(a, q0.w, q0.x)), __fmaf_rn(b, q1.w, __fmaf_rn(a, q1.x, q0.y)),
                     __fmaf_rn(b, q2.x, __fmaf_rn(a, q1.y, q0.z))};
  const u32    kind = Kind == ~0u ? affine_kind_of(r) : Kind;
  if(kind == kAffineFlat)
    return P;
  const float4 q3 = r.q[3], q4 = r.q[4], q5 = r.q[5], q6 = r.q[6];
  const f3     N  = {__fmaf_rn(b, q3.w, __fmaf_rn(a, q3.x, q2.y)), __fmaf_rn(b, q4.x, __fmaf_rn(a, q3.y, q2.z)),
                     __fmaf_rn(b, q4.y, __fmaf_rn(a, q3.z, q2.w))};
  const float  u  = __fmaf_rn(b, q5.z, __fmaf_rn(a, q5.x, q4.z));
  const float  v  = __fmaf_rn(b, q5.w, __fmaf_rn(a, q5.y, q4.w));
  const float hraw = sample_kind(kind, r.q[7], r.q[8], u, v);
  // displace along the renormalised interpolated normal
  const float height = __fmaf_rn(hraw, q6.x, q6.y);
  const float k      = height * rsqrtf(__fmaf_rn(N.z, N.z, __fmaf_rn(N.y, N.y, N.x * N.x)));
  return fma3(k, N, P);
}

// affine_vertex_k for a record whose map, scale and offset (the same for
// every part of a chunk) are passed in registers: only q0-q5 are read from `r`.
// Same operations, so the same bits.
template <u32 Kind>
__device__ __forceinline__ f3 affine_vertex_u(const PartAffine& r, u32 tableVertex, const MapDesc& m, float scale,
                                              float offset)
{
  const float  a  = __uint2float_rn(tableVertex & 0xFFFFu) * (1.0f / 32768.0f);
  const float  b  = __uint2float_rn(tableVertex >> 16) * (1.0f / 32768.0f);
  const float4 q0 = r.q[0], q1 = r.q[1], q2 = r.q[2];
  f3           P  = {__fmaf_rn(b, q1.z, __fmaf_rn(a, q0.w, q0.x)), __fmaf_rn(b, q1.w, __fmaf_rn(a, q1.x, q0.y)),
                     __fmaf_rn(b, q2.x, __fmaf_rn(a, q1.y, q0.z))};
  const u32    kind = Kind == ~0u ? m.kind : Kind;
  if(kind == kAffineFlat)
    return P;
  const float4 q3 = r.q[3], q4 = r.q[4], q5 = r.q[5];
  const f3     N  = {__fmaf_rn(b, q3.w, __fmaf_rn(a, q3.x, q2.y)), __fmaf_rn(b, q4.x, __fmaf_rn(a, q3.y, q2.z)),
                     __fmaf_rn(b, q4.y, __fmaf_rn(a, q3.z, q2.w))};
  const float  u  = __fmaf_rn(b, q5.z, __fmaf_rn(a, q5.x, q4.z));
  const float  v  = __fmaf_rn(b, q5.w, __fmaf_rn(a, q5.y, q4.w));
  const float hraw   = sample_kind(kind, m.q7, m.q8, u, v);
  const float height = __fmaf_rn(hraw, scale, offset);
  const float k      = height * rsqrtf(__fmaf_rn(N.z, N.z, __fmaf_rn(N.y, N.y, N.x * N.x)));
  return fma3(k, N, P);
}

}  // namespace tc

namespace tc {

// ---------------------------------------------------------------------------
// The ripple deformation (displacement.glsl), written like the CPU
// restatement: separate IEEE multiplies, adds and divisions in the shader's
// order.
// ---------------------------------------------------------------------------

// the FrameConstants terms of displacement.glsl:106-120
struct RippleParams
{
  float frequency;  // animationRippleFrequency
  float phase;      // animationState * animationRippleSpeed
  float amplitude;  // animationRippleAmplitude
  u32   enabled;
};

__device__ __forceinline__ RippleParams ripple_params(const tc_FrameConstants& view, bool enabled)
{
  return {view.animationRippleFrequency, view.animationState * view.animationRippleSpeed,
          view.animationRippleAmplitude, enabled ? 1u : 0u};
}

// displacement.glsl:106-120 rippleDeform(vertex, instance id, geometry size)
__device__ __forceinline__ f3 ripple(f3 p, u32 seed, float size, const RippleParams& rp)
{
  const float maxCoord  = fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z)));
  const float frequency = __fdiv_rn(rp.frequency, size);
  const float s         = __uint2float_rn(seed);
  const f3    wave      = {sinf((maxCoord * frequency + s) + rp.phase), cosf((maxCoord * frequency * 3.0f + s) + rp.phase),
                           sinf((maxCoord * frequency * 1.2f + s) + rp.phase)};
  const f3    dir       = normalize3({p.z, p.y, p.x});
  const float amp       = rp.amplitude * size;
  return {p.x + dir.x * (amp * wave.x), p.y + dir.y * (amp * wave.y), p.z + dir.z * (amp * wave.z)};
}

// ---------------------------------------------------------------------------
// The PN-triangle cubic of a part in per-part form (TC_FLAG_PN): the base
// triangle's control points with the cubic's binomial factors multiplied in,
// and the base barycentrics of a table vertex w = (1 - a - b, a, b) as
// W0 + a W1 + b W2 (the composition with the sub-triangle's corners, exact up
// to one rounding per term: the corners are multiples of 2^-15). A vertex
// takes ten weights shared by x, y and z and three fused multiply-adds for
// each control point (displacement.glsl:80-104 deform_getPN). The control
// points (displacement.glsl:47-78 deform_setupPN) take the thirds of an edge
// as fused products with 1/3 and 2/3: one rounding where the shader's
// division and addition have two, without 21 divisions per part.
// ---------------------------------------------------------------------------

// a + (b - a) t, moved along n into the plane of `plane` and n
__device__ __forceinline__ f3 pn_edge_point(f3 a, f3 edge, float t, f3 plane, f3 n)
{
  const f3    p = fma3(t, edge, a);
  const f3    d = sub3(p, plane);
  const float k = __fmaf_rn(d.z, n.z, __fmaf_rn(d.y, n.y, d.x * n.x));
  return fma3(-k, n, p);
}

// 176-byte stride: records of an array start in different bank groups.
struct __align__(16) PartPn
{
  float4 q[11];
  // q[0]..q[7].y: b300, b030, b003, 3 b210, 3 b120, 3 b201, 3 b021, 3 b102, 3 b012, 6 b111 (xyz each)
  // q[7].zw, q[8].x: W0; q[8].yzw: W1; q[9].xyz: W2
};

// v, n: the base triangle's positions and normalised normals
__device__ __forceinline__ void write_part_pn(PartPn& r, const u32 corner[3], bool flipped, const f3 v[3], const f3 n[3])
{
  f3 c0 = decode_bary(corner[0]), c1 = decode_bary(corner[1]), c2 = decode_bary(corner[2]);
  if(flipped)
  {
    const f3 t = c0;
    c0         = c1;
    c1         = t;
  }
  const f3        w1 = sub3(c1, c0), w2 = sub3(c2, c0);
  constexpr float kThird = 1.0f / 3.0f, kTwoThirds = 2.0f / 3.0f;
  // b030 = v0, b003 = v1, b300 = v2
  const f3 e300 = sub3(v[1], v[0]), e030 = sub3(v[2], v[1]), e003 = sub3(v[0], v[2]);
  const f3 b021 = pn_edge_point(v[0], e300, kThird, v[0], n[0]), b012 = pn_edge_point(v[0], e300, kTwoThirds, v[1], n[1]);
  const f3 b102 = pn_edge_point(v[1], e030, kThird, v[1], n[1]), b201 = pn_edge_point(v[1], e030, kTwoThirds, v[2], n[2]);
  const f3 b210 = pn_edge_point(v[2], e003, kThird, v[2], n[2]), b120 = pn_edge_point(v[2], e003, kTwoThirds, v[0], n[0]);
  // 6 b111 = 6 (E + (E - V) / 2), E = the six points' mean, V = the corners' = 1.5 (6 E) - 3 V
  const f3 six  = {((((b021.x + b012.x) + b102.x) + b201.x) + b210.x) + b120.x,
                   ((((b021.y + b012.y) + b102.y) + b201.y) + b210.y) + b120.y,
                   ((((b021.z + b012.z) + b102.z) + b201.z) + b210.z) + b120.z};
  const f3 b111 = fma3(1.5f, six, {-((v[1].x + v[0].x) + v[2].x), -((v[1].y + v[0].y) + v[2].y), -((v[1].z + v[0].z) + v[2].z)});
  r.q[0] = make_float4(v[2].x, v[2].y, v[2].z, v[0].x);
  r.q[1] = make_float4(v[0].y, v[0].z, v[1].x, v[1].y);
  r.q[2] = make_float4(v[1].z, 3.0f * b210.x, 3.0f * b210.y, 3.0f * b210.z);
  r.q[3] = make_float4(3.0f * b120.x, 3.0f * b120.y, 3.0f * b120.z, 3.0f * b201.x);
  r.q[4] = make_float4(3.0f * b201.y, 3.0f * b201.z, 3.0f * b021.x, 3.0f * b021.y);
  r.q[5] = make_float4(3.0f * b021.z, 3.0f * b102.x, 3.0f * b102.y, 3.0f * b102.z);
  r.q[6] = make_float4(3.0f * b012.x, 3.0f * b012.y, 3.0f * b012.z, b111.x);
  r.q[7] = make_float4(b111.y, b111.z, c0.x, c0.y);
  r.q[8] = make_float4(c0.z, w1.x, w1.y, w1.z);
  r.q[9] = make_float4(w2.x, w2.y, w2.z, 0.0f);
}

// Position on the cubic at table vertex `tableVertex` (displacement.glsl:80-104)
__device__ __forceinline__ f3 part_pn_position(const PartPn& r, u32 tableVertex)
{
  const float  a  = __uint2float_rn(tableVertex & 0xFFFFu) * (1.0f / 32768.0f);
  const float  b  = __uint2float_rn(tableVertex >> 16) * (1.0f / 32768.0f);
  const float4 q7 = r.q[7], q8 = r.q[8], q9 = r.q[9];
  const float  u = __fmaf_rn(b, q9.x, __fmaf_rn(a, q8.y, q7.z)), v = __fmaf_rn(b, q9.y, __fmaf_rn(a, q8.z, q7.w)),
               w = __fmaf_rn(b, q9.z, __fmaf_rn(a, q8.w, q8.x));
  const float u2 = u * u, v2 = v * v, w2 = w * w;
  f3          p;
  {
    const float4 q0 = r.q[0], q1 = r.q[1];
    const float  k300 = w2 * w, k030 = u2 * u, k003 = v2 * v;
    const float4 q2 = r.q[2];
    p = {k300 * q0.x, k300 * q0.y, k300 * q0.z};
    p = fma3(k030, {q0.w, q1.x, q1.y}, p);
    p = fma3(k003, {q1.z, q1.w, q2.x}, p);
    p = fma3(w2 * u, {q2.y, q2.z, q2.w}, p);
  }
  {
    const float4 q3 = r.q[3], q4 = r.q[4];
    p = fma3(w * u2, {q3.x, q3.y, q3.z}, p);
    p = fma3(w2 * v, {q3.w, q4.x, q4.y}, p);
    const float4 q5 = r.q[5];
    p = fma3(u2 * v, {q4.z, q4.w, q5.x}, p);
    p = fma3(w * v2, {q5.y, q5.z, q5.w}, p);
  }
  const float4 q6 = r.q[6];
  p = fma3(u * v2, {q6.x, q6.y, q6.z}, p);
  return fma3((w * u) * v, {q6.w, q7.x, q7.y}, p);
}

// Displacement of the part in `r` at table vertex `tableVertex` added to `P`
// (its map, scale and offset from the record; Kind ~0u: of any kind).
template <u32 Kind>
__device__ __forceinline__ f3 affine_displace(const PartAffine& r, u32 tableVertex, f3 P)
{
  const u32 kind = Kind == ~0u ? affine_kind_of(r) : Kind;
  if(kind == kAffineFlat)
    return P;
  const float  a  = __uint2float_rn(tableVertex & 0xFFFFu) * (1.0f / 32768.0f);
  const float  b  = __uint2float_rn(tableVertex >> 16) * (1.0f / 32768.0f);
  const float4 q2 = r.q[2], q3 = r.q[3], q4 = r.q[4], q5 = r.q[5], q6 = r.q[6];
  const f3     N = {__fmaf_rn(b, q3.w, __fmaf_rn(a, q3.x, q2.y)), __fmaf_rn(b, q4.x, __fmaf_rn(a, q3.y, q2.z)),
                    __fmaf_rn(b, q4.y, __fmaf_rn(a, q3.z, q2.w))};
  const float  u      = __fmaf_rn(b, q5.z, __fmaf_rn(a, q5.x, q4.z));
  const float  v      = __fmaf_rn(b, q5.w, __fmaf_rn(a, q5.y, q4.w));
  const float  height = __fmaf_rn(sample_kind(kind, r.q[7], r.q[8], u, v), q6.x, q6.y);
  const float  k      = height * rsqrtf(__fmaf_rn(N.z, N.z, __fmaf_rn(N.y, N.y, N.x * N.x)));
  return fma3(k, N, P);
}

}  // namespace tc
