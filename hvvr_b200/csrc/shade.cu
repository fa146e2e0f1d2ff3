// shade.cu - fused intersect + G-buffer compression + MSAA shade/resolve, and the remap.
//
// intersectShadeKernel<N, FMA> runs one 128-thread CTA per tile (thread = sample), like
// the reference's IntersectKernel and ResolveKernel (libraries/hvvr/raycaster/intersect.cu:298-342,
// libraries/hvvr/raycaster/resolve.cu:324-458), but as one launch: the per-subsample hit
// IDs stay in registers, are grouped into (triangle, coverage mask) pairs exactly as
// EmitGBuffer does (intersect.cu:28-89), and are shaded and resolved in the same thread
// (ShadeMSAA, resolve.cu:161-284). The G-buffer therefore never goes to HBM.
//
// The tile's triangle list is consumed in chunks of 128 entries. The tile's own tests (frustum planes,
// ray-origin half space, corner-ray barycentrics: FrustumPlanes::test, IntersectTriangleTile<false>::setup,
// TestTriangleFrustaUVW; libraries/hvvr/raycaster/prim_tests.h:18-164) decide which triangles its
// samples are tested against, and each sample takes those in list order, so depth ties resolve as in
// the reference. Before and between them, bounds that no rounding can break (edgePlane) pass by what
// a tile, a warp of its samples, or one sample cannot hit: a sample runs its N subsample tests on the
// few triangles that its footprint meets in front of what it has already found, not on its tile's.
#include <algorithm>

#include "../../include/hvvr_c.h"
#include "dev_common.cuh"

namespace hvb {

// unit offsets for rates 1,2,4,8,16,32: rows 0-5 the spiral, rows 6-11 the rotated grid
__constant__ float2 cMsaa[12][32];
// each offset's x and y duplicated into both halves of a 64-bit pair, the operands of the packed
// tests that run one subsample against two triangles
__constant__ __align__(8) float2 cMsaaXX[12][32];
__constant__ __align__(8) float2 cMsaaYY[12][32];

namespace {

constexpr unsigned kFull = 0xffffffffu;

#ifdef HVVR_VISIT_CLOCKS
// Profiling build only (make -C hvvr_b200/csrc visit-clocks): per global tile, the SM cycles that
// thread 0 of its intersect/shade CTA spends in each phase (the CTA's barriers make thread 0's
// clock the CTA's), its chunk count and its list length, read back through hvvr_dbg_shade_clocks.
constexpr uint32_t kShadeClockTiles = 1u << 17;
enum : uint32_t {
    kScSetup, // view, frustum planes, beams, first chunk staged
    kScCull,  // per chunk: staged triangles arrive, per-triangle tile tests, survivor compaction
    kScTest,  // per chunk: depth skip and the packed subsample tests, next chunk staged
    kScShade, // hit and depth outputs, G-buffer grouping, shading, resolve
    kScPhases
};
__device__ unsigned long long gShadeClocks[kShadeClockTiles][kScPhases + 2];
#define SHADE_MARK(phase, dep)                                                                                         \
    do {                                                                                                               \
        const long long t_ = phaseClock(dep);                                                                          \
        scAcc[phase] += t_ - scLast;                                                                                   \
        scLast = t_;                                                                                                   \
    } while (0)
#else
#define SHADE_MARK(phase, dep) do { } while (0)
#endif

template <uint32_t N> struct RateIndex;
template <> struct RateIndex<1> { static constexpr int v = 0; };
template <> struct RateIndex<2> { static constexpr int v = 1; };
template <> struct RateIndex<4> { static constexpr int v = 2; };
template <> struct RateIndex<8> { static constexpr int v = 3; };
template <> struct RateIndex<16> { static constexpr int v = 4; };
template <> struct RateIndex<32> { static constexpr int v = 5; };

// Loads a pointer field of the view table where it is used. The asm is volatile so the
// compiler re-issues the (L1-resident) load instead of keeping ten 64-bit pointers live in
// registers across the tile loop, which costs two CTAs per SM of occupancy.
template <class T>
__device__ __forceinline__ T* viewPtr(T* const& field) {
    uint64_t v;
    asm volatile("ld.global.nc.u64 %0, [%1];" : "=l"(v) : "l"(&field));
    return reinterpret_cast<T*>(v);
}

struct TriGeom {
    F3 v0, e0, e1;
};
__device__ __forceinline__ TriGeom loadTri(const float4* __restrict__ tris, uint32_t i) {
    const float4 a = __ldg(tris + 3 * size_t(i) + 0);
    const float4 b = __ldg(tris + 3 * size_t(i) + 1);
    const float4 c = __ldg(tris + 3 * size_t(i) + 2);
    return TriGeom{f3(a.x, a.y, a.z), f3(a.w, b.x, b.y), f3(b.z, b.w, c.x)};
}

// per-thread scaled barycentric setup (IntersectTriangleThread ctor + GetDifferentials,
// prim_tests.h:118-134, 175-188)
struct TriThread {
    float dc, vc, wc, ddx, ddy, dvx, dvy, dwx, dwy;
};
__device__ __forceinline__ TriThread threadSetupN(F3 normal, F3 e0, F3 e1, F3 v0r, F3 c, F3 du, F3 dv) {
    TriThread r;
    r.dc = dot3(-c, normal);
    const F3 ec = cross3(-c, v0r);
    r.vc = dot3(e1, ec);
    r.wc = -dot3(e0, ec);
    r.ddx = dot3(-du, normal);
    r.ddy = dot3(-dv, normal);
    const F3 cu = cross3(-du, v0r), cv = cross3(-dv, v0r);
    r.dvx = dot3(e1, cu);
    r.dvy = dot3(e1, cv);
    r.dwx = -dot3(e0, cu);
    r.dwy = -dot3(e0, cv);
    return r;
}
// the same with normal = e0 x e1 computed here (the per-triangle part, which the tile loop
// computes once per triangle instead of once per thread)
__device__ __forceinline__ TriThread threadSetup(F3 e0, F3 e1, F3 v0r, F3 c, F3 du, F3 dv) {
    return threadSetupN(cross3(e0, e1), e0, e1, v0r, c, du, dv);
}

// Packed FP32 (sm_100 f32x2): two floats in one 64-bit register pair, each lane an ordinary IEEE
// single-precision operation (round to nearest, flush to zero like every other operation here), so
// a packed result equals the two scalar results bit for bit.
typedef unsigned long long P2;
__device__ __forceinline__ P2 pk(float lo, float hi) {
    P2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void upk(P2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ P2 fma2(P2 a, P2 b, P2 c) {
    P2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// The rounded product a*b of both lanes, written as fma(a, b, z) with z = (-0, -0): x + (-0) = x
// for every x (zeros keep their sign), so this is exactly mul.rn.ftz. The compiler contracts a
// packed mul.rn with the add that consumes it into one FMA, and it does the same to
// fma(a, b, -0) when it can see the -0 (both measured on sm_100a: the uncontracted expressions
// then round differently from their scalar forms). So z comes from constant memory that the host
// writes at run time (cNegZero2, with the offset tables), a value the compiler cannot know: the
// FMA stays a rounded product, and every product and sum below keeps its own rounding.
__constant__ P2 cNegZero2;
__device__ __forceinline__ P2 mul2(P2 a, P2 b) {
    P2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(cNegZero2));
    return r;
}
__device__ __forceinline__ P2 add2(P2 a, P2 b) {
    P2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ P2 sub2(P2 a, P2 b) {
    P2 r;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// exact negation of both lanes (a sign-bit flip, as the scalar unary minus)
__device__ __forceinline__ P2 neg2(P2 a) { return a ^ 0x8000000080000000ull; }

struct V2 {
    P2 x, y, z;
};
// dot3 / cross3 (same association) on two triangles at once
__device__ __forceinline__ P2 dot2(const V2& a, const V2& b) {
    return add2(add2(mul2(a.x, b.x), mul2(a.y, b.y)), mul2(a.z, b.z));
}
__device__ __forceinline__ V2 cross2(const V2& a, const V2& b) {
    return V2{sub2(mul2(a.y, b.z), mul2(a.z, b.y)), sub2(mul2(a.z, b.x), mul2(a.x, b.z)),
              sub2(mul2(a.x, b.y), mul2(a.y, b.x))};
}

// threadSetupN for two triangles j, k (lane 0 / lane 1 of every pair) against this thread's
// sample: nc, ndu, ndv are -c, -du, -dv duplicated into both lanes
struct TriPair {
    P2 dc, vc, wc, ddx, ddy, dvx, dvy, dwx, dwy;
};
__device__ __forceinline__ TriPair pairSetup(const V2& n, const V2& e0, const V2& e1, const V2& v0r, const V2& nc,
                                             const V2& ndu, const V2& ndv) {
    TriPair r;
    r.dc = dot2(nc, n);
    const V2 ec = cross2(nc, v0r);
    r.vc = dot2(e1, ec);
    r.wc = neg2(dot2(e0, ec));
    r.ddx = dot2(ndu, n);
    r.ddy = dot2(ndv, n);
    const V2 cu = cross2(ndu, v0r), cv = cross2(ndv, v0r);
    r.dvx = dot2(e1, cu);
    r.dvy = dot2(e1, cv);
    r.dwx = neg2(dot2(e0, cu));
    r.dwy = neg2(dot2(e0, cv));
    return r;
}

__device__ __forceinline__ bool signsClear(float a, float b, float c, float d) {
    return (__float_as_int(a) | __float_as_int(b) | __float_as_int(c) | __float_as_int(d)) >= 0;
}

// The depth of a hit, t / denom as the reference computes it (t times the IEEE reciprocal). Out of
// line: it runs only on a hit, and one copy of the division replaces one per unrolled subsample
// test, which keeps the pair-test loop small in the instruction cache.
__device__ __noinline__ float hitDepth(float t, float denom) { return t * (1.0f / denom); }

// IntersectTriangleThread::test (prim_tests.h:192-231) of one subsample (unit offset ax, ay
// duplicated into both lanes) against triangles j and k in that order, with the scalar test's
// operations in its order: denom, depthDelta, v, w as FMA chains (FMA) or as rounded products and
// sums (STRICT), u = (denom - v) - w, the sign-bit test and the depth update. Both depth deltas are
// formed from the depth before j; when j hits, k's is formed again from the new depth, so k sees
// exactly the depth the sequential fold gives it.
// tt holds (-t_j, -t_k) in FMA mode, (t_j, t_k) in STRICT mode.
template <bool FMA>
__device__ __forceinline__ void pairTest(const TriPair& p, P2 tt, float tj, float tk, uint32_t ij, uint32_t ik,
                                         P2 ax, P2 ay, float& depth, uint32_t& hit) {
    const P2 d2 = pk(depth, depth);
    P2 denom, dd, v, w;
    if (FMA) {
        denom = fma2(p.ddy, ay, fma2(p.ddx, ax, p.dc));
        dd = fma2(d2, denom, tt);
        v = fma2(p.dvy, ay, fma2(p.dvx, ax, p.vc));
        w = fma2(p.dwy, ay, fma2(p.dwx, ax, p.wc));
    } else {
        denom = add2(add2(p.dc, mul2(p.ddx, ax)), mul2(p.ddy, ay));
        dd = sub2(mul2(d2, denom), tt);
        v = add2(add2(p.vc, mul2(p.dvx, ax)), mul2(p.dvy, ay));
        w = add2(add2(p.wc, mul2(p.dwx, ax)), mul2(p.dwy, ay));
    }
    const P2 u = sub2(sub2(denom, v), w);
    float den0, den1, dd0, dd1, u0, u1, v0, v1, w0, w1;
    upk(denom, den0, den1);
    upk(dd, dd0, dd1);
    upk(u, u0, u1);
    upk(v, v0, v1);
    upk(w, w0, w1);
    if (signsClear(dd0, u0, v0, w0)) {
        depth = hitDepth(tj, den0);
        hit = ij;
        dd1 = FMA ? fmaf(depth, den1, -tk) : depth * den1 - tk;
    }
    if (signsClear(dd1, u1, v1, w1)) {
        depth = hitDepth(tk, den1);
        hit = ik;
    }
}

// IntersectTriangleThread::calcUVW (prim_tests.h:233-245)
template <bool FMA>
__device__ __forceinline__ F3 calcUVW(const TriThread& th, float ax, float ay) {
    float denom, v, w;
    if (FMA) {
        denom = fmaf(th.ddy, ay, fmaf(th.ddx, ax, th.dc));
        v = fmaf(th.dvy, ay, fmaf(th.dvx, ax, th.vc));
        w = fmaf(th.dwy, ay, fmaf(th.dwx, ax, th.wc));
    } else {
        denom = th.dc + th.ddx * ax + th.ddy * ay;
        v = th.vc + th.dvx * ax + th.dvy * ay;
        w = th.wc + th.dwx * ax + th.dwy * ay;
    }
    const float u = denom - v - w;
    const float inv = 1.0f / denom;
    return f3(u * inv, v * inv, w * inv);
}

// TestRayTriangle<false> barycentrics (prim_tests.h:53-82)
__device__ __forceinline__ void rayTriUVW(F3 ro, F3 rd, const TriGeom& tri, float& u, float& v, float& w) {
    const F3 n = cross3(tri.e0, tri.e1);
    const float denom = dot3(-rd, n);
    const F3 v0r = ro - tri.v0;
    const F3 e = cross3(-rd, v0r);
    v = dot3(tri.e1, e);
    w = -dot3(tri.e0, e);
    const float ood = 1.0f / denom;
    v = v * ood;
    w = w * ood;
    u = 1.0f - v - w;
}

// SimpleMaterial (material.h:15-49): textureIDsAndShadingModel holds the shading model in bits
// 0-15 and the glossiness, specular and diffuse/emissive texture ids in bits 16-31, 32-47, 48-63
constexpr uint32_t kNoTexture = 0xffffu;
struct Material {
    F3 emissive, diffuse, specular;
    float glossiness;
    uint32_t model, texGloss, texSpecular, texDiffuse;
};

__device__ __forceinline__ float pow5(float x) {
    const float x2 = x * x;
    return x2 * x2 * x;
}

// GGX_SchlickFresnel_SchlickSmithGGX + PBR_BRDF1 (libraries/hvvr/raycaster/shading_helpers.h:89-122)
__device__ F3 pbr(F3 L, F3 N, F3 V, F3 base, float roughness, F3 F0, F3 lightColor) {
    const float alpha = roughness * roughness;
    const F3 H = normalize3(L + V);
    const float alpha2 = alpha * alpha;
    const float NdotH = satf(dot3(N, H));
    const float q = (NdotH * NdotH) * (alpha2 - 1.0f) + 1.0f;
    const float D = alpha2 / (3.141592653589f * (q * q));
    const float LdotH = satf(dot3(L, H));
    const F3 F = F0 + (f3(1.0f, 1.0f, 1.0f) - F0) * pow5(1.0f - LdotH);
    const float NdotL = satf(dot3(N, L));
    const float NdotV = satf(dot3(N, V));
    const float k = alpha * 0.5f;
    const float vis = (1.0f / (NdotL * (1.0f - k) + k)) * (1.0f / (NdotV * (1.0f - k) + k));
    const F3 spec = ((F * D) * vis) * (1.0f / 4.0f);
    const float NdotL2 = satf(dot3(N, L));
    const F3 diffuse = ((base * lightColor) * (f3(1.0f, 1.0f, 1.0f) - spec)) * NdotL2;
    return diffuse + lightColor * spec;
}

// the phong branch of GGXShade (libraries/hvvr/raycaster/shading.h:127-160) once the base colour,
// F0 and roughness are known (material constants or texture reads): emissive, ambient and the
// lights, clamped at zero
__device__ F3 ggxLit(F3 emissive, F3 base, F3 F0, float roughness, F3 pos, F3 normal, F3 V, const LightEnvDev& env) {
    F3 radiance = emissive + base * f3(.15f, .15f, .165f);
    if (env.nd > 0) {
        radiance = radiance + pbr(f3(env.dir[0][0], env.dir[0][1], env.dir[0][2]), normal, V, base, roughness, F0,
                                  f3(env.dir[0][3], env.dir[0][4], env.dir[0][5]));
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (i >= env.np) break;
        const float* l = env.pt[i];
        const F3 delta = f3(l[0], l[1], l[2]) - pos;
        const float r = sqrtf(dot3(delta, delta));
        const F3 L = normalize3(delta);
        const float fd = satf((l[3] - r) * l[7]);
        radiance = radiance + pbr(L, normal, V, base, roughness, F0, f3(l[4], l[5], l[6]) * fd);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (i >= env.ns) break;
        const float* l = env.spot[i];
        const F3 delta = f3(l[0], l[1], l[2]) - pos;
        const float r = sqrtf(dot3(delta, delta));
        const F3 L = normalize3(delta);
        const float fd = satf((l[3] - r) * l[7]);
        const F3 lit = pbr(L, normal, V, base, roughness, F0, f3(l[8], l[9], l[10]) * fd);
        const float cosA = dot3(f3(l[4], l[5], l[6]), -L);
        const float fa = satf((cosA - l[11]) * l[12]);
        radiance = radiance + lit * fa;
    }
    return f3(tmaxf(radiance.x, 0.0f), tmaxf(radiance.y, 0.0f), tmaxf(radiance.z, 0.0f));
}

// GGXShade for a material without textures (shading.h:84-161)
__device__ F3 ggxShade(const Material& m, F3 pos, F3 nrm, F3 camPos, const LightEnvDev& env) {
    const F3 normal = normalize3(nrm);
    if (m.model == 2u) return m.emissive;
    const F3 V = normalize3(camPos - pos);
    const float roughness = 1.0f - m.glossiness;
    return ggxLit(m.emissive, m.diffuse, m.specular, roughness, pos, normal, V, env);
}

// true when GGXShade reads a texture for m: the emissive id for the emissive model, else any of
// the diffuse, specular and glossiness ids
__device__ __forceinline__ bool readsTextures(const Material& m) {
    return m.model == 2u ? m.texDiffuse != kNoTexture : (m.texDiffuse & m.texSpecular & m.texGloss) != kNoTexture;
}

// ReadTexture for material texture `id` (shading.h:45-47); false (the material's constant stays)
// for no texture, and for an id that names no live texture of the scene
__device__ __forceinline__ bool materialTexture(const ViewDev& V, uint32_t id, float2 uv, float2 dx, float2 dy,
                                                float4& out) {
    if (id == kNoTexture || id >= V.textureCount) return false;
    const unsigned long long t = __ldg(viewPtr(V.textures) + id);
    if (!t) return false;
    out = readTexture(t, uv.x, uv.y, dx, dy);
    return true;
}

// ACESFilm, linearToSRgb, ToColor4Unorm8SRgb (shading_helpers.h:158-200; libraries/hvvr/shared/util_graphics.h:26-28)
__device__ __forceinline__ float aces(float x) { return satf((x * (2.51f * x + 0.03f)) / (x * (2.43f * x + 0.59f) + 0.14f)); }
__device__ __forceinline__ float toSrgb(float x) {
    return (x <= 0.0031308f) ? (x * 12.92f) : (powf(x, (1.0f / 2.4f)) * 1.055f - .055f);
}
__device__ __forceinline__ uint32_t packColor(F3 c) {
    const uint32_t r = uint32_t(toSrgb(c.x) * 255.0f);
    const uint32_t g = uint32_t(toSrgb(c.y) * 255.0f);
    const uint32_t b = uint32_t(toSrgb(c.z) * 255.0f);
    return r | (g << 8) | (b << 16) | 0xFF000000u;
}

__device__ __forceinline__ F3 halfNormal(float4 a, float4 b) {
    const uint32_t n01 = __float_as_uint(a.w), n23 = __float_as_uint(b.x);
    return f3(__half2float(__ushort_as_half((unsigned short)(n01 & 0xffffu))),
              __half2float(__ushort_as_half((unsigned short)(n01 >> 16))),
              __half2float(__ushort_as_half((unsigned short)(n23 & 0xffffu))));
}

// ascending sort of N unique keys held in registers (odd-even transposition; N <= 32)
template <uint32_t N>
__device__ __forceinline__ void sortKeys(uint32_t (&k)[N]) {
#pragma unroll
    for (uint32_t r = 0; r < N; r++) {
#pragma unroll
        for (uint32_t i = (r & 1u); i + 1 < N; i += 2) {
            const uint32_t a = k[i], b = k[i + 1];
            k[i] = a < b ? a : b;
            k[i + 1] = a < b ? b : a;
        }
    }
}

__device__ __forceinline__ Material loadMaterial(const ViewDev& V, uint32_t index) {
    const float4* __restrict__ materials = viewPtr(V.materials);
    const float4 m0 = __ldg(materials + 4 * size_t(index) + 0);
    const float4 m1 = __ldg(materials + 4 * size_t(index) + 1);
    const float4 m2 = __ldg(materials + 4 * size_t(index) + 2);
    const float4 m3 = __ldg(materials + 4 * size_t(index) + 3);
    Material mat;
    mat.emissive = f3(m0.x, m0.y, m0.z);
    mat.diffuse = f3(m1.x, m1.y, m1.z);
    mat.specular = f3(m2.x, m2.y, m2.z);
    mat.glossiness = m3.x;
    const uint32_t code0 = __float_as_uint(m3.z), code1 = __float_as_uint(m3.w);
    mat.model = code0 & 0xffffu;
    mat.texGloss = code0 >> 16;
    mat.texSpecular = code1 & 0xffffu;
    mat.texDiffuse = code1 >> 16;
    return mat;
}

// interpolate (shading.h:18-36) of a vertex attribute pair
__device__ __forceinline__ float2 interp2(float2 t0, float2 t1, float2 t2, F3 b) {
    return make_float2((t0.x * b.x + t1.x * b.y) + t2.x * b.z, (t0.y * b.x + t1.y * b.y) + t2.y * b.z);
}

// GGXShade (shading.h:84-161) of a hit whose material reads textures. The texture coordinates and
// their screen derivatives come from the hit's barycentrics at the shading point (bc) and one
// sample step along x (bx) and y (by): dUVdX = uv(bx) - uv(bc), dUVdY = uv(by) - uv(bc)
// (ShadeMSAA, resolve.cu:230-270). Kept out of line so the untextured path's registers do not
// grow.
__device__ __noinline__ F3 shadeTextured(const ViewDev& V, uint32_t triIndex, F3 bc, F3 bx, F3 by, F3 camPos,
                                         const LightEnvDev& env) {
    const uint4 ts = __ldg(viewPtr(V.triShade) + triIndex);
    const Material m = loadMaterial(V, ts.w);
    const float4* __restrict__ verts = viewPtr(V.verts);
    const float4 a0 = __ldg(verts + 2 * size_t(ts.x)), a1 = __ldg(verts + 2 * size_t(ts.x) + 1);
    const float4 p0 = __ldg(verts + 2 * size_t(ts.y)), p1 = __ldg(verts + 2 * size_t(ts.y) + 1);
    const float4 q0 = __ldg(verts + 2 * size_t(ts.z)), q1 = __ldg(verts + 2 * size_t(ts.z) + 1);
    const F3 pos = (f3(a0.x, a0.y, a0.z) * bc.x + f3(p0.x, p0.y, p0.z) * bc.y) + f3(q0.x, q0.y, q0.z) * bc.z;
    const F3 nrm = (halfNormal(a0, a1) * bc.x + halfNormal(p0, p1) * bc.y) + halfNormal(q0, q1) * bc.z;
    const float2 t0 = make_float2(a1.y, a1.z), t1 = make_float2(p1.y, p1.z), t2 = make_float2(q1.y, q1.z);
    const float2 uv = interp2(t0, t1, t2, bc);
    const float2 uvx = interp2(t0, t1, t2, bx), uvy = interp2(t0, t1, t2, by);
    const float2 dx = make_float2(uvx.x - uv.x, uvx.y - uv.y), dy = make_float2(uvy.x - uv.x, uvy.y - uv.y);
    const F3 normal = normalize3(nrm);
    float4 tex;
    if (m.model == 2u) return materialTexture(V, m.texDiffuse, uv, dx, dy, tex) ? f3(tex.x, tex.y, tex.z) : m.emissive;
    F3 base = m.diffuse;
    if (materialTexture(V, m.texDiffuse, uv, dx, dy, tex)) base = f3(tex.x, tex.y, tex.z);
    const F3 Vd = normalize3(camPos - pos);
    F3 F0 = m.specular;
    if (materialTexture(V, m.texSpecular, uv, dx, dy, tex)) F0 = f3(tex.x, tex.y, tex.z);
    float roughness = 1.0f - m.glossiness;
    if (materialTexture(V, m.texGloss, uv, dx, dy, tex)) roughness = 1.0f - tex.x;
    return ggxLit(m.emissive, base, F0, roughness, pos, normal, Vd, env);
}

// interpolate (shading.h:18-36) the hit's vertices at barycentrics bc and GGXShade it.
// deriv(bx, by) gives the barycentrics one sample step along x and y; it runs only when the
// material reads textures.
template <class Deriv>
__device__ __forceinline__ F3 shadeHit(const ViewDev& V, uint32_t triIndex, F3 bc, F3 camPos, const LightEnvDev& env,
                                       Deriv deriv) {
    const uint4 ts = __ldg(viewPtr(V.triShade) + triIndex);
    const Material mat = loadMaterial(V, ts.w);
    // with no texture in the scene every read falls back to the constants, which is the
    // untextured path
    if (V.textureCount && readsTextures(mat)) {
        F3 bx, by;
        deriv(bx, by);
        return shadeTextured(V, triIndex, bc, bx, by, camPos, env);
    }
    const float4* __restrict__ verts = viewPtr(V.verts);
    const float4 a0 = __ldg(verts + 2 * size_t(ts.x)), a1 = __ldg(verts + 2 * size_t(ts.x) + 1);
    const float4 p0 = __ldg(verts + 2 * size_t(ts.y)), p1 = __ldg(verts + 2 * size_t(ts.y) + 1);
    const float4 q0 = __ldg(verts + 2 * size_t(ts.z)), q1 = __ldg(verts + 2 * size_t(ts.z) + 1);
    const F3 pos = (f3(a0.x, a0.y, a0.z) * bc.x + f3(p0.x, p0.y, p0.z) * bc.y) + f3(q0.x, q0.y, q0.z) * bc.z;
    const F3 nrm = (halfNormal(a0, a1) * bc.x + halfNormal(p0, p1) * bc.y) + halfNormal(q0, q1) * bc.z;
    return ggxShade(mat, pos, nrm, camPos, env);
}

// TestTriangleFrustaUVW (prim_tests.h:89-116) over the tile's four world-space corner rays:
// true when every barycentric coordinate is out of [0, 1] on the same side for all four
__device__ __forceinline__ bool uvwAllOut(const float (&ro)[4][3], const float (&rd)[4][3], const TriGeom& tri) {
    float uMin = FLT_MAX, uMax = -FLT_MAX, vMin = FLT_MAX, vMax = -FLT_MAX, wMin = FLT_MAX, wMax = -FLT_MAX;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        float u, v, w;
        rayTriUVW(f3(ro[r][0], ro[r][1], ro[r][2]), f3(rd[r][0], rd[r][1], rd[r][2]), tri, u, v, w);
        uMin = tminf(uMin, u); uMax = tmaxf(uMax, u);
        vMin = tminf(vMin, v); vMax = tmaxf(vMax, v);
        wMin = tminf(wMin, w); wMax = tmaxf(wMax, w);
    }
    return uMax < 0 || uMin > 1 || vMax < 0 || vMin > 1 || wMax < 0 || wMin > 1;
}

// FrustumPlanes::test (prim_tests.h:30-50)
__device__ __forceinline__ bool inFrustum(const float (&pl)[4][4], const TriGeom& tri) {
    bool in = true;
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const F3 dir = f3(pl[p][0], pl[p][1], pl[p][2]);
        const float dist = pl[p][3];
        const float d0 = dot3(dir, tri.v0);
        const float d1 = d0 + dot3(dir, tri.e0);
        const float d2 = d0 + dot3(dir, tri.e1);
        if (d0 > dist && d1 > dist && d2 > dist) in = false;
    }
    return in;
}

// A long list is one CTA's: its four warps share the tile's tests and wait for one another after every batch, and
// where triangles are far smaller than samples a batch belongs to one warp. While few tiles have long lists (the
// order kernel's rule: at most kSplitTiles of at least 191 visits and 592 of 47, so that the chip has room) four
// CTAs take such a tile, each for one warp's samples: a list of at least kSplitEntries is culled against that
// warp's box alone, and nothing waits for another warp. Launch alone, one CTA and four, 57k triangles: from far above
// N = 8 160 x 120 11,855 and 9,174 us, 640 x 480 7,705 and 4,508; N = 2 1920 x 1080 893 and 574; from near 160 x 120
// N = 1 276 and 239. Of the longest 256 of many long lists it is slower (stereo 1,304 and 1,454, 1280 x 720 N = 32
// 872 and 1,060), hence the rule.
constexpr uint32_t kSplitEntries = 1024, kWhole = 4;

// The list is culled kBatchChunks chunks at a time; the next ones are copied in while their samples are tested.
constexpr uint32_t kBatchChunks = 2, kBatchSlots = kBatchChunks * kChunk;

struct ShadeSmem {
    float ro[4][3], rd[4][3]; // world corner rays
    float pl[4][4];           // frustum planes
    uint16_t cand[kBatchSlots];     // slots (chunk of the batch * 128 + thread) of the entries that can meet the
                                    // tile, in list order; they are tested kChunk at a time:
    float4 edge[4][kChunk];         // their edge planes through the camera and normals, with slack (edgePlane),
    float t[kChunk];
    uint32_t idx[kChunk];           // t and triangle index,
    uint32_t need[kChunk / 32][4];  // and per 32 of them and warp: which the warp's samples may hit
    float dir[6][kTileSize];        // -du, -dv of every sample
    float axis[3][4];          // three axes, about along the tile's beams' du, dv and c (orthonormal)
    float4 box[3][5];          // along axis k, of warp 0-3's and (4) the whole tile's -c: middle, half extent
    float warpT[4];            // per warp: the largest depth of its samples
    float warpMax[2][4];       // per warp: the largest footprint radius and beam length
    uint32_t warpCount[kBatchChunks][4];
    // the list triangles, 48 bytes per entry (three float4 rows of the triangle array), copied in by
    // cp.async
    float4 tri[kBatchSlots][3];
};

// cp.async of 16 bytes, global to shared, cached in L2 only (the triangle rows are gathered once
// per tile; neighbouring tiles share them through L2)
__device__ __forceinline__ void cpAsync16(void* dst, const void* src) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cpAsyncWaitAll() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// resident CTAs per SM that the register allocation must allow. Launch alone, one B200: N = 8 (1M triangles,
// stereo) 1,260 us with 7 CTAs of 72 registers, 1,305 with 8 of 64; N = 2 (1M, 1280 x 720) 484 and 565;
// N = 16 (foveated) 2,450 us with 6 CTAs of 80 registers, 2,526 with 5 of 96; N = 32 863 us with 4 of
// 128, 906 with 3 of 168.
template <uint32_t N> struct MinCtas { static constexpr int v = N <= 8 ? 7 : (N == 16 ? 6 : 4); };

// Where a shade launch takes its tiles from; item i of the launch is
//   kFromOrder: order[first + i] (order == nullptr: first + i), i < count;
//   kFromParts: the same, item i of the first kSplitTiles by the CTAs 4i to 4i + 3;
//   kFromReady: the tile published in ready[first + i] by the concurrent tile cull, waited for;
//   kFromList:  list[first + i], for i < *listCount (the retry list, counted on the device).
struct ShadeSource {
    const uint32_t* order;
    const uint32_t* ready;
    const uint32_t* list;
    const uint32_t* listCount;
    uint32_t first, count;
    const uint32_t* parts; // kFromParts: how many of the first items have use for four CTAs
};

// Waits (one thread) until the tile cull publishes a ready slot. A wait that runs past about a
// second gives up: it sets kStatusPipelineTimeout and returns kReadyEmpty, whose kReadyRetry bit
// makes the caller skip the slot.
__device__ uint32_t waitReady(const uint32_t* slot, uint32_t* counters) {
    for (uint32_t i = 0;; i++) {
        uint32_t v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(slot) : "memory");
        if (v != kReadyEmpty) return v;
        if (i >= (1u << 20)) {
            atomicOr(&counters[1], kStatusPipelineTimeout);
            return kReadyEmpty;
        }
        __nanosleep(i < 32 ? 128 : 1024);
    }
}

// Most of a tile's list never meets a given sample: it lies beside it, or behind what the sample has
// found. Testing every warp's 32 samples against every triangle that passed the tile's tests took
// 14.9M (warp, triangle) pairs of N tests on the 1M-triangle stereo frame; with the bounds below 6.6M
// (sample, triangle) pairs are left, tested two at a time. Launch alone, before and after: 1M triangles
// stereo N = 8 3,253 and 1,260 us, 1280 x 720 N = 2 1,313 and 484, 500k 1280 x 720 N = 32 3,857 and 863, foveated N = 16
// 7,941 and 2,450, 57k 640 x 480 N = 1 142 and 130. What bounds it now: issue (0.5 of the slots) and the
// latency of the chain list entry - tile - warp - sample - test.
//
// Which samples can a triangle hit at all? A subsample's v, w and u are linear in its direction dir =
// c + ax du + ay dv: v = -dir . gv with gv = v0r x e1, w = -dir . gw with gw = e0 x v0r, and u =
// -dir . gu with gu = n - gv - gw. Each has to have its sign bit clear, so a sample is passed by
// when for one of the three -c . g + radius |g| + (rounding) < 0, radius bounding |ax du + ay dv| (the
// unit offsets lie in the unit disk). With one or two subsamples the middle of their directions takes c's
// place and half their distance (0 for one) the radius: the disk is four times the area that two need, and a
// sample then tests little more than what it hits. The rounding term covers what the test's own operations and
// these may be off by: S = |v0r| (|e0| + |e1|) + |n| bounds every partial result over |dir|, each of
// the two sides loses less than 45 half-ulps of S |dir| (the middle's own rounding adds 8), and flushed
// denormals less than the last term. Launch alone with the disk and so: 57k triangles N = 1 640 x 480 137 and 85
// us, 160 x 120 615 and 276; from far above, dozens of triangles in a pixel, N = 1 7,216 and 1,768, N = 2 7,358
// and 6,368 (such a view was slower than without bounds: 4,106 and 4,678).
// The test also rejects a subsample when depth * denom < t: with denom = -dir . n at most d = -c . n +
// radius |n| + (rounding), and no subsample's depth above T, t > T d passes the sample by (with d < 0
// no subsample sees the front; the product's rounding is inside the slack).
// The samples that are left are tested as before, so hits and depths are the same bits.
// edge[e] = {g, slack}: -c . g + slack < 0 passes the sample by. (NaN keeps it.)
__device__ __forceinline__ float length(F3 g) { // (at least the length)
    const float g2 = fmaxf(fmaf(g.x, g.x, fmaf(g.y, g.y, g.z * g.z)), 1e-30f);
    float len;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(len) : "f"(g2));
    return len * 1.00001f;
}
__device__ __forceinline__ float4 edgePlane(F3 g, float radius, float slack) {
    return make_float4(g.x, g.y, g.z, fmaf(radius, length(g), slack));
}
__device__ __forceinline__ float norm1(F3 v) { return (fabsf(v.x) + fabsf(v.y)) + fabsf(v.z); }
__device__ __forceinline__ F3 cross3fma(F3 a, F3 b) {
    return f3(fmaf(a.y, b.z, -(a.z * b.y)), fmaf(a.z, b.x, -(a.x * b.z)), fmaf(a.x, b.y, -(a.y * b.x)));
}
__device__ __forceinline__ float edgeValue(F3 nc, float4 e) { return fmaf(nc.x, e.x, fmaf(nc.y, e.y, fmaf(nc.z, e.z, e.w))); }
__device__ __forceinline__ F3 unit(F3 v) { // (its length within 4 half-ulps of 1)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(dot3(v, v)));
    return v * r;
}
// Orthonormal axes about along du and dv, to a few half-ulps whatever du and dv are: the boxes' 2e-6 of the
// beam length is all that their error may cost. One step of dv - U (U . dv) leaves a share of U that grows as
// du and dv near each other (a viewport scaled very unequally under rotated ellipses), hence the second. A
// direction lost to rounding, to squares below the normal range, or because it is zero, is replaced. (One
// thread's chain, which the CTA waits for: no IEEE roots and divisions.)
__device__ __forceinline__ void boxAxes(F3 du, F3 dv, F3& U, F3& A, F3& W) {
    U = unit(du);
    if (!(fabsf(dot3(U, U) - 1.0f) < 1e-5f)) U = f3(1.0f, 0.0f, 0.0f);
    A = unit(dv - U * dot3(U, dv));
    A = A - U * dot3(U, A);
    if (!(dot3(A, A) > 0.5f && dot3(A, A) <= 2.0f)) { // the coordinate axis farthest from U, without its share of U
        const float x = fabsf(U.x), y = fabsf(U.y), z = fabsf(U.z);
        A = x <= y && x <= z ? f3(1.0f, 0.0f, 0.0f) : (y <= z ? f3(0.0f, 1.0f, 0.0f) : f3(0.0f, 0.0f, 1.0f));
        A = A - U * dot3(U, A);
    }
    A = unit(A);
    W = cross3(U, A);
}
// a plane's components along the tile's axes, and its value over a box of beams (its largest)
__device__ __forceinline__ F3 edgeAlong(const ShadeSmem& sm, float4 e) {
    const F3 g = f3(e.x, e.y, e.z);
    float a[3];
#pragma unroll
    for (int k = 0; k < 3; k++) a[k] = fmaf(sm.axis[k][0], g.x, fmaf(sm.axis[k][1], g.y, sm.axis[k][2] * g.z));
    return f3(a[0], a[1], a[2]);
}
__device__ __forceinline__ float edgeValue(const ShadeSmem& sm, uint32_t box, F3 a, float slack) {
    const float2 x = *reinterpret_cast<const float2*>(&sm.box[0][box]), y = *reinterpret_cast<const float2*>(&sm.box[1][box]),
                 z = *reinterpret_cast<const float2*>(&sm.box[2][box]);
    return fmaf(x.x, a.x, fmaf(y.x, a.y, fmaf(z.x, a.z, fmaf(x.y, fabsf(a.x), fmaf(y.y, fabsf(a.y), fmaf(z.y, fabsf(a.z), slack))))));
}
// a triangle's planes: gv, gw, gu and the normal, and its t
struct TriPlanes {
    float4 e[4];
    float t;
};
__device__ __forceinline__ TriPlanes trianglePlanes(const TriGeom& tri, F3 camPos, float radius, float maxLen) {
    TriPlanes x;
    const F3 nrm = cross3(tri.e0, tri.e1), v0r = camPos - tri.v0;
    x.t = dot3(v0r, nrm);
    const F3 gv = cross3fma(v0r, tri.e1), gw = cross3fma(tri.e0, v0r), gu = (nrm - gv) - gw;
    const float s1 = norm1(tri.e0) + norm1(tri.e1);
    const float slack = maxLen * (7e-6f * (norm1(v0r) * s1 + norm1(nrm)) + 1e-33f * (1.0f + s1));
    x.e[0] = edgePlane(gv, radius, slack);
    x.e[1] = edgePlane(gw, radius, slack);
    x.e[2] = edgePlane(gu, radius, slack);
    x.e[3] = edgePlane(nrm, radius, slack);
    return x;
}
// whether some sample of a box (depths at most farT) may be hit; a0-a3 the planes along the axes
__device__ __forceinline__ bool planesMeet(const ShadeSmem& sm, uint32_t box, F3 a0, F3 a1, F3 a2, F3 a3, const TriPlanes& x, float farT) {
    const float lowest = fminf(edgeValue(sm, box, a0, x.e[0].w), fminf(edgeValue(sm, box, a1, x.e[1].w), edgeValue(sm, box, a2, x.e[2].w)));
    return !(lowest < 0.0f) && !(x.t > farT * edgeValue(sm, box, a3, x.e[3].w));
}
// the larger depth, NaN if one is (a depth that is not a number rules nothing out)
__device__ __forceinline__ float farther(float a, float b) {
    float r;
    asm("max.NaN.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float warpMin(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fminf(v, __shfl_xor_sync(kFull, v, o));
    return v;
}
__device__ __forceinline__ float warpMax(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
    return v;
}

// the sample's subsamples against triangle ij, then ik, given by the first nine words of their rows
template <uint32_t N, bool FMA, int ROW>
__device__ __forceinline__ void testRows(const ShadeSmem& sm, F3 camPos, F3 ncs, const float4& j0, const float4& j1, float j2,
                                         uint32_t ij, const float4& k0, const float4& k1, float k2, uint32_t ik,
                                         float (&tmax)[N], uint32_t (&hit)[N]) {
    const V2 e0 = {pk(j0.w, k0.w), pk(j1.x, k1.x), pk(j1.y, k1.y)};
    const V2 e1 = {pk(j1.z, k1.z), pk(j1.w, k1.w), pk(j2, k2)};
    const V2 vr = {pk(camPos.x - j0.x, camPos.x - k0.x), pk(camPos.y - j0.y, camPos.y - k0.y),
                   pk(camPos.z - j0.z, camPos.z - k0.z)};
    const V2 nn = cross2(e0, e1);
    const P2 t2 = dot2(vr, nn);
    float tj, tk;
    upk(t2, tj, tk);
    const uint32_t tid = threadIdx.x;
    const F3 du = f3(sm.dir[0][tid], sm.dir[1][tid], sm.dir[2][tid]), dv = f3(sm.dir[3][tid], sm.dir[4][tid], sm.dir[5][tid]);
    const TriPair tp = pairSetup(nn, e0, e1, vr, V2{pk(ncs.x, ncs.x), pk(ncs.y, ncs.y), pk(ncs.z, ncs.z)},
                                 V2{pk(du.x, du.x), pk(du.y, du.y), pk(du.z, du.z)},
                                 V2{pk(dv.x, dv.x), pk(dv.y, dv.y), pk(dv.z, dv.z)});
    const P2 tt = FMA ? neg2(t2) : t2;
#pragma unroll
    for (uint32_t i = 0; i < N; i++) {
        const P2 ax = *reinterpret_cast<const P2*>(&cMsaaXX[ROW][i]);
        const P2 ay = *reinterpret_cast<const P2*>(&cMsaaYY[ROW][i]);
        pairTest<FMA>(tp, tt, tj, tk, ij, ik, ax, ay, tmax[i], hit[i]);
    }
}

// A list of at most kFewEntries is tested by every sample as it stands, without boxes and bounds, at up to 8
// subsamples: their setup, and a lane's rounds over its own triangles, cost more than the tests that they save.
// Launch alone, 1920 x 1080, one B200, with the bounds and so: a room of 14 triangles N = 1 143 and 106 us, N = 8
// 178 and 137; 768 triangles N = 4 208 and 158; 5,600 triangles N = 8 313 and 270. Up to 64 entries the last takes
// 248, but a textured frame over 57k triangles (N = 4) 228 us instead of 222 (218 with the bounds throughout).
constexpr uint32_t kFewEntries = 32;
template <uint32_t N> struct SampleHits {
    float t[N];
    uint32_t id[N];
};
// (out of line, so that the long lists' loop keeps its registers) returns how many entries pass the tile's tests
template <uint32_t N, bool FMA, int ROW>
__device__ __noinline__ uint32_t testFew(ShadeSmem& sm, const uint32_t* __restrict__ entries, uint32_t count,
                                         const float4* __restrict__ tris, F3 camPos, F3 ncs, SampleHits<N>& out) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    bool keep = false;
    if (tid < count) {
        const uint32_t ix = __ldcg(entries + tid);
        const float4* row = tris + 3 * size_t(ix);
        const float4 ra = __ldg(row), rb = __ldg(row + 1), rc = __ldg(row + 2);
        const TriGeom tri{f3(ra.x, ra.y, ra.z), f3(ra.w, rb.x, rb.y), f3(rb.z, rb.w, rc.x)};
        // IntersectTriangleTile<false>::setup, FrustumPlanes::test, TestTriangleFrustaUVW != intersect_all_out
        keep = !(dot3(camPos - tri.v0, cross3(tri.e0, tri.e1)) < 0.0f) && inFrustum(sm.pl, tri) && !uvwAllOut(sm.ro, sm.rd, tri);
        sm.tri[tid][0] = ra;
        sm.tri[tid][1] = rb;
        sm.tri[tid][2] = make_float4(rc.x, __uint_as_float(ix), 0.0f, 0.0f);
    }
    const uint32_t kept = __ballot_sync(kFull, keep);
    if (lane == 0) sm.need[warp][0] = kept;
    __syncthreads();
    float tmax[N];
    uint32_t hit[N];
#pragma unroll
    for (uint32_t i = 0; i < N; i++) {
        tmax[i] = FLT_MAX;
        hit[i] = ~0u;
    }
    // two at a time in list order; a last one alone as the pair (j, j)
    const uint32_t groups = (count + 31u) / 32u;
    uint32_t total = 0, g = 0, live = groups ? sm.need[0][0] : 0u, pend = ~0u;
    for (;;) {
        while (!live && g + 1 < groups) live = sm.need[++g][0];
        const bool end = !live;
        uint32_t j = pend;
        if (!end) {
            j = g * 32u + uint32_t(__ffs(live) - 1);
            live &= live - 1u;
            total++;
            if (pend == ~0u) {
                pend = j;
                continue;
            }
        }
        if (pend != ~0u) {
            const float4 *a = sm.tri[pend], *b = sm.tri[j];
            testRows<N, FMA, ROW>(sm, camPos, ncs, a[0], a[1], a[2].x, __float_as_uint(a[2].y), b[0], b[1], b[2].x,
                                  __float_as_uint(b[2].y), tmax, hit);
            pend = ~0u;
        }
        if (end) break;
    }
#pragma unroll
    for (uint32_t i = 0; i < N; i++) {
        out.t[i] = tmax[i];
        out.id[i] = hit[i];
    }
    return total;
}

// One tile: intersect, G-buffer grouping, shading and resolve of its 128 samples. The tile's
// list (TileList, chunk links, pool entries) is read through L2 (ld.cg): in a pipelined launch
// another SM wrote it while this launch was running.
// ROW: the row of the offset tables (the rate's spiral row, or + 6 for the rotated grid), a
// compile-time constant so that the offsets stay immediate constant-bank operands
// SPLIT: the tile may be one of four CTAs' (kWhole: it is not), of which each tests and shades one warp's samples.
template <uint32_t N, bool FMA, int ROW, bool SPLIT = false>
__device__ __forceinline__ void shadeTile(const FrameDev& fr, uint32_t gt, ShadeSmem& sm, LightEnvDev& env, Mat4& M,
                                          uint32_t part = kWhole) {
    const ViewDev& V = fr.views[fr.viewCount == 1 ? 0u : __ldg(fr.blockView + gt / kTilesPerBlock)];
    const uint32_t tile = gt - V.tileStart;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t sid = tile * kTileSize + tid;
    const uint2 lw = __ldcg(reinterpret_cast<const uint2*>(V.tileLists + tile));
    const TileList L{lw.x, lw.y};
    const bool split = SPLIT && part != kWhole && L.count >= kSplitEntries;
    if (SPLIT && !split && part != kWhole && part != 0) return;
    if (L.count == 0) {
        // ClearEmptyKernel (resolve.cu:527-542)
        V.colors[sid] = 0xFF000000u;
        if (V.tmaxOut) V.tmaxOut[sid] = INFINITY;
        uint32_t* __restrict__ hitOut = V.hitIds;
        float* __restrict__ depthOut = V.depth;
        if (hitOut) {
#pragma unroll
            for (uint32_t i = 0; i < N; i++) {
                hitOut[size_t(sid) * N + i] = ~0u;
                depthOut[size_t(sid) * N + i] = INFINITY;
            }
        }
        return;
    }
#ifdef HVVR_VISIT_CLOCKS
    long long scAcc[kScPhases] = {0, 0, 0, 0};
    long long scLast = phaseClock(L.count);
    uint32_t scChunks = 0;
#endif
    const int rate = ROW;
    for (uint32_t i = tid; i < sizeof(LightEnvDev) / 4; i += kTileSize)
        reinterpret_cast<uint32_t*>(&env)[i] = reinterpret_cast<const uint32_t*>(&V.env)[i];
    if (tid < 16) reinterpret_cast<float*>(&M)[tid] = reinterpret_cast<const float*>(&V.M)[tid];
    __syncthreads();
    // world-space tile rays (the SimpleRayFrustum of transformHierarchyCameraToWorld) and
    // FrustumPlanes (prim_tests.h:22-28)
    if (tid < 8) {
        const Rays4& cr = V.tileRays[tile];
        const uint32_t i = tid & 3u;
        if (tid < 4) {
            const F3 o = xformPoint(M, f3(cr.o[i][0], cr.o[i][1], cr.o[i][2]));
            sm.ro[i][0] = o.x; sm.ro[i][1] = o.y; sm.ro[i][2] = o.z;
        } else {
            const F3 d = xformDir(M, f3(cr.d[i][0], cr.d[i][1], cr.d[i][2]));
            sm.rd[i][0] = d.x; sm.rd[i][1] = d.y; sm.rd[i][2] = d.z;
        }
    }
    __syncthreads();
    if (tid < 4) {
        const F3 d0 = f3(sm.rd[tid][0], sm.rd[tid][1], sm.rd[tid][2]);
        const F3 d1 = f3(sm.rd[(tid + 1) & 3][0], sm.rd[(tid + 1) & 3][1], sm.rd[(tid + 1) & 3][2]);
        const F3 n = cross3(d0, d1);
        sm.pl[tid][0] = n.x; sm.pl[tid][1] = n.y; sm.pl[tid][2] = n.z;
        sm.pl[tid][3] = dot3(f3(sm.ro[tid][0], sm.ro[tid][1], sm.ro[tid][2]), n);
    }
    const F3 camPos = f3(M.m[3][0], M.m[3][1], M.m[3][2]);
    // this thread's beam, rotated to world space (GetDirectionalSample3D, gpu_samples.h:78-82)
    // this thread's beam, rotated to world space (GetDirectionalSample3D, gpu_samples.h:78-82): c,
    // du, dv; loaded again after the triangle loop so that they need no registers during it
    auto beamDirs = [&](F3& c, F3& du, F3& dv) {
        const float4* __restrict__ beams = V.beams;
        const float4 b0 = __ldg(beams + 3 * size_t(sid) + 0);
        const float4 b1 = __ldg(beams + 3 * size_t(sid) + 1);
        const float4 b2 = __ldg(beams + 3 * size_t(sid) + 2);
        c = xformDir(M, f3(b0.x, b0.y, b0.z));
        du = xformDir(M, f3(b0.w, b1.x, b1.y));
        dv = xformDir(M, f3(b1.z, b1.w, b2.x));
    };
    const bool few = N <= 8 && L.count <= kFewEntries;
    F3 ncs, mid; // -c, and minus the direction that the bounds are taken around
    {
        F3 c, du, dv;
        beamDirs(c, du, dv);
        mid = ncs = -c;
        sm.dir[0][tid] = -du.x; sm.dir[1][tid] = -du.y; sm.dir[2][tid] = -du.z;
        sm.dir[3][tid] = -dv.x; sm.dir[4][tid] = -dv.y; sm.dir[5][tid] = -dv.z;
        if (!few) {
            // Upper bound on |denom| / |e0 x e1| over this sample's subsamples: denom = -dir . n with
            // dir = c + ax du + ay dv and |ax|,|ay| <= 1, so |denom| <= (|c| + |du| + |dv|) |n|.
            const float dirLen = (sqrtf(dot3(c, c)) + sqrtf(dot3(du, du)) + sqrtf(dot3(dv, dv))) * 1.0001f;
            // |ax du + ay dv| over the subsamples: the larger singular value of (du dv); of one or two, half their
            // distance, around their middle
            float radius;
            if constexpr (N <= 2) {
                const float2 o0 = cMsaa[rate][0], o1 = cMsaa[rate][N - 1];
                mid = -(c + du * (0.5f * (o0.x + o1.x)) + dv * (0.5f * (o0.y + o1.y)));
                const F3 half = du * (0.5f * (o0.x - o1.x)) + dv * (0.5f * (o0.y - o1.y));
                radius = sqrtf(dot3(half, half)) * 1.00002f;
            } else {
                const float uu = dot3(du, du), vv = dot3(dv, dv), uv = dot3(du, dv), hd = 0.5f * (uu - vv);
                radius = sqrtf(0.5f * (uu + vv) + sqrtf(hd * hd + uv * uv)) * 1.00002f;
            }
            // (a beam that is not finite has to pass nothing by: its NaN or infinity must survive the maxima)
            const float finite = (norm1(c) + norm1(du)) + norm1(dv);
            const uint32_t r = __reduce_max_sync(kFull, __float_as_uint(finite <= FLT_MAX ? radius : INFINITY));
            const uint32_t d = __reduce_max_sync(kFull, __float_as_uint(finite <= FLT_MAX ? dirLen : INFINITY));
            if (tid == 0) {
                F3 U, A, W;
                boxAxes(du, dv, U, A, W);
                sm.axis[0][0] = U.x; sm.axis[0][1] = U.y; sm.axis[0][2] = U.z;
                sm.axis[1][0] = A.x; sm.axis[1][1] = A.y; sm.axis[1][2] = A.z;
                sm.axis[2][0] = W.x; sm.axis[2][1] = W.y; sm.axis[2][2] = W.z;
            }
            if (lane == 0) {
                sm.warpMax[0][warp] = __uint_as_float(r);
                sm.warpMax[1][warp] = __uint_as_float(d);
                sm.warpT[warp] = FLT_MAX;
            }
            __syncthreads();
            // the warp's beams in a box along the axes
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float p = dot3(mid, f3(sm.axis[k][0], sm.axis[k][1], sm.axis[k][2])), lo = warpMin(p), hi = warpMax(p);
                if (lane == 0) sm.box[k][warp] = make_float4(0.5f * (lo + hi), 0.5f * (hi - lo) * 1.0001f + 2e-6f * __uint_as_float(d), lo, hi);
            }
        }
    }
    float tmax[N];
    uint32_t hit[N];
#pragma unroll
    for (uint32_t i = 0; i < N; i++) {
        tmax[i] = FLT_MAX;
        hit[i] = ~0u;
    }
    __syncthreads();
    const float4* __restrict__ trisG = viewPtr(V.tris);
    uint32_t survivors = 0, tested = 0, lanesTested = 0;
    if (few) {
        SHADE_MARK(kScSetup, L.first);
        SampleHits<N> hits;
        lanesTested = tested = testFew<N, FMA, ROW>(sm, fr.pool + size_t(L.first) * kChunk, L.first < fr.poolChunks ? L.count : 0u, trisG,
                                                    camPos, ncs, hits);
        survivors = warp ? 0u : tested;
#pragma unroll
        for (uint32_t i = 0; i < N; i++) {
            tmax[i] = hits.t[i];
            hit[i] = hits.id[i];
        }
        SHADE_MARK(kScTest, tested);
#ifdef HVVR_VISIT_CLOCKS
        ++scChunks;
#endif
    } else {
        const float maxRadius = fmaxf(fmaxf(sm.warpMax[0][0], sm.warpMax[0][1]), fmaxf(sm.warpMax[0][2], sm.warpMax[0][3]));
        const float maxLen = fmaxf(fmaxf(sm.warpMax[1][0], sm.warpMax[1][1]), fmaxf(sm.warpMax[1][2], sm.warpMax[1][3]));
        if (tid < 3) {
            const float lo = fminf(fminf(sm.box[tid][0].z, sm.box[tid][1].z), fminf(sm.box[tid][2].z, sm.box[tid][3].z));
            const float hi = fmaxf(fmaxf(sm.box[tid][0].w, sm.box[tid][1].w), fmaxf(sm.box[tid][2].w, sm.box[tid][3].w));
            sm.box[tid][4] = make_float4(0.5f * (lo + hi), 0.5f * (hi - lo) * 1.0001f + 2e-6f * maxLen, lo, hi);
        }
        __syncthreads();
        SHADE_MARK(kScSetup, L.first);

        // Entry tid of a chunk is copied into shared memory by cp.async (the 48-byte triangle record that its
        // index names) while the CTA is still testing the batch before.
        uint32_t chunk = L.first, remaining = L.count; // the chunk to copy next and its entries, with all after them
        uint32_t ready[kBatchChunks], idx[kBatchChunks]; // the copied chunks' entries, this thread's entry of each
        auto copyBatch = [&] {
#pragma unroll
            for (uint32_t b = 0; b < kBatchChunks; b++) {
                ready[b] = chunk < fr.poolChunks ? (remaining < kChunk ? remaining : kChunk) : 0u;
                idx[b] = 0;
                if (tid < ready[b]) {
                    idx[b] = __ldcg(fr.pool + size_t(chunk) * kChunk + tid);
                    const float4* src = trisG + 3 * size_t(idx[b]);
                    for (uint32_t k = 0; k < 3; k++) cpAsync16(&sm.tri[b * kChunk + tid][k], src + k);
                }
                if (ready[b]) {
                    remaining -= ready[b];
                    chunk = remaining ? __ldcg(fr.chunkNext + chunk) : kNoChunk;
                }
            }
            cpAsyncCommit();
        };
        // Triangles that wait to be tested by this lane (kNone: none): when a lane gets a third, or the list
        // ends, every lane tests those it has, in list order - the first in lane 0 and the second in lane 1
        // of every packed operation (pairTest). A lone one is tested as the pair (j, j): a second test of the
        // same triangle on the same subsample changes nothing (it either fails or writes the same depth and
        // index again).
        constexpr uint32_t kNone = ~0u;
        uint32_t wait0 = kNone, wait1 = kNone;
        float laneT = FLT_MAX; // the largest depth of the lane's subsamples
        copyBatch();
        for (bool more = true; more;) {
            // Which entries of the batch can meet the tile: the triangle's planes against the tile's box of beams
            uint32_t kept = 0;
            const float tileT = split ? sm.warpT[part] : farther(farther(sm.warpT[0], sm.warpT[1]), farther(sm.warpT[2], sm.warpT[3]));
            cpAsyncWaitAll();
#pragma unroll
            for (uint32_t b = 0; b < kBatchChunks; b++) {
                bool keep = false;
                const uint32_t slot = b * kChunk + tid;
                if (tid < ready[b]) {
                    const float4 ra = sm.tri[slot][0], rb = sm.tri[slot][1], rc = sm.tri[slot][2];
                    const TriGeom tri{f3(ra.x, ra.y, ra.z), f3(ra.w, rb.x, rb.y), f3(rb.z, rb.w, rc.x)};
                    const TriPlanes x = trianglePlanes(tri, camPos, maxRadius, maxLen);
                    if (!(x.t < 0.0f)) // IntersectTriangleTile<false>::setup
                        keep = planesMeet(sm, split ? part : 4u, edgeAlong(sm, x.e[0]), edgeAlong(sm, x.e[1]), edgeAlong(sm, x.e[2]),
                                          edgeAlong(sm, x.e[3]), x, tileT);
                }
                const uint32_t bal = __ballot_sync(kFull, keep);
                if (lane == 0) sm.warpCount[b][warp] = __popc(bal);
                kept |= (keep ? 1u : 0u) << b;
                if (keep) sm.tri[slot][2].y = __uint_as_float(idx[b]); // (a triangle row's last three words are unused)
            }
            __syncthreads();
            uint32_t have = 0;
#pragma unroll
            for (uint32_t b = 0; b < kBatchChunks; b++) {
                const uint32_t bal = __ballot_sync(kFull, (kept >> b) & 1u);
                uint32_t off = have + __popc(bal & ((1u << lane) - 1u));
#pragma unroll
                for (uint32_t w = 0; w < 4; w++) {
                    const uint32_t cw = sm.warpCount[b][w];
                    off += (w < warp) ? cw : 0u;
                    have += cw;
                }
                if ((kept >> b) & 1u) sm.cand[off] = uint16_t(b * kChunk + tid);
            }
            __syncthreads();
            SHADE_MARK(kScCull, have);
            for (uint32_t first = 0; first == 0 || first < have; first += kChunk) {
                // The tile's own tests on those, one per thread, and which warps need them. The depth bounds are
                // the last round's; depths only fall, so they skip no triangle that could hit.
                const uint32_t groups = first < have ? (min(have - first, kChunk) + 31u) / 32u : 0u;
                if (warp < groups) {
                    const uint32_t js = first + tid;
                    uint32_t warps = 0;
                    if (js < have) {
                        const uint32_t slot = sm.cand[js];
                        const float4 ra = sm.tri[slot][0], rb = sm.tri[slot][1], rc = sm.tri[slot][2];
                        const TriGeom tj{f3(ra.x, ra.y, ra.z), f3(ra.w, rb.x, rb.y), f3(rb.z, rb.w, rc.x)};
                        const TriPlanes x = trianglePlanes(tj, camPos, maxRadius, maxLen);
                        const F3 a0 = edgeAlong(sm, x.e[0]), a1 = edgeAlong(sm, x.e[1]), a2 = edgeAlong(sm, x.e[2]), a3 = edgeAlong(sm, x.e[3]);
#pragma unroll
                        for (uint32_t w = 0; w < 4; w++)
                            if ((!split || w == part) && planesMeet(sm, w, a0, a1, a2, a3, x, sm.warpT[w])) warps |= 1u << w;
                        // FrustumPlanes::test, TestTriangleFrustaUVW != intersect_all_out
                        if (warps && !(inFrustum(sm.pl, tj) && !uvwAllOut(sm.ro, sm.rd, tj))) warps = 0;
                        if (warps) {
#pragma unroll
                            for (int e = 0; e < 4; e++) sm.edge[e][tid] = x.e[e];
                            sm.t[tid] = x.t;
                            sm.idx[tid] = __float_as_uint(rc.y);
                        }
                    }
                    survivors += __popc(__ballot_sync(kFull, warps != 0));
#pragma unroll
                    for (uint32_t w = 0; w < 4; w++) {
                        const uint32_t b = __ballot_sync(kFull, (warps >> w) & 1u);
                        if (lane == w) sm.need[warp][w] = b;
                    }
                }
                const bool last = first + kChunk >= have; // (of the batch)
                __syncthreads();
                if (last) {
                    copyBatch();
                    more = ready[0] != 0;
                }
                auto mayHit = [&](uint32_t slot) {
                    const float lowest = fminf(edgeValue(mid, sm.edge[0][slot]),
                                               fminf(edgeValue(mid, sm.edge[1][slot]), edgeValue(mid, sm.edge[2][slot])));
                    return !(lowest < 0.0f) && !(sm.t[slot] > laneT * edgeValue(mid, sm.edge[3][slot]));
                };
                uint32_t g = 0, mine = 0; // mine: the group's triangles that the lane still has to take
                for (;;) {
                    if (!__any_sync(kFull, mine != 0)) {
                        if (g == groups) {
                            if (more || !last) break;
                        } else {
                            // every lane decides which of its warp's triangles its own sample needs (two at a time;
                            // an odd one twice)
                            for (uint32_t live = sm.need[g][warp]; live;) {
                                const uint32_t b0 = uint32_t(__ffs(live) - 1);
                                live &= live - 1u;
                                const uint32_t b1 = live ? uint32_t(__ffs(live) - 1) : b0;
                                live &= live - 1u;
                                const bool p0 = mayHit(g * 32u + b0), p1 = mayHit(g * 32u + b1);
                                mine |= (p0 ? 1u << b0 : 0u) | (p1 ? 1u << b1 : 0u);
                            }
                            tested += __popc(__reduce_or_sync(kFull, mine));
                            g++;
                        }
                    }
                    // take up to two
                    for (int k = 0; k < 2; k++)
                        if (mine && wait1 == kNone) {
                            const uint32_t tri = sm.idx[(g - 1u) * 32u + uint32_t(__ffs(mine) - 1)];
                            mine &= mine - 1u;
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(trisG + 3 * size_t(tri)));
                            if (wait0 == kNone) wait0 = tri;
                            else wait1 = tri;
                        }
                    const bool end = g == groups && !more && last && !__any_sync(kFull, mine != 0);
                    if (__any_sync(kFull, end ? wait0 != kNone : mine != 0)) {
                        if (wait0 != kNone) {
                            const uint32_t ij = wait0, ik = wait1 == kNone ? wait0 : wait1;
                            lanesTested += wait1 == kNone ? 1u : 2u;
                            const float4* rj = trisG + 3 * size_t(ij);
                            const float4* rk = trisG + 3 * size_t(ik);
                            const float4 j0 = __ldg(rj), j1 = __ldg(rj + 1), k0 = __ldg(rk), k1 = __ldg(rk + 1);
                            const float j2 = __ldg(&rj[2].x), k2 = __ldg(&rk[2].x);
                            testRows<N, FMA, ROW>(sm, camPos, ncs, j0, j1, j2, ij, k0, k1, k2, ik, tmax, hit);
                            laneT = 0.0f;
#pragma unroll
                            for (uint32_t i = 0; i < N; i++) laneT = farther(laneT, tmax[i]);
                            wait0 = wait1 = kNone;
                        }
                        __syncwarp();
                    }
                    if (end) break;
                }
                const uint32_t far = __reduce_max_sync(kFull, __float_as_uint(laneT));
                if (lane == 0) sm.warpT[warp] = __uint_as_float(far);
                __syncthreads();
            }
            SHADE_MARK(kScTest, remaining);
#ifdef HVVR_VISIT_CLOCKS
            scChunks += kBatchChunks;
#endif
        }
    }

    if (lane == 0 && survivors) atomicAdd(&fr.counters[kSurvivorWord], survivors);
    if (lane == 0 && tested) atomicAdd(&fr.counters[kTestedWord], tested);
    lanesTested = __reduce_add_sync(kFull, lanesTested);
    if (lane == 0 && lanesTested) atomicAdd(&fr.counters[kSampleTestedWord], lanesTested);
    if (split && warp != part) return;
    F3 c, du, dv;
    beamDirs(c, du, dv);
    if (uint32_t* hitOut = viewPtr(V.hitIds)) {
        float* depthOut = viewPtr(V.depth);
#pragma unroll
        for (uint32_t i = 0; i < N; i++) {
            hitOut[size_t(sid) * N + i] = hit[i];
            depthOut[size_t(sid) * N + i] = hit[i] == ~0u ? INFINITY : tmax[i];
        }
    }
    // ResolveKernel's TMaxBuffer (resolve.cu:386-457): depth along the view axis of subsample 0's
    // triangle at subsample 0's position
    if (float* tmaxOut = viewPtr(V.tmaxOut)) {
        float tv = INFINITY;
        if (hit[0] != ~0u) {
            const TriGeom tri = loadTri(viewPtr(V.tris), hit[0]);
            const TriThread th = threadSetup(tri.e0, tri.e1, camPos - tri.v0, c, du, dv);
            const float2 a0 = cMsaa[rate][0];
            const F3 uvw = calcUVW<FMA>(th, a0.x, a0.y);
            const F3 p = (tri.v0 * uvw.x + (tri.v0 + tri.e0) * uvw.y) + (tri.v0 + tri.e1) * uvw.z;
            const F3 look = f3(-M.m[2][0], -M.m[2][1], -M.m[2][2]);
            tv = dot3(p - camPos, look);
        }
        tmaxOut[sid] = tv;
    }

    // G-buffer grouping (EmitGBuffer): (triangle, mask) pairs in ascending triangle order,
    // misses (~0) last; then ShadeMSAA over the groups in that order.
    uint32_t keys[N];
#pragma unroll
    for (uint32_t i = 0; i < N; i++) keys[i] = (hit[i] << 5) | i;
    bool uniform = true;
#pragma unroll
    for (uint32_t i = 1; i < N; i++) uniform = uniform && (hit[i] == hit[0]);
    if (!uniform) sortKeys<N>(keys);
    float rx = 0.0f, ry = 0.0f, rz = 0.0f;
    const uint32_t maskAll = N < 32 ? ((1u << N) - 1u) : ~0u;
    uint32_t combined = 0;
    uint32_t gi = 0;
    while (gi < N) {
        if (combined == maskAll) break;
        const uint32_t triIndex = uint32_t(int32_t(keys[gi]) >> 5);
        if (triIndex == ~0u) break;
        uint32_t sampleMask = 0;
        uint32_t gj = gi;
        if (uniform) {
            sampleMask = maskAll;
            gj = N;
        } else {
            while (gj < N && uint32_t(int32_t(keys[gj]) >> 5) == triIndex) {
                sampleMask |= 1u << (keys[gj] & 31u);
                gj++;
            }
        }
        gi = gj;
        combined |= sampleMask;
        const float pc = float(__popc(sampleMask));
        const float inv = 1.0f / pc;
        float cax = 0.0f, cay = 0.0f;
        for (uint32_t cm = sampleMask; cm;) {
            const int si = __ffs(cm) - 1;
            cm &= ~(1u << si);
            const float2 a = cMsaa[rate][si];
            cax = cax + a.x * inv;
            cay = cay + a.y * inv;
        }
        const TriGeom tri = loadTri(viewPtr(V.tris), triIndex);
        const F3 v0r = camPos - tri.v0;
        const TriThread th = threadSetup(tri.e0, tri.e1, v0r, c, du, dv);
        const F3 bc = calcUVW<FMA>(th, cax, cay);
        const F3 col = shadeHit(V, triIndex, bc, camPos, env, [&](F3& bx, F3& by) {
            bx = calcUVW<FMA>(th, cax + 1.0f, cay + 0.0f);
            by = calcUVW<FMA>(th, cax + 0.0f, cay + 1.0f);
        });
        rx = rx + col.x * pc;
        ry = ry + col.y * pc;
        rz = rz + col.z * pc;
    }
    const float sN = 1.0f / float(N);
    viewPtr(V.colors)[sid] = packColor(f3(aces(rx * sN), aces(ry * sN), aces(rz * sN)));
#ifdef HVVR_VISIT_CLOCKS
    __syncthreads();
    SHADE_MARK(kScShade, gi);
    if (tid == 0 && gt < kShadeClockTiles) {
        for (uint32_t k = 0; k < kScPhases; k++) gShadeClocks[gt][k] = uint64_t(scAcc[k]);
        gShadeClocks[gt][kScPhases] = scChunks;
        gShadeClocks[gt][kScPhases + 1] = L.count;
    }
#endif
}

// SRC selects where the launch's tiles come from (ShadeSource): kFromOrder and kFromReady run one
// tile per CTA; kFromList walks the list with a grid-stride loop.
enum : int { kFromOrder = 0, kFromReady = 1, kFromList = 2, kFromParts = 3 };

template <uint32_t N, bool FMA, int SRC, int ROW>
__global__ void __launch_bounds__(kTileSize, MinCtas<N>::v) intersectShadeKernel(FrameDev fr, ShadeSource src) {
    __shared__ ShadeSmem sm;
    __shared__ LightEnvDev env;
    __shared__ Mat4 M;
    // (the cull, where this launch was scheduled before its end)
    if constexpr (SRC == kFromOrder || SRC == kFromParts) asm volatile("griddepcontrol.wait;" ::: "memory");
    if constexpr (SRC == kFromOrder) {
        const uint32_t gt = src.order ? src.order[src.first + blockIdx.x] : src.first + blockIdx.x;
        shadeTile<N, FMA, ROW>(fr, gt, sm, env, M);
    } else if constexpr (SRC == kFromParts) {
        const uint32_t four = min(src.count, uint32_t(kSplitTiles)); // the items that have four CTAs
        uint32_t item = blockIdx.x, part = kWhole;
        if (item < 4 * four) {
            part = item & 3u;
            item >>= 2;
            if (item >= __ldcg(src.parts)) {
                if (part) return;
                part = kWhole;
            }
        } else {
            item -= 3 * four;
        }
        shadeTile<N, FMA, ROW, true>(fr, src.order[src.first + item], sm, env, M, part);
    } else if constexpr (SRC == kFromReady) {
        __shared__ uint32_t readyTile;
        if (threadIdx.x == 0) readyTile = waitReady(src.ready + src.first + blockIdx.x, fr.counters);
        __syncthreads();
        const uint32_t gt = readyTile;
        if (gt & kReadyRetry) return; // culled and shaded by the retry passes (or the wait gave up)
        shadeTile<N, FMA, ROW>(fr, gt, sm, env, M);
    } else {
        const uint32_t count = *src.listCount;
        for (uint32_t item = blockIdx.x; item < count; item += gridDim.x) {
            shadeTile<N, FMA, ROW>(fr, src.list[src.first + item] & ~kRetryGiant, sm, env, M);
            __syncthreads();
        }
    }
}

// ------------------------------------------------------------------ thin lens (depth of field)
// IntersectTriangleTile<true>, IntersectTriangleThreadDoF (prim_tests.h:247-392), TileData<true>
// (tile_data.h:33-60), GetSampleUVsDoF (gpu_samples.h:84-103), and the DoF branches of
// IntersectSamples / ShadeMSAA (intersect.cu:117-168, resolve.cu:161-284). FMA selects the
// contraction the kernel comments mark (per-subsample t, denom, depth, ray origin/direction,
// cross and dot products).
__device__ __forceinline__ F3 fma3(float s, F3 a, F3 c) { return f3(fmaf(s, a.x, c.x), fmaf(s, a.y, c.y), fmaf(s, a.z, c.z)); }

template <bool FMA>
__device__ __forceinline__ void dofBary(F3 e0, F3 e1, F3 v0l, float ddx, float ddy, float dc, F3 lc2fc, F3 lu, F3 lv,
                                        float2 luv, float2 duv, float& denom, float& v, float& w) {
    if (FMA) {
        denom = fmaf(ddy, duv.y, fmaf(ddx, duv.x, dc));
        const F3 o = fma3(luv.y, lv, fma3(luv.x, lu, v0l));
        const F3 a = -fma3(duv.y, lv, fma3(duv.x, lu, lc2fc));
        const F3 e = f3(fmaf(a.y, o.z, -(a.z * o.y)), fmaf(a.z, o.x, -(a.x * o.z)), fmaf(a.x, o.y, -(a.y * o.x)));
        v = fmaf(e1.z, e.z, fmaf(e1.y, e.y, e1.x * e.x));
        w = -fmaf(e0.z, e.z, fmaf(e0.y, e.y, e0.x * e.x));
    } else {
        denom = dc + ddx * duv.x + ddy * duv.y;
        const F3 o = (v0l + lu * luv.x) + lv * luv.y;
        const F3 rd = (lc2fc + lu * duv.x) + lv * duv.y;
        const F3 e = cross3(-rd, o);
        v = dot3(e1, e);
        w = -dot3(e0, e);
    }
}

// dirUV = aaOffset * focalToLensScale - lensUV
template <bool FMA>
__device__ __forceinline__ float2 dofDirUV(float2 aa, float fx, float fy, float2 luv) {
    return FMA ? make_float2(fmaf(aa.x, fx, -luv.x), fmaf(aa.y, fy, -luv.y))
               : make_float2(aa.x * fx - luv.x, aa.y * fy - luv.y);
}

struct DofSmem {
    float ro[4][3], rd[4][3]; // world corner rays
    float pl[4][4];           // frustum planes
    float lensU[3], lensV[3], fls[2];
    uint32_t idx[kChunk];
    float tc[kChunk], tu[kChunk], tv[kChunk], ddx[kChunk], ddy[kChunk];
    float e0[3][kChunk];
    float e1[3][kChunk];
    float4 vl[kChunk];      // lens centre - v0; at most any subsample's t
    float4 edge[4][kChunk]; // edge planes through the lens centre and normal, with their slack
    float4 blur[kChunk];    // lensR times the lengths of e1, e0, e1 - e0
    float warpMax[4];
    uint32_t warpCount[4];
};

// The thin lens's form of the pinhole's bounds (edgePlane): which samples can a triangle hit? A
// subsample's ray starts at d from the lens centre (|d| at most lensR) and passes the focal plane at
// c + A, c the sample's lens centre to focal point and |A| at most footR, so its direction is c + A - d.
// With q = v0l + c + A (v0 to that point) the terms in d collect:
//   v = -(c + A) . gv + d . (q x e1)     w = -(c + A) . gw + d . (e0 x q)
//   u = -(c + A) . gu + d . ((e0 - q) x (e1 - e0))
// so that each is at most -c . g + footR |g| + lensR |q| |edge| (u: + lensR |n|): the blur of a point
// grows with its distance from the sample's focal point. t is at least tc - lensR |n|, and denom at
// most -c . n + (footR + lensR) |n|. The rounding terms are four times the pinhole's (the per-subsample
// origin and direction are rounded too). A sample is passed by when v, w or u is negative everywhere,
// or when t > T denom for the largest depth T of its subsamples.
// 57k triangles 640 x 480, N = 8, launch alone, one B200: every sample against every triangle of its tile
// 651 us (13.5M sample tests); with d and c bounded apart (the blur of the whole depth) 445 us (3.2M); so
// 330 us (1.0M). Bounded by issue: a third is shading. (At 80 registers for six CTAs 378 us.)
template <uint32_t N, bool FMA>
__global__ void __launch_bounds__(kTileSize) intersectShadeDofKernel(FrameDev fr, const uint32_t* __restrict__ order,
                                                                     uint32_t first) {
    __shared__ DofSmem sm;
    __shared__ LightEnvDev env;
    __shared__ Mat4 M;
    const uint32_t gt = order ? order[first + blockIdx.x] : first + blockIdx.x;
    const ViewDev& V = fr.views[fr.viewCount == 1 ? 0u : __ldg(fr.blockView + gt / kTilesPerBlock)];
    const uint32_t tile = gt - V.tileStart;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t sid = tile * kTileSize + tid;
    const TileList L = V.tileLists[tile];
    if (L.count == 0) {
        V.colors[sid] = 0xFF000000u;
        if (uint32_t* hitOut = V.hitIds) {
#pragma unroll
            for (uint32_t i = 0; i < N; i++) {
                hitOut[size_t(sid) * N + i] = ~0u;
                V.depth[size_t(sid) * N + i] = INFINITY;
            }
        }
        return;
    }
    const int rate = RateIndex<N>::v;
    for (uint32_t i = tid; i < sizeof(LightEnvDev) / 4; i += kTileSize)
        reinterpret_cast<uint32_t*>(&env)[i] = reinterpret_cast<const uint32_t*>(&V.env)[i];
    if (tid < 16) reinterpret_cast<float*>(&M)[tid] = reinterpret_cast<const float*>(&V.M)[tid];
    __syncthreads();
    const float4* __restrict__ beams = V.beams;
    const float4 b0 = __ldg(beams + 3 * size_t(sid) + 0);
    const float4 b1 = __ldg(beams + 3 * size_t(sid) + 1);
    const float4 b2 = __ldg(beams + 3 * size_t(sid) + 2);
    const F3 c = xformDir(M, f3(b0.x, b0.y, b0.z));
    if (tid < 8) {
        const Rays4& cr = V.tileRays[tile];
        const uint32_t i = tid & 3u;
        if (tid < 4) {
            const F3 o = xformPoint(M, f3(cr.o[i][0], cr.o[i][1], cr.o[i][2]));
            sm.ro[i][0] = o.x; sm.ro[i][1] = o.y; sm.ro[i][2] = o.z;
        } else {
            const F3 d = xformDir(M, f3(cr.d[i][0], cr.d[i][1], cr.d[i][2]));
            sm.rd[i][0] = d.x; sm.rd[i][1] = d.y; sm.rd[i][2] = d.z;
        }
    }
    if (tid == kTileSize / 2) {
        // TileData<true>::load on this sample's world-space beam; the reference rotates the
        // already rotated du/dv a second time (cameraToWorldRotation * sample.du); kept
        const F3 fu = xformDir(M, xformDir(M, f3(b0.w, b1.x, b1.y)));
        const F3 fv = xformDir(M, xformDir(M, f3(b1.z, b1.w, b2.x)));
        const float uInv = 1.0f / sqrtf(dot3(fu, fu)), vInv = 1.0f / sqrtf(dot3(fv, fv));
        const float uMag = 1.0f / uInv, vMag = 1.0f / vInv;
        const F3 lu = fu * (V.lensRadius * uInv), lv = fv * (V.lensRadius * vInv);
        sm.lensU[0] = lu.x; sm.lensU[1] = lu.y; sm.lensU[2] = lu.z;
        sm.lensV[0] = lv.x; sm.lensV[1] = lv.y; sm.lensV[2] = lv.z;
        const float sc = V.focalDistance / V.lensRadius;
        sm.fls[0] = sc * uMag;
        sm.fls[1] = sc * vMag;
    }
    __syncthreads();
    if (tid < 4) {
        const F3 d0 = f3(sm.rd[tid][0], sm.rd[tid][1], sm.rd[tid][2]);
        const F3 d1 = f3(sm.rd[(tid + 1) & 3][0], sm.rd[(tid + 1) & 3][1], sm.rd[(tid + 1) & 3][2]);
        const F3 n = cross3(d0, d1);
        sm.pl[tid][0] = n.x; sm.pl[tid][1] = n.y; sm.pl[tid][2] = n.z;
        sm.pl[tid][3] = dot3(f3(sm.ro[tid][0], sm.ro[tid][1], sm.ro[tid][2]), n);
    }
    const F3 camPos = f3(M.m[3][0], M.m[3][1], M.m[3][2]);
    // IntersectSamples: lens centre to the focal point of this sample's centre ray
    const F3 centerDir = normalize3(c);
    const float zed = dot3(xformDir(M, f3(0.0f, 0.0f, -1.0f)), centerDir);
    const F3 lc2fc = centerDir * (V.focalDistance / zed);
    {
        const float len = sqrtf(dot3(lc2fc, lc2fc)) * 1.00001f; // (one that is not finite passes nothing by)
        const uint32_t m = __reduce_max_sync(kFull, __float_as_uint(len <= FLT_MAX ? len : INFINITY));
        if (lane == 0) sm.warpMax[warp] = __uint_as_float(m);
    }
    // GetSampleUVsDoF: table tile = the reference's occupied-tile CTA index mod 4
    const float2* __restrict__ lensPos = V.lensPos + (V.occRank[tile] & 3u) * kTileSize * N + tid;
    float tmax[N];
    uint32_t hit[N];
#pragma unroll
    for (uint32_t i = 0; i < N; i++) {
        tmax[i] = FLT_MAX;
        hit[i] = ~0u;
    }
    __syncthreads();
    const F3 lu = f3(sm.lensU[0], sm.lensU[1], sm.lensU[2]), lv = f3(sm.lensV[0], sm.lensV[1], sm.lensV[2]);
    const float flsx = sm.fls[0], flsy = sm.fls[1];
    const float uu = dot3(lu, lu), vv = dot3(lv, lv);
    const float uv = dot3(lu, lv);
    // the larger singular values of (lu lv) and (lu flsx, lv flsy)
    auto sigma = [](float a, float b, float c) {
        const float h = 0.5f * (a - b);
        return sqrtf(0.5f * (a + b) + sqrtf(h * h + c * c)) * 1.00002f;
    };
    const float lensR = sigma(uu, vv, uv), footR = sigma(uu * (flsx * flsx), vv * (flsy * flsy), uv * (flsx * flsy));
    const float maxLen = fmaxf(fmaxf(sm.warpMax[0], sm.warpMax[1]), fmaxf(sm.warpMax[2], sm.warpMax[3])) + footR + lensR;
    const F3 toward = -lc2fc;

    uint32_t chunk = L.first;
    uint32_t remaining = L.count;
    uint32_t survivors = 0, tested = 0, lanesTested = 0;
    while (remaining > 0 && chunk < fr.poolChunks) {
        const uint32_t n = remaining < kChunk ? remaining : kChunk;
        const uint32_t nextChunk = fr.chunkNext[chunk];
        bool keep = false;
        uint32_t idx = 0;
        TriGeom tri{};
        F3 v0l = f3(0, 0, 0);
        float tc = 0.0f, tu = 0.0f, tv = 0.0f, ddx = 0.0f, ddy = 0.0f;
        if (tid < n) {
            idx = fr.pool[size_t(chunk) * kChunk + tid];
            tri = loadTri(viewPtr(V.tris), idx);
            bool in = true;
#pragma unroll
            for (int p = 0; p < 4; p++) {
                const F3 dir = f3(sm.pl[p][0], sm.pl[p][1], sm.pl[p][2]);
                const float dist = sm.pl[p][3];
                const float d0 = dot3(dir, tri.v0);
                const float d1 = d0 + dot3(dir, tri.e0);
                const float d2 = d0 + dot3(dir, tri.e1);
                if (d0 > dist && d1 > dist && d2 > dist) in = false;
            }
            if (in) {
                // IntersectTriangleTile<true>::setup
                const F3 normal = cross3(tri.e0, tri.e1);
                v0l = camPos - tri.v0;
                tc = dot3(v0l, normal);
                tu = dot3(lu, normal);
                tv = dot3(lv, normal);
                const float tExtent = fabsf(tu) + fabsf(tv);
                if (!(tc + tExtent < 0.0f)) {
                    ddx = dot3(-lu, normal);
                    ddy = dot3(-lv, normal);
                    // the corner-ray test only when every lens position sees the front of the plane
                    keep = (tc - tExtent < 0.0f) || !uvwAllOut(sm.ro, sm.rd, tri);
                }
            }
        }
        const uint32_t bal = __ballot_sync(kFull, keep);
        if (lane == 0) sm.warpCount[warp] = __popc(bal);
        __syncthreads();
        uint32_t off = __popc(bal & ((1u << lane) - 1u));
        uint32_t total = 0;
#pragma unroll
        for (uint32_t w = 0; w < 4; w++) {
            const uint32_t cw = sm.warpCount[w];
            off += (w < warp) ? cw : 0u;
            total += cw;
        }
        if (keep) {
            sm.idx[off] = idx;
            sm.tc[off] = tc; sm.tu[off] = tu; sm.tv[off] = tv; sm.ddx[off] = ddx; sm.ddy[off] = ddy;
            sm.e0[0][off] = tri.e0.x; sm.e0[1][off] = tri.e0.y; sm.e0[2][off] = tri.e0.z;
            sm.e1[0][off] = tri.e1.x; sm.e1[1][off] = tri.e1.y; sm.e1[2][off] = tri.e1.z;
            const F3 gv = cross3fma(v0l, tri.e1), gw = cross3fma(tri.e0, v0l), nn = cross3(tri.e0, tri.e1), gu = (nn - gv) - gw;
            const float s1 = norm1(tri.e0) + norm1(tri.e1), nv = norm1(v0l) + lensR, nl = norm1(nn);
            const float slack = maxLen * (2.4e-5f * (nv * s1 + nl) + 1e-33f * (1.0f + s1)), lenN = length(nn);
            const float b1 = lensR * length(tri.e1), b0 = lensR * length(tri.e0), b01 = lensR * length(tri.e1 - tri.e0);
            sm.edge[0][off] = edgePlane(gv, footR, fmaf(footR, b1, slack));
            sm.edge[1][off] = edgePlane(gw, footR, fmaf(footR, b0, slack));
            sm.edge[2][off] = edgePlane(gu, footR, fmaf(footR, b01, fmaf(lensR, lenN, slack)));
            sm.edge[3][off] = edgePlane(nn, footR + lensR, slack);
            sm.blur[off] = make_float4(b1, b0, b01, 0.0f);
            sm.vl[off] = make_float4(v0l.x, v0l.y, v0l.z, tc - fmaf(lensR * 1.00001f, lenN, 2.4e-5f * nv * nl));
        }
        survivors += total;
        __syncthreads();
        for (uint32_t g0 = 0; g0 < total; g0 += 32) {
            // every lane decides which triangles its own sample needs, then tests those in list order
            float laneT = 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < N; i++) laneT = fmaxf(laneT, tmax[i]);
            uint32_t mine = 0;
            for (uint32_t j = g0; j < min(total, g0 + 32u); j++) {
                const float4 vl = sm.vl[j], blur = sm.blur[j];
                const float q = length(f3(vl.x - toward.x, vl.y - toward.y, vl.z - toward.z));
                const float lowest = fminf(fmaf(q, blur.x, edgeValue(toward, sm.edge[0][j])),
                                           fminf(fmaf(q, blur.y, edgeValue(toward, sm.edge[1][j])),
                                                 fmaf(q, blur.z, edgeValue(toward, sm.edge[2][j]))));
                if (!(lowest < 0.0f) && !(vl.w > laneT * edgeValue(toward, sm.edge[3][j]))) mine |= 1u << (j - g0);
            }
            tested += __popc(__reduce_or_sync(kFull, mine));
            lanesTested += __popc(mine);
            for (; mine; mine &= mine - 1u) {
                const uint32_t j = g0 + uint32_t(__ffs(mine) - 1);
                const F3 je0 = f3(sm.e0[0][j], sm.e0[1][j], sm.e0[2][j]);
                const F3 je1 = f3(sm.e1[0][j], sm.e1[1][j], sm.e1[2][j]);
                const float4 vl = sm.vl[j];
                const F3 jvl = f3(vl.x, vl.y, vl.z);
                const float jtc = sm.tc[j], jtu = sm.tu[j], jtv = sm.tv[j], jdx = sm.ddx[j], jdy = sm.ddy[j];
                const uint32_t jidx = sm.idx[j];
                // IntersectTriangleThreadDoF ctor
                const float dc = dot3(-lc2fc, cross3(je0, je1));
#pragma unroll
                for (uint32_t i = 0; i < N; i++) {
                    const float2 luv = __ldg(lensPos + i * kTileSize);
                    const float2 duv = dofDirUV<FMA>(cMsaa[rate][i], flsx, flsy, luv);
                    const float t = FMA ? fmaf(jtv, luv.y, fmaf(jtu, luv.x, jtc)) : jtc + jtu * luv.x + jtv * luv.y;
                    float denom, v, w;
                    dofBary<FMA>(je0, je1, jvl, jdx, jdy, dc, lc2fc, lu, lv, luv, duv, denom, v, w);
                    const float depthDelta = FMA ? fmaf(tmax[i], denom, -t) : tmax[i] * denom - t;
                    const float u = denom - v - w;
                    const int test = __float_as_int(t) | __float_as_int(depthDelta) | __float_as_int(u) |
                                     __float_as_int(v) | __float_as_int(w);
                    // NaN fails (a padding sample's zero beam normalises to NaN; the sign-bit test alone
                    // would depend on which NaN the hardware produces)
                    if (test >= 0 && u == u && depthDelta == depthDelta) {
                        tmax[i] = hitDepth(t, denom);
                        hit[i] = jidx;
                    }
                }
            }
        }
        __syncthreads();
        remaining -= n;
        chunk = nextChunk;
    }
    if (tid == 0 && survivors) atomicAdd(&fr.counters[kSurvivorWord], survivors);
    if (lane == 0 && tested) atomicAdd(&fr.counters[kTestedWord], tested);
    lanesTested = __reduce_add_sync(kFull, lanesTested);
    if (lane == 0 && lanesTested) atomicAdd(&fr.counters[kSampleTestedWord], lanesTested);

    if (uint32_t* hitOut = viewPtr(V.hitIds)) {
        float* depthOut = viewPtr(V.depth);
#pragma unroll
        for (uint32_t i = 0; i < N; i++) {
            hitOut[size_t(sid) * N + i] = hit[i];
            depthOut[size_t(sid) * N + i] = hit[i] == ~0u ? INFINITY : tmax[i];
        }
    }

    // EmitGBuffer grouping, then ShadeMSAA's DoF branch: centroid lens and direction UVs
    uint32_t keys[N];
#pragma unroll
    for (uint32_t i = 0; i < N; i++) keys[i] = (hit[i] << 5) | i;
    bool uniform = true;
#pragma unroll
    for (uint32_t i = 1; i < N; i++) uniform = uniform && (hit[i] == hit[0]);
    if (!uniform) sortKeys<N>(keys);
    float rx = 0.0f, ry = 0.0f, rz = 0.0f;
    const uint32_t maskAll = N < 32 ? ((1u << N) - 1u) : ~0u;
    uint32_t combined = 0;
    uint32_t gi = 0;
    while (gi < N) {
        if (combined == maskAll) break;
        const uint32_t triIndex = uint32_t(int32_t(keys[gi]) >> 5);
        if (triIndex == ~0u) break;
        uint32_t sampleMask = 0;
        uint32_t gj = gi;
        if (uniform) {
            sampleMask = maskAll;
            gj = N;
        } else {
            while (gj < N && uint32_t(int32_t(keys[gj]) >> 5) == triIndex) {
                sampleMask |= 1u << (keys[gj] & 31u);
                gj++;
            }
        }
        gi = gj;
        combined |= sampleMask;
        const float pc = float(__popc(sampleMask));
        const float inv = 1.0f / pc;
        float clx = 0.0f, cly = 0.0f, cdx = 0.0f, cdy = 0.0f;
        for (uint32_t cm = sampleMask; cm;) {
            const int si = __ffs(cm) - 1;
            cm &= ~(1u << si);
            const float2 luv = __ldg(lensPos + uint32_t(si) * kTileSize);
            const float2 duv = dofDirUV<FMA>(cMsaa[rate][si], flsx, flsy, luv);
            clx = clx + luv.x * inv; cly = cly + luv.y * inv;
            cdx = cdx + duv.x * inv; cdy = cdy + duv.y * inv;
        }
        const TriGeom tri = loadTri(viewPtr(V.tris), triIndex);
        const F3 normal = cross3(tri.e0, tri.e1);
        const F3 v0l = camPos - tri.v0;
        const float tdx = dot3(-lu, normal), tdy = dot3(-lv, normal), tdc = dot3(-lc2fc, normal);
        // IntersectTriangleThreadDoF::calcUVW at the centroid lens position and direction duv
        auto baryAt = [&](float2 duv) {
            float denom, v, w;
            dofBary<FMA>(tri.e0, tri.e1, v0l, tdx, tdy, tdc, lc2fc, lu, lv, make_float2(clx, cly), duv, denom, v, w);
            const float u = denom - v - w;
            const float dinv = 1.0f / denom;
            return f3(u * dinv, v * dinv, w * dinv);
        };
        // the derivatives step the centroid direction by (1, 0) and (0, 1) (ShadeMSAA's DoF branch)
        const F3 col = shadeHit(V, triIndex, baryAt(make_float2(cdx, cdy)), camPos, env, [&](F3& bx, F3& by) {
            bx = baryAt(make_float2(cdx + 1.0f, cdy + 0.0f));
            by = baryAt(make_float2(cdx + 0.0f, cdy + 1.0f));
        });
        rx = rx + col.x * pc;
        ry = ry + col.y * pc;
        rz = rz + col.z * pc;
    }
    const float sN = 1.0f / float(N);
    viewPtr(V.colors)[sid] = packColor(f3(aces(rx * sN), aces(ry * sN), aces(rz * sN)));
}

// a launch over tiles in their order; parts: see launchIntersectShade; early: the launch before it in the stream is
// the retry pass of the cull, and this one may be scheduled before that ends
template <uint32_t N, bool FMA, int ROW>
cudaError_t launchOrdered(const FrameDev& fr, const uint32_t* order, uint32_t first, uint32_t count, const uint32_t* parts,
                          bool early, cudaStream_t st) {
    const ShadeSource src{order, nullptr, nullptr, nullptr, first, count, parts};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(count + (parts ? 3u * std::min<uint32_t>(count, kSplitTiles) : 0u));
    cfg.blockDim = dim3(kTileSize);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    return parts ? cudaLaunchKernelEx(&cfg, intersectShadeKernel<N, FMA, kFromParts, ROW>, fr, src)
                 : cudaLaunchKernelEx(&cfg, intersectShadeKernel<N, FMA, kFromOrder, ROW>, fr, src);
}

template <uint32_t N>
cudaError_t launchRate(const FrameDev& fr, uint32_t pattern, bool fpStrict, bool dof, const uint32_t* order,
                       uint32_t first, uint32_t count, const uint32_t* parts, bool early, cudaStream_t st) {
    constexpr int S = RateIndex<N>::v, G = RateIndex<N>::v + 6; // spiral / rotated-grid offset rows
    if (dof) {
        if (fpStrict) intersectShadeDofKernel<N, false><<<count, kTileSize, 0, st>>>(fr, order, first);
        else intersectShadeDofKernel<N, true><<<count, kTileSize, 0, st>>>(fr, order, first);
        return cudaGetLastError();
    }
    if (fpStrict)
        return pattern ? launchOrdered<N, false, G>(fr, order, first, count, parts, early, st)
                       : launchOrdered<N, false, S>(fr, order, first, count, parts, early, st);
    return pattern ? launchOrdered<N, true, G>(fr, order, first, count, parts, early, st)
                   : launchOrdered<N, true, S>(fr, order, first, count, parts, early, st);
}

// The cull -> shade pipeline of one rate class (launchCullShadePipeline).
template <uint32_t N, bool FMA, int ROW>
cudaError_t launchPipelineRate(const FrameDev& fr, uint32_t first, uint32_t count, uint32_t* queues, uint32_t* pipe,
                               uint32_t warps, uint32_t stackLimit, cudaStream_t st) {
    cudaError_t e = launchTileCullMain(fr, fr.order, first, count, queues, warps, stackLimit, fr.ready, pipe, st);
    if (e != cudaSuccess) return e;
    // CTA i shades the i-th tile the cull finishes; the launch may start once every cull CTA runs
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(count);
    cfg.blockDim = dim3(kTileSize);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const ShadeSource ready{nullptr, fr.ready, nullptr, nullptr, first, count, nullptr};
    if ((e = cudaLaunchKernelEx(&cfg, intersectShadeKernel<N, FMA, kFromReady, ROW>, fr, ready)) != cudaSuccess) return e;
    // tiles whose stack outgrew the main pass: culled again, then shaded by a small grid that walks
    // the retry list (its length is only known on the device)
    if ((e = launchTileCullRetryPass(fr, fr.order, first, count, queues, stackLimit, false, st)) != cudaSuccess) return e;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t grid = std::min<uint32_t>(count, uint32_t(2 * (sms > 0 ? sms : 148)));
    const ShadeSource retried{nullptr, nullptr, fr.retry, queues + 1, first, count, nullptr};
    intersectShadeKernel<N, FMA, kFromList, ROW><<<grid, kTileSize, 0, st>>>(fr, retried);
    return cudaGetLastError();
}

template <uint32_t N>
cudaError_t launchPipelineFp(const FrameDev& fr, uint32_t pattern, bool fpStrict, uint32_t first, uint32_t count,
                             uint32_t* queues, uint32_t* pipe, uint32_t warps, uint32_t stackLimit, cudaStream_t st) {
    constexpr int S = RateIndex<N>::v, G = RateIndex<N>::v + 6;
    if (pattern)
        return fpStrict ? launchPipelineRate<N, false, G>(fr, first, count, queues, pipe, warps, stackLimit, st)
                        : launchPipelineRate<N, true, G>(fr, first, count, queues, pipe, warps, stackLimit, st);
    return fpStrict ? launchPipelineRate<N, false, S>(fr, first, count, queues, pipe, warps, stackLimit, st)
                    : launchPipelineRate<N, true, S>(fr, first, count, queues, pipe, warps, stackLimit, st);
}

// RemapKernel (libraries/hvvr/raycaster/remap.cu:35-77) for split-colour 1, 2 (pentile) and 3
__global__ void remapKernel(const uint32_t* __restrict__ src, const int32_t* __restrict__ remap,
                            uint32_t* __restrict__ dst, uint32_t width, uint32_t height, uint64_t stride,
                            uint32_t split) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= width || y >= height) return;
    const size_t p = size_t(y) * width + x;
    if (split == 1) {
        const int32_t o = remap[p];
        if (o >= 0) dst[size_t(y) * stride + x] = src[o];
        return;
    }
    uint32_t cc[3] = {0, 0, 0};
    for (uint32_t ch = 0; ch < split; ch++) {
        const int32_t o = remap[p * split + ch];
        if (o >= 0) cc[ch] = src[o];
    }
    dst[size_t(y) * stride + x] = split == 2
                                      ? ((cc[1] & 0xffu) | (cc[0] & 0xff00u) | (cc[1] & 0xff0000u) | 0xff000000u)
                                      : ((cc[0] & 0xffu) | (cc[1] & 0xff00u) | (cc[2] & 0xff0000u) | 0xff000000u);
}

} // namespace

cudaError_t launchIntersectShade(const FrameDev& fr, uint32_t msaa, uint32_t pattern, bool fpStrict, bool dof,
                                 const uint32_t* order, uint32_t first, uint32_t count, const uint32_t* parts,
                                 bool early, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    switch (msaa) {
    case 1: return launchRate<1>(fr, pattern, fpStrict, dof, order, first, count, parts, early, st);
    case 2: return launchRate<2>(fr, pattern, fpStrict, dof, order, first, count, parts, early, st);
    case 4: return launchRate<4>(fr, pattern, fpStrict, dof, order, first, count, parts, early, st);
    case 8: return launchRate<8>(fr, pattern, fpStrict, dof, order, first, count, parts, early, st);
    case 16: return launchRate<16>(fr, pattern, fpStrict, dof, order, first, count, parts, early, st);
    case 32: return launchRate<32>(fr, pattern, fpStrict, dof, order, first, count, parts, early, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launchCullShadePipeline(const FrameDev& fr, uint32_t msaa, uint32_t pattern, bool fpStrict, uint32_t first,
                                    uint32_t count, uint32_t* queues, uint32_t* pipe, uint32_t warps,
                                    uint32_t stackLimit, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    if (!fr.ready) return cudaErrorInvalidValue;
    switch (msaa) {
    case 1: return launchPipelineFp<1>(fr, pattern, fpStrict, first, count, queues, pipe, warps, stackLimit, st);
    case 2: return launchPipelineFp<2>(fr, pattern, fpStrict, first, count, queues, pipe, warps, stackLimit, st);
    case 4: return launchPipelineFp<4>(fr, pattern, fpStrict, first, count, queues, pipe, warps, stackLimit, st);
    case 8: return launchPipelineFp<8>(fr, pattern, fpStrict, first, count, queues, pipe, warps, stackLimit, st);
    case 16: return launchPipelineFp<16>(fr, pattern, fpStrict, first, count, queues, pipe, warps, stackLimit, st);
    case 32: return launchPipelineFp<32>(fr, pattern, fpStrict, first, count, queues, pipe, warps, stackLimit, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launchRemap(const CameraDev& c, cudaStream_t st) {
    if (!c.image || !c.remap || c.width == 0 || c.height == 0) return cudaSuccess;
    const dim3 block(16, 8);
    const dim3 grid((c.width + 15) / 16, (c.height + 7) / 8);
    remapKernel<<<grid, block, 0, st>>>(c.colors, c.remap, c.image, c.width, c.height, c.imageStride, c.split);
    return cudaGetLastError();
}

cudaError_t uploadMsaaTable(uint32_t n, uint32_t pattern, const float* offsets, cudaStream_t st) {
    int idx = -1;
    switch (n) {
    case 1: idx = 0; break;
    case 2: idx = 1; break;
    case 4: idx = 2; break;
    case 8: idx = 3; break;
    case 16: idx = 4; break;
    case 32: idx = 5; break;
    default: return cudaErrorInvalidValue;
    }
    if (pattern > 1) return cudaErrorInvalidValue;
    idx += 6 * int(pattern);
    // the packed products' addend (-0, -0), written with every table upload (mul2)
    const unsigned long long negZero2 = 0x8000000080000000ull;
    cudaError_t ez = cudaMemcpyToSymbolAsync(cNegZero2, &negZero2, sizeof(negZero2), 0, cudaMemcpyHostToDevice, st);
    if (ez != cudaSuccess) return ez;
    cudaError_t e = cudaMemcpyToSymbolAsync(cMsaa, offsets, n * sizeof(float2), size_t(idx) * 32 * sizeof(float2),
                                            cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    // the duplicated per-axis copies (pageable host staging: the copy completes before the call returns)
    float2 xs[32], ys[32];
    for (uint32_t i = 0; i < n; i++) {
        xs[i] = make_float2(offsets[2 * i], offsets[2 * i]);
        ys[i] = make_float2(offsets[2 * i + 1], offsets[2 * i + 1]);
    }
    e = cudaMemcpyToSymbolAsync(cMsaaXX, xs, n * sizeof(float2), size_t(idx) * 32 * sizeof(float2),
                                cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    return cudaMemcpyToSymbolAsync(cMsaaYY, ys, n * sizeof(float2), size_t(idx) * 32 * sizeof(float2),
                                   cudaMemcpyHostToDevice, st);
}

} // namespace hvb

#ifdef HVVR_VISIT_CLOCKS
// profiling build only: per global tile [0, tiles), kScPhases phase cycle sums of the intersect/shade
// CTA's thread 0, then its chunk count and list length
extern "C" int hvvr_dbg_shade_clocks(unsigned long long* out, uint32_t tiles) {
    if (!out || tiles > hvb::kShadeClockTiles) return HVVR_ERR_INVALID;
    return cudaMemcpyFromSymbol(out, hvb::gShadeClocks, size_t(tiles) * sizeof(hvb::gShadeClocks[0])) == cudaSuccess
               ? HVVR_OK
               : HVVR_ERR_CUDA;
}
#endif

