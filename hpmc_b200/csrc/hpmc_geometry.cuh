// hpmc_geometry.cuh -- vertex geometry of one MC edge crossing
// (shadergen.cpp:512-563): crossing parameter t, position and normal.
//
// FP32 samples and FP32 outputs.  The crossing parameter and the normal lerp
// are evaluated in "float-float" arithmetic (error-free TwoSum / FMA
// transformations, ~44 significant bits) on the FP32 pipes: a normal that
// nearly cancels, (1-t) A + t B with A ~ -B, keeps its direction to the
// rounding of the FP32 result, and no float<->double conversions are issued.
#pragma once
#include "hpmc_fetch.cuh"

namespace hpmc {

struct FF {
    float hi, lo;
};

// a + b = s + e exactly (Knuth)
__device__ __forceinline__ FF two_sum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    const float e = (a - (s - bb)) + (b - bb);
    return {s, e};
}

__device__ __forceinline__ FF ff_sub(FF a, FF b) {
    FF s = two_sum(a.hi, -b.hi);
    s.lo += a.lo - b.lo;
    return two_sum(s.hi, s.lo);
}

__device__ __forceinline__ FF ff_add(FF a, FF b) {
    FF s = two_sum(a.hi, b.hi);
    s.lo += a.lo + b.lo;
    return two_sum(s.hi, s.lo);
}

__device__ __forceinline__ FF ff_mul(FF a, FF b) {
    const float p = a.hi * b.hi;
    const float e = fmaf(a.hi, b.hi, -p) + (a.hi * b.lo + a.lo * b.hi);
    return two_sum(p, e);
}

// (a - b) / (c - d) for floats, as float-float
__device__ __forceinline__ FF ff_ratio_of_diffs(float a, float b, float c, float d) {
    const FF num = two_sum(a, -b);
    const FF den = two_sum(c, -d);
    const float q = num.hi / den.hi;
    float r = fmaf(-q, den.hi, num.hi);  // exact residual of the leading terms
    r += num.lo;
    r = fmaf(-q, den.lo, r);
    return two_sum(q, r / den.hi);
}

// lerp(A, B, t) = A + t (B - A), all float-float
__device__ __forceinline__ float ff_lerp(FF A, FF B, FF t) {
    const FF r = ff_add(A, ff_mul(t, ff_sub(B, A)));
    return r.hi + r.lo;
}

// A + t (B - A) with A = a - b, B = c - d for floats and t float-float, rounded
// once: every rounding error of a difference, the product and the sum is found
// exactly and added up with the low parts, so what is lost is of second order,
// as with ff_lerp (35 operations instead of 62).
__device__ __forceinline__ float lerp_of_diffs(float a, float b, float c, float d, FF t) {
    const FF A = two_sum(a, -b), B = two_sum(c, -d);
    const FF D = two_sum(B.hi, -A.hi);
    const float dlo = D.lo + (B.lo - A.lo);
    const float p = t.hi * D.hi;
    const float pe = fmaf(t.hi, D.hi, -p);
    const FF s = two_sum(A.hi, p);
    return s.hi + (s.lo + (pe + (fmaf(t.hi, dlo, t.lo * D.hi) + A.lo)));
}

// Integer lattice index -> float without the conversion pipe (0 <= v < 2^23).
__device__ __forceinline__ float index_to_float(int v) { return __int_as_float(0x4B000000 | v) - 8388608.0f; }

// One crossed edge: from lattice point a (its cell's corner, offset g & 7) along
// `axis` = g >> 3 = u; v, w are the next two axes (cyclically).
struct EdgeAt {
    int a[3];
    int axis;
    bool interior;      // every sample the vertex reads lies in an array field indexed with 32 bits ...
    uint32_t at;        // ... the element index of a ...
    int ou, ov, ow;     // ... and the element strides along u, v, w
};

// The samples of a cell's edges span cell-1 .. cell+3 on each axis.
__device__ __forceinline__ bool interior_cell(const Volume& V, int x, int y, int z) {
    return x >= 1 && x <= V.lattice[0] - 4 && y >= 1 && y <= V.lattice[1] - 4 && z >= 1 && z <= V.lattice[2] - 4;
}

// {element index of a - that of its cell, strides along u, v, w} of edge geometry g.
__device__ __forceinline__ int4 edge_strides(const Volume& V, uint32_t g) {
    const int oy = (int)V.row_pitch, oz = (int)V.slice_pitch, axis = (int)(g >> 3);
    return make_int4((int)(g & 1u) + (g & 2u ? oy : 0) + (g & 4u ? oz : 0), axis == 0 ? 1 : axis == 1 ? oy : oz,
                     axis == 0 ? oy : axis == 1 ? oz : 1, axis == 0 ? oz : axis == 1 ? 1 : oy);
}

// The edge of geometry g of cell (x, y, z).
__device__ __forceinline__ EdgeAt edge_at(const Volume& V, int x, int y, int z, uint32_t g) {
    const int4 o = edge_strides(V, g);
    EdgeAt E;
    E.a[0] = x + (int)(g & 1u);
    E.a[1] = y + (int)((g >> 1) & 1u);
    E.a[2] = z + (int)((g >> 2) & 1u);
    E.axis = (int)(g >> 3);
    E.interior = V.idx32 && interior_cell(V, x, y, z);
    E.at = (uint32_t)z * (uint32_t)V.slice_pitch + (uint32_t)y * (uint32_t)V.row_pitch + (uint32_t)x + (uint32_t)o.x;
    E.ou = o.y;
    E.ov = o.z;
    E.ow = o.w;
    return E;
}

// The field samples one vertex reads: f(a), f(b) with b = a + e_u, f(a - e_u),
// f(b + e_u), f(a +- e_v), ... -- 12 samples for central differences, 7 forward
// (f(a + e_u) is f(b), f(b - e_u) is f(a)).  All loads of a vertex are issued
// in one branch-free block: interior cells through 32-bit element offsets,
// boundary cells and fields of 2^31 elements through 64-bit ones that stay inside
// the lattice (GL_CLAMP + NEAREST), functor fields by evaluating the functor.
struct EdgeField {
    float va, vb;
    float am, bp;              // f(a - e_u) (central differences only), f(b + e_u)
    float ap[2], bpv[2];       // f(a + e_v), f(a + e_w); the same at b
    float amv[2], bmv[2];      // f(a - e_v), f(a - e_w); the same at b (central differences only)
};

// Component i of a vector given along (u, v, w).
__device__ __forceinline__ float unrotate(int axis, int i, const float r[3]) {
    const int at = i - axis;  // -2 .. 2, mod 3 the index along (u, v, w)
    return at == 0 ? r[0] : (at == 1 || at == -2) ? r[1] : r[2];
}

template <int FT, bool CENTRAL, class UF = NoUserField>
__device__ __forceinline__ void gather_edge(const Volume& V, const EdgeAt& E, EdgeField& F) {
    constexpr bool kArray = FT != kFieldFunctor && FT != kFieldUser;
    if (kArray && E.interior) {
        using T = typename std::conditional<
            FT == kFieldF32, float, typename std::conditional<FT == kFieldF32X4, float4, unsigned char>::type>::type;
        const T* field = static_cast<const T*>(V.field);
        auto ld = [&](uint32_t at) -> float {
            if constexpr (FT == kFieldF32) return __ldg(field + at);
            else if constexpr (FT == kFieldF32X4) return __ldg(&field[at].w);
            else if constexpr (FT == kFieldU8) return u8_to_float(__ldg(field + at));
            else return unorm8_to_float(__ldg(field + at));
        };
        const uint32_t pa = E.at, pb = E.at + (uint32_t)E.ou;
        const uint32_t o[2] = {(uint32_t)E.ov, (uint32_t)E.ow};
        F.va = ld(pa);
        F.vb = ld(pb);
        F.bp = ld(pb + (uint32_t)E.ou);
        if (CENTRAL) F.am = ld(pa - (uint32_t)E.ou);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            F.ap[i] = ld(pa + o[i]);
            F.bpv[i] = ld(pb + o[i]);
            if (CENTRAL) {
                F.amv[i] = ld(pa - o[i]);
                F.bmv[i] = ld(pb - o[i]);
            }
        }
    } else if constexpr (kArray) {
        // One offset per direction from a and from b (both inside the lattice), 0
        // where it would leave the lattice.  Clamping the three coordinates of each
        // sample instead costs a 64-bit index per sample and the registers for it:
        // the byte noise at 256^3 with a slice pitch of 8 MB took 1768 (forward)
        // and 2088 us (central) instead of 1648 and 1912, the batched traversal
        // spilled 188 bytes instead of 100 and took 4 to 5 % longer.
        auto along = [&](auto x, auto y, auto z, int i) {  // component i of (u, v, w)
            if (i == 0) return E.axis == 0 ? x : E.axis == 1 ? y : z;
            if (i == 1) return E.axis == 0 ? y : E.axis == 1 ? z : x;
            return E.axis == 0 ? z : E.axis == 1 ? x : y;
        };
        auto step = [&](int i, int d) -> long long {
            const uint32_t at = (uint32_t)(along(E.a[0], E.a[1], E.a[2], i) + d);
            const long long stride = along(1ll, V.row_pitch, V.slice_pitch, i);
            return at < (uint32_t)along(V.lattice[0], V.lattice[1], V.lattice[2], i) ? (d < 0 ? -stride : stride) : 0ll;
        };
        const long long pa = (long long)E.a[2] * V.slice_pitch + (long long)E.a[1] * V.row_pitch + E.a[0];
        const long long su = step(0, 1), pb = pa + su;
        F.va = fetch_raw<FT>(V, pa);
        F.vb = fetch_raw<FT>(V, pb);
        F.bp = fetch_raw<FT>(V, pb + step(0, 2));
        if (CENTRAL) F.am = fetch_raw<FT>(V, pa + step(0, -1));
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const long long up = step(i + 1, 1);
            F.ap[i] = fetch_raw<FT>(V, pa + up);
            F.bpv[i] = fetch_raw<FT>(V, pb + up);
            if (CENTRAL) {
                const long long down = step(i + 1, -1);
                F.amv[i] = fetch_raw<FT>(V, pa + down);
                F.bmv[i] = fetch_raw<FT>(V, pb + down);
            }
        }
    } else {
        const int u[3] = {E.axis == 0, E.axis == 1, E.axis == 2};
        auto at = [&](int nu, int nv, int nw) {
            // v is the axis after u, w the one before it
            return fetch<FT, UF>(V, E.a[0] + nu * u[0] + nv * u[2] + nw * u[1], E.a[1] + nu * u[1] + nv * u[0] + nw * u[2],
                                 E.a[2] + nu * u[2] + nv * u[1] + nw * u[0]);
        };
        F.va = at(0, 0, 0);
        F.vb = at(1, 0, 0);
        F.bp = at(2, 0, 0);
        if (CENTRAL) F.am = at(-1, 0, 0);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            F.ap[i] = at(0, i == 0, i == 1);
            F.bpv[i] = at(1, i == 0, i == 1);
            if (CENTRAL) {
                F.amv[i] = at(0, -(i == 0), -(i == 1));
                F.bmv[i] = at(1, -(i == 0), -(i == 1));
            }
        }
    }
}

enum { kGeomForward = 0, kGeomCentral = 1, kGeomBinary = 2 };

// Position (lattice index * extent / cells) and normal (scaled by extent /
// cells like the reference, shadergen.cpp:556-563) of the vertex on the edge
// from a (cell + shift) along `axis`.  Forward: n_i = iso - lerp(f(a+e_i),
// f(b+e_i), t); central: n_i = -lerp(g_i(a), g_i(b), t), g_i = half the
// central difference.
//
// The normal is first evaluated in plain FP32 (n_i = A_i + t (B_i - A_i) with
// A_i, B_i the end-point differences).  Its rounding error is bounded by
// 7u sqrt(sum_i (|A_i|+|B_i|)^2), u = 2^-24; when that bound exceeds 2e-6 of
// |n| (a normal that nearly cancels) the vertex is recomputed in float-float.
template <int FT, int MODE, class UF = NoUserField>
__device__ __forceinline__ void edge_vertex(const Volume& V, const EdgeAt& E, float p[3], float n[3], float& t_out) {
    const int* a = E.a;
    const int axis = E.axis;
    float t;
    if (MODE == kGeomBinary) {
        t = 0.5f;
        n[0] = n[1] = n[2] = 0.0f;  // the caller has the table normal of the vertex's case
    } else if (V.gradient) {
        // gradient mode (shadergen.cpp:539-551): t from the values at a and b,
        // the gradients from HPMC_fetchGrad -- a functor's analytic gradient or
        // the .xyz of an RGBA field (single-channel fields read zero there, as
        // GL's alpha textures do); forward mode keeps the reference's
        // n = iso - lerp(grad a, grad b, t), central mode gives -lerp(grad a, grad b, t)
        const int b[3] = {a[0] + (axis == 0), a[1] + (axis == 1), a[2] + (axis == 2)};
        float va, vb, ga[3] = {0.f, 0.f, 0.f}, gb[3] = {0.f, 0.f, 0.f};
        if constexpr (FT == kFieldFunctor) {
            const float pa[3] = {texel_centre(a[0], V.lattice[0]), texel_centre(a[1], V.lattice[1]),
                                 texel_centre(a[2], V.lattice[2])};
            const float pb[3] = {texel_centre(b[0], V.lattice[0]), texel_centre(b[1], V.lattice[1]),
                                 texel_centre(b[2], V.lattice[2])};
            va = functor_value(V.functor, pa[0], pa[1], pa[2]);
            vb = functor_value(V.functor, pb[0], pb[1], pb[2]);
            functor_gradient(V.functor, pa[0], pa[1], pa[2], ga[0], ga[1], ga[2]);
            functor_gradient(V.functor, pb[0], pb[1], pb[2], gb[0], gb[1], gb[2]);
        } else if constexpr (FT == kFieldUser) {
            const float pa[3] = {texel_centre(a[0], V.lattice[0]), texel_centre(a[1], V.lattice[1]),
                                 texel_centre(a[2], V.lattice[2])};
            const float pb[3] = {texel_centre(b[0], V.lattice[0]), texel_centre(b[1], V.lattice[1]),
                                 texel_centre(b[2], V.lattice[2])};
            va = UF::value(V.functor.p, V.functor.count, pa[0], pa[1], pa[2]);
            vb = UF::value(V.functor.p, V.functor.count, pb[0], pb[1], pb[2]);
            if constexpr (UF::kHasGradient) {
                UF::gradient(V.functor.p, V.functor.count, pa[0], pa[1], pa[2], ga);
                UF::gradient(V.functor.p, V.functor.count, pb[0], pb[1], pb[2], gb);
            }
        } else if constexpr (FT == kFieldF32X4) {
            const float4 sa = fetch_rgba(V, a[0], a[1], a[2]), sb = fetch_rgba(V, b[0], b[1], b[2]);
            va = sa.w;
            vb = sb.w;
            ga[0] = sa.x; ga[1] = sa.y; ga[2] = sa.z;
            gb[0] = sb.x; gb[1] = sb.y; gb[2] = sb.z;
        } else {
            va = fetch<FT, UF>(V, a[0], a[1], a[2]);
            vb = fetch<FT, UF>(V, b[0], b[1], b[2]);
        }
        const float iso = V.iso;
        const FF tf = ff_ratio_of_diffs(va, iso, va, vb);
        t = tf.hi + tf.lo;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const float g = ff_lerp(FF{ga[i], 0.0f}, FF{gb[i], 0.0f}, tf);
            n[i] = (MODE == kGeomCentral) ? -g : iso - g;
        }
    } else {
        EdgeField F{};
        gather_edge<FT, MODE == kGeomCentral, UF>(V, E, F);
        const float iso = V.iso;
        t = (F.va - iso) / (F.va - F.vb);  // (f(a) - iso) / (f(a) - f(b)), relative error <= 3u
        float s2 = 0.0f, n2 = 0.0f, r[3];  // r: the normal along (u, v, w)
        // end-point samples (forward) or differences (central) along u, v, w
        const float hiA[3] = {F.vb, F.ap[0], F.ap[1]}, hiB[3] = {F.bp, F.bpv[0], F.bpv[1]};
        const float loA[3] = {F.am, F.amv[0], F.amv[1]}, loB[3] = {F.va, F.bmv[0], F.bmv[1]};
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const float A = MODE == kGeomForward ? iso - hiA[i] : hiA[i] - loA[i];
            const float B = MODE == kGeomForward ? iso - hiB[i] : hiB[i] - loB[i];
            r[i] = fmaf(t, B - A, A);
            const float s = fabsf(A) + fabsf(B);
            s2 = fmaf(s, s, s2);
            n2 = fmaf(r[i], r[i], n2);
        }
        if (s2 > 23.0f * n2) {
            // ill-conditioned: float-float crossing parameter and lerps
            const FF tf = ff_ratio_of_diffs(F.va, iso, F.va, F.vb);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                r[i] = MODE == kGeomForward ? lerp_of_diffs(iso, hiA[i], iso, hiB[i], tf)
                                            : lerp_of_diffs(hiA[i], loA[i], hiB[i], loB[i], tf);
            }
            t = tf.hi + tf.lo;
        }
#pragma unroll
        for (int i = 0; i < 3; i++) n[i] = unrotate(axis, i, r) * (MODE == kGeomCentral ? -0.5f : 1.0f);
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
        float q = index_to_float(a[i]);
        if (i == axis) q += t;
        p[i] = q * V.scale[i];
        n[i] *= V.scale[i];
    }
    t_out = t;
}

}  // namespace hpmc
