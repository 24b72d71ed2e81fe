// What every kernel that shades and walks shares: the arithmetic, the random numbers, the primitive tests and the tree
// walk, the materials, lights and camera, one vertex of a path under either integrator, and where a sample lies in a
// launch. Included by each source that has kernels of its own, inside namespace rtb's anonymous namespace.
//
// The including source names its table `rounds` first: how each dot product below is rounded (rounding.cuh). With
// RTB_COMPACT_CODE defined, the random numbers and the large spheres' quadratic are called rather than inlined at each
// use: the NEE/MIS kernels' code outgrows the instruction cache, and a warp shading its paths waits for its
// instructions (measured in pool_quality.cu).
#pragma once

// ---- float3 arithmetic --------------------------------------------------------------------------------------
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator-(float3 a) { return make_float3(-a.x, -a.y, -a.z); }
__device__ __forceinline__ float3 operator*(float t, float3 v) { return make_float3(t * v.x, t * v.y, t * v.z); }
__device__ __forceinline__ float3 operator*(float3 a, float3 b) { return make_float3(a.x * b.x, a.y * b.y, a.z * b.z); }
// A dot product's rounding, written out or left to the compiler. Left to it, a * b + c * d becomes one multiply-add or
// the other by what surrounds it in each kernel, a last bit apart, and a path through glass makes another path of a
// last bit; written out, two kernels that render the same samples render the same image.
template <rounding R = rounds::other>
__device__ __forceinline__ float dot(float3 a, float3 b)
{
    if constexpr (R == rounding::x) // x fused onto y's product, z onto both
    {
        return __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)));
    }
    else if constexpr (R == rounding::y) // y fused onto x's product, z onto both
    {
        return __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)));
    }
    else if constexpr (R == rounding::yz) // y fused onto x's product, z's product rounded and added
    {
        return __fadd_rn(__fmul_rn(a.z, b.z), __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)));
    }
    else
    {
        return a.x * b.x + a.y * b.y + a.z * b.z;
    }
}
__device__ __forceinline__ float3 cross(float3 u, float3 v)
{
    return make_float3(u.y * v.z - u.z * v.y, u.z * v.x - u.x * v.z, u.x * v.y - u.y * v.x);
}
template <rounding R = rounds::other>
__device__ __forceinline__ float length_squared(float3 v)
{
    return dot<R>(v, v);
}
template <rounding R = rounds::other>
__device__ __forceinline__ float3 unit_vector(float3 v)
{
    return rsqrtf(length_squared<R>(v)) * v;
}
template <rounding R = rounds::other>
__device__ __forceinline__ float3 reflect(float3 v, float3 n)
{
    return v - (2.0f * dot<R>(v, n)) * n;
}
__device__ __forceinline__ float3 refract(float3 uv, float3 n, float etai_over_etat) // vec3.cuh refract
{
    const float cos_theta = fminf(dot<rounds::dielectric_cosine>(-uv, n), 1.0f);
    const float3 perp = etai_over_etat * (uv + cos_theta * n);
    const float3 parallel = (-sqrtf(fabsf(1.0f - length_squared(perp)))) * n;
    return perp + parallel;
}
__device__ __forceinline__ float3 f3v(const f3& v) { return make_float3(v.x, v.y, v.z); }
__device__ __forceinline__ float largest_channel(float3 c) { return fmaxf(fmaxf(c.x, c.y), c.z); }
constexpr float pi_f = 3.14159265358979323846f;
constexpr float inverse_pi_f = 0.318309886183790671538f;
constexpr float uniform_sphere_density = 0.0795774715459476678844f; // 1 / (4 pi)
constexpr float infinity_f = __builtin_huge_valf();

// ---- counter-based random numbers (philox.cuh) -------------------------------------------------------------------
// n / d by the divisor's multiplier (fast_divisor), for n < 2^32
__device__ __forceinline__ uint32_t quotient(uint32_t n, const fast_divisor& v)
{
    return v.magic != 0 ? static_cast<uint32_t>(__umul64hi(static_cast<unsigned long long>(n), v.magic)) : n;
}

// A pass's stratum within its round: column s_i = round_pass % sqrt_spp, row s_j = round_pass / sqrt_spp
__device__ __forceinline__ void stratum_of(const camera_params& cam, int round_pass, int& s_i, int& s_j)
{
    s_j = static_cast<int>(quotient(static_cast<uint32_t>(round_pass), cam.div_sqrt_spp));
    s_i = round_pass - s_j * cam.sqrt_spp;
}

// 24 random bits as a float in [0, 1 - 2^-24]: every value k / 2^24 exactly, as random_real<float> (random.cuh:79-93)
__device__ __forceinline__ float to_unit(uint32_t x) { return static_cast<float>(x >> 8) * 0x1p-24f; }

#ifdef RTB_COMPACT_CODE
#define RTB_CALLED __device__ __noinline__
#else
#define RTB_CALLED __device__ __forceinline__
#endif
RTB_CALLED uint4 random_bits(uint4 counter, uint2 key) { return philox4x32_10(counter, key); }

struct sampler
{
    uint2 key;
    uint32_t pixel;
    uint32_t pass;
    uint32_t job;

    // Four 32-bit numbers for dimension block `block` of the vertex at depth `depth` (0: the camera ray)
    __device__ __forceinline__ uint4 draw_bits(int depth, int block) const
    {
        return random_bits(make_uint4(pixel, pass, (static_cast<uint32_t>(depth) << 4) | block, job), key);
    }

    // The same as uniform floats
    __device__ __forceinline__ float4 draw(int depth, int block) const
    {
        const uint4 r = draw_bits(depth, block);
        return make_float4(to_unit(r.x), to_unit(r.y), to_unit(r.z), to_unit(r.w));
    }
};

// The fixed dimension blocks of a vertex: block 0 the material's own sample (direction u0 u1, lobe or mixture
// choice u2, the lights list's pick u3; a books' vertex that aims at the lights list takes the point from u0 u1, which
// its direction then does not use, so a books' vertex draws one block), blocks 2-3 the NEE light sample (the pick, a
// lamp's point or the map's bin bits, coin and cell position), blocks 4-15 the free flights through the volumes of
// smoke, one number per volume. At depth 0, block 0 is the camera ray's (stratum jitter, lens) and block 1's first
// number the ray's time in a scene where something moves.
constexpr int block_material = 0;
constexpr int block_time = 1;
constexpr int block_nee = 2;

// ---- sampling of directions (random.cuh:95-140, material.cuh:55-64) --------------------------------------------
__device__ __forceinline__ float3 random_unit_vector(float u, float v)
{
    float s, c;
    sincospif(2.0f * v, &s, &c);
    const float r = 2.0f * sqrtf(u * (1.0f - u));
    return make_float3(r * c, r * s, 1.0f - 2.0f * u);
}

__device__ __forceinline__ float3 random_cosine_direction(float r1, float r2)
{
    float s, c;
    sincospif(2.0f * r1, &s, &c);
    const float sin_theta = sqrtf(r2);
    return make_float3(c * sin_theta, s * sin_theta, sqrtf(1.0f - r2));
}

// v given in a basis whose z axis is the unit vector n, in world coordinates: the branchless orthonormal basis of
// Duff, Burgess, Christensen, Hery, Kensler, Liani and Villemin, "Building an Orthonormal Basis, Revisited" (JCGT 2017)
__device__ __forceinline__ float3 around(float3 n, float3 v)
{
    const float sign = copysignf(1.0f, n.z);
    const float a = -1.0f / (sign + n.z);
    const float b = n.x * n.y * a;
    const float3 x_axis = make_float3(1.0f + sign * n.x * n.x * a, sign * b, -sign * n.x);
    const float3 y_axis = make_float3(b, sign + n.y * n.y * a, -n.y);
    return v.x * x_axis + v.y * y_axis + v.z * n;
}

__device__ __forceinline__ float cosine_density(float3 unit_normal, float3 direction) // pdf.cuh:21-26
{
    const float cosine = dot(unit_normal, direction) * rsqrtf(length_squared(direction));
    return cosine > 0.0f ? cosine * inverse_pi_f : 0.0f;
}

// Schlick's reflectance (material.cuh:67-76)
__device__ __forceinline__ float reflectance(float cosine, float ri)
{
    float r0 = (1.0f - ri) / (1.0f + ri);
    r0 = r0 * r0;
    const float x = 1.0f - cosine;
    const float x2 = x * x;
    return r0 + (1.0f - r0) * (x2 * x2 * x);
}

// ---- primitive tests ------------------------------------------------------------------------------------------
// 1 / x, never infinite (bvh.cuh:475-488): |x| below 2^-80 moves out to +-2^-80
__device__ __forceinline__ float safe_inverse(float x)
{
    const float tiny = 0x1p-80f;
    return 1.0f / (fabsf(x) > tiny ? x : copysignf(tiny, x));
}

// A large sphere's dot products, written out where the others are (a last bit of a double moves the float distance it is
// rounded to in one hit of some ten million)
__device__ __forceinline__ double dot_double(double ax, double ay, double az, double bx, double by, double bz)
{
    return rounds::other == rounding::compiler ? ax * bx + ay * by + az * bz
                                               : __fma_rn(az, bz, __fma_rn(ax, bx, __dmul_rn(ay, by)));
}

// A large sphere's (negative radius): the same quadratic in FP64, where FP32's 24 bits cancel on its scale
RTB_CALLED bool sphere_roots_double(float4 s, float3 o, float3 d, float& near, float& far)
{
    const double r = -static_cast<double>(s.w);
    const double ox = static_cast<double>(s.x) - o.x;
    const double oy = static_cast<double>(s.y) - o.y;
    const double oz = static_cast<double>(s.z) - o.z;
    const double dx = d.x, dy = d.y, dz = d.z;
    const double ia = 1.0 / dot_double(dx, dy, dz, dx, dy, dz);
    const double hoa = dot_double(dx, dy, dz, ox, oy, oz) * ia;
    const double lx = ox - hoa * dx, ly = oy - hoa * dy, lz = oz - hoa * dz;
    const double disc = fma(-lx, lx, fma(-ly, ly, fma(-lz, lz, r * r)));
    if (disc < 0.0)
    {
        return false;
    }
    const double half_chord = sqrt(disc * ia);
    if constexpr (rounds::other == rounding::compiler)
    {
        near = static_cast<float>(hoa - half_chord);
        far = static_cast<float>(hoa + half_chord);
    }
    else
    {
        near = static_cast<float>(__dadd_rn(hoa, -half_chord));
        far = static_cast<float>(__dadd_rn(hoa, half_chord));
    }
    return true;
}

// The two roots of the line with a sphere, as (h/a) -+ sqrt(r^2 - |l|^2)/sqrt(a) with l the vector from the line's
// closest point to the center (sphere.cuh:70-97, after Haines et al., Ray Tracing Gems ch. 7): nothing larger than
// r^2 is subtracted, and the three squares go into r^2 through fused multiply-adds.
__device__ __forceinline__ bool sphere_roots(float4 s, float3 o, float3 d, float inverse_a, float& near, float& far)
{
    if (s.w >= 0.0f)
    {
        const float3 oc = make_float3(s.x - o.x, s.y - o.y, s.z - o.z);
        const float h_over_a = dot(d, oc) * inverse_a;
        const float3 l = oc - h_over_a * d;
        const float disc = fmaf(-l.x, l.x, fmaf(-l.y, l.y, fmaf(-l.z, l.z, s.w * s.w)));
        if (disc < 0.0f)
        {
            return false;
        }
        const float half_chord = sqrtf(disc * inverse_a);
        if constexpr (rounds::other == rounding::compiler)
        {
            near = h_over_a - half_chord;
            far = h_over_a + half_chord;
        }
        else // not fused with h_over_a's product (a volume's boundary and its glass must meet at one distance)
        {
            near = __fadd_rn(h_over_a, -half_chord);
            far = __fadd_rn(h_over_a, half_chord);
        }
        return true;
    }
    return sphere_roots_double(s, o, d, near, far);
}

// hit_sphere (sphere.cuh:99-117): the nearest root in (t_min, t_max); far_only for the sphere the ray leaves inward
__device__ __forceinline__ bool hit_sphere(float4 s, float3 o, float3 d, float inverse_a, float t_min, float t_max,
                                           bool far_only, float& t, bool& entering)
{
    float near, far;
    if (!sphere_roots(s, o, d, inverse_a, near, far))
    {
        return false;
    }
    t = near;
    entering = !far_only && t > t_min;
    if (!entering)
    {
        t = far;
    }
    return t_min < t && t < t_max;
}

struct quad_v
{
    float3 q, n, a, b;
};

__device__ __forceinline__ quad_v load_quad(const quad12* quads, int i)
{
    const float4* p = reinterpret_cast<const float4*>(quads + i);
    const float4 a = __ldg(p);
    const float4 b = __ldg(p + 1);
    const float4 c = __ldg(p + 2);
    return {make_float3(a.x, a.y, a.z), make_float3(a.w, b.x, b.y), make_float3(b.z, b.w, c.x),
            make_float3(c.y, c.z, c.w)};
}

// hit_quad (quad.cuh:60-84): t in [t_min, t_max] and alpha, beta in [0, 1], closed; the corner taken relative to the
// origin first. NaNs fail every comparison (a degenerate quad stays invisible).
__device__ __forceinline__ bool hit_quad(const quad_v& s, float3 o, float3 d, float t_min, float t_max, float& t,
                                         bool& front)
{
    const float denominator = dot(s.n, d);
    if (!(fabsf(denominator) >= 1e-8f))
    {
        return false;
    }
    const float3 origin_to_q = s.q - o;
    t = dot(s.n, origin_to_q) / denominator;
    if (!(t_min <= t && t <= t_max))
    {
        return false;
    }
    const float3 p = t * d - origin_to_q;
    const float alpha = dot(p, s.a);
    const float beta = dot(p, s.b);
    if (!(0.0f <= alpha && alpha <= 1.0f && 0.0f <= beta && beta <= 1.0f))
    {
        return false;
    }
    front = denominator < 0.0f;
    return true;
}

struct triangle_v
{
    float3 a, b, c;
};

__device__ __forceinline__ triangle_v load_triangle(const triangle12* tris, int i)
{
    const float4* p = reinterpret_cast<const float4*>(tris + i);
    const float4 a = __ldg(p);
    const float4 b = __ldg(p + 1);
    const float4 c = __ldg(p + 2);
    return {make_float3(a.x, a.y, a.z), make_float3(a.w, b.x, b.y), make_float3(b.z, b.w, c.x)};
}

__device__ __forceinline__ float axis_of(float3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

// A ray's shear for the watertight triangle test: the axis along which the direction is largest (z after the
// permutation, the other two swapped when it points backwards so the winding is kept), and the shear that makes the
// direction (0, 0, 1). Computed once per leaf; the same floats for every triangle the ray meets.
struct ray_shear
{
    int kx, ky, kz;
    float sx, sy, sz;
};

__device__ __forceinline__ ray_shear shear_of(float3 d)
{
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    ray_shear r;
    r.kz = ax > ay ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    r.kx = r.kz == 2 ? 0 : r.kz + 1;
    r.ky = r.kx == 2 ? 0 : r.kx + 1;
    const float dz = axis_of(d, r.kz);
    if (dz < 0.0f)
    {
        const int k = r.kx;
        r.kx = r.ky;
        r.ky = k;
    }
    r.sz = 1.0f / dz;
    r.sx = axis_of(d, r.kx) * r.sz;
    r.sy = axis_of(d, r.ky) * r.sz;
    return r;
}

// The signed area of an edge seen along the sheared ray, rounded so that the same edge walked the other way by the
// neighbouring triangle gives exactly the opposite number (no fused multiply-add), and in double when it comes out 0
__device__ __forceinline__ float edge_function(float px, float py, float qx, float qy)
{
    const float e = __fsub_rn(__fmul_rn(px, qy), __fmul_rn(py, qx));
    if (e != 0.0f)
    {
        return e;
    }
    return static_cast<float>(static_cast<double>(px) * qy - static_cast<double>(py) * qx);
}

// The same test in double, for a ray whose float edge functions are too close to 0 to be sure of their signs: one
// grazing the triangle (its projection a sliver) or passing within rounding of an edge
__device__ __noinline__ bool hit_triangle_double(const triangle_v& tr, const ray_shear& r, float3 o, float3 d,
                                                 float t_min, float t_max, float& t, bool& front)
{
    const double ox = o.x, oy = o.y, oz = o.z;
    const double rel[3][3] = {{tr.a.x - ox, tr.a.y - oy, tr.a.z - oz},
                              {tr.b.x - ox, tr.b.y - oy, tr.b.z - oz},
                              {tr.c.x - ox, tr.c.y - oy, tr.c.z - oz}};
    const double dir[3] = {d.x, d.y, d.z};
    const double sz = 1.0 / dir[r.kz];
    const double sx = dir[r.kx] * sz, sy = dir[r.ky] * sz;
    double px[3], py[3], pz[3];
    for (int k = 0; k < 3; ++k)
    {
        pz[k] = rel[k][r.kz];
        px[k] = rel[k][r.kx] - sx * pz[k];
        py[k] = rel[k][r.ky] - sy * pz[k];
    }
    const double u = px[2] * py[1] - py[2] * px[1];
    const double v = px[0] * py[2] - py[0] * px[2];
    const double w = px[1] * py[0] - py[1] * px[0];
    if ((u < 0.0 || v < 0.0 || w < 0.0) && (u > 0.0 || v > 0.0 || w > 0.0))
    {
        return false;
    }
    const double det = u + v + w;
    if (det == 0.0)
    {
        return false;
    }
    const double tt = (u * pz[0] + v * pz[1] + w * pz[2]) * sz / det;
    t = static_cast<float>(tt);
    if (!(t_min < t && t < t_max))
    {
        return false;
    }
    front = dot(d, cross(tr.b - tr.a, tr.c - tr.a)) < 0.0f;
    return true;
}

__device__ __forceinline__ float max_abs(float3 v) { return fmaxf(fabsf(v.x), fmaxf(fabsf(v.y), fabsf(v.z))); }

// Woop, Benthin and Wald, "Watertight Ray/Triangle Intersection" (JCGT 2013): the triangle's vertices sheared into
// the ray's frame, the three edge functions of the origin's projection, all of one sign; so a ray through an edge or a
// vertex shared by triangles hits at least one of them, with no crack between (Möller-Trumbore in float lets such a
// ray through both, about 4 rays in a million on the 1.3M-triangle mesh). An edge function within its float rounding
// of 0 (a grazing ray, or one within rounding of an edge) sends the test to double. Barycentrics closed, t open. The
// front is the side (b - a) x (c - a) points to.
__device__ __forceinline__ bool hit_triangle(const triangle_v& tr, const ray_shear& r, float3 o, float3 d,
                                             float t_min, float t_max, float& t, bool& front)
{
    const float3 pa = tr.a - o, pb = tr.b - o, pc = tr.c - o;
    const float az = axis_of(pa, r.kz), bz = axis_of(pb, r.kz), cz = axis_of(pc, r.kz);
    const float ax = axis_of(pa, r.kx) - r.sx * az, ay = axis_of(pa, r.ky) - r.sy * az;
    const float bx = axis_of(pb, r.kx) - r.sx * bz, by = axis_of(pb, r.ky) - r.sy * bz;
    const float cx = axis_of(pc, r.kx) - r.sx * cz, cy = axis_of(pc, r.ky) - r.sy * cz;
    const float u = edge_function(cx, cy, bx, by);
    const float v = edge_function(ax, ay, cx, cy);
    const float w = edge_function(bx, by, ax, ay);
    // The edge functions' rounding: the shear's (a few units of the vertices' largest coordinate's last place) times
    // the projected coordinates' size, with a margin
    const float coords = fmaxf(max_abs(pa), fmaxf(max_abs(pb), max_abs(pc)));
    const float sheared = fmaxf(fmaxf(fmaxf(fabsf(ax), fabsf(ay)), fmaxf(fabsf(bx), fabsf(by))),
                                fmaxf(fabsf(cx), fabsf(cy)));
    const float rounding = 5e-7f * coords * sheared;
    if (fabsf(u) <= rounding || fabsf(v) <= rounding || fabsf(w) <= rounding)
    {
        return hit_triangle_double(tr, r, o, d, t_min, t_max, t, front);
    }
    if ((u < 0.0f || v < 0.0f || w < 0.0f) && (u > 0.0f || v > 0.0f || w > 0.0f))
    {
        return false;
    }
    const float det = u + v + w;
    if (det == 0.0f)
    {
        return false;
    }
    const float depth = u * (r.sz * az) + v * (r.sz * bz) + w * (r.sz * cz);
    t = depth / det;
    if (!(t_min < t && t < t_max))
    {
        return false;
    }
    front = dot(d, cross(tr.b - tr.a, tr.c - tr.a)) < 0.0f;
    return true;
}

// ---- traversal ------------------------------------------------------------------------------------------------
struct hit_info
{
    int id;     // global id, -1 for none
    float t;
    bool front; // the near root of a sphere, the front of a quad or a triangle
};

constexpr float t_min = 0.001f;

// What one traversal fetched, for the counting build (the roofline's algorithmic bytes); compiled away otherwise
struct fetch_counts
{
    uint32_t nodes = 0;
    uint32_t spheres = 0;
    uint32_t quads = 0;
    uint32_t triangles = 0;
};

// Sphere i (leaf order) where it is at the ray's time: its center moved by time * displacement in a scene where
// something moves (moving_sphere::at, sphere.cuh)
// FEATURES (here and below): the code of the second book's features (moving spheres, textures, smoke) is compiled in;
// the render kernels of scenes without them are compiled with FEATURES = false and keep none of its registers
template <bool FEATURES = true>
__device__ __forceinline__ float4 sphere_at(const scene_view& S, int i, float time)
{
    float4 s = __ldg(reinterpret_cast<const float4*>(S.spheres + i));
    if (FEATURES && S.has_motion)
    {
        const float4 m = __ldg(S.sphere_motion + i);
        s.x = fmaf(time, m.x, s.x);
        s.y = fmaf(time, m.y, s.y);
        s.z = fmaf(time, m.z, s.z);
    }
    return s;
}

// The leaf's primitives against the ray, shrinking hit.t; true at the first hit for a shadow ray (SHADOW, or `any`
// for a kernel that walks both kinds of ray)
template <bool SHADOW, bool COUNT, bool FEATURES>
__device__ __forceinline__ bool test_leaf(const scene_view& S, int link, float3 o, float3 d, float time,
                                          float inverse_a, int from, bool inward, int skip, hit_info& hit,
                                          fetch_counts* counts, bool any = false)
{
    const int kind = leaf_kind(link);
    const int count = leaf_count(link);
    const int start = leaf_start(link);
    if (COUNT)
    {
        (kind == kind_sphere ? counts->spheres : kind == kind_quad ? counts->quads : counts->triangles) += count;
    }
    if (kind == kind_sphere)
    {
        for (int i = start; i < start + count; ++i)
        {
            const int id = i; // spheres' global ids are their indices
            const bool own = id == from;
            if ((own && !inward) || id == skip)
            {
                continue;
            }
            const float4 s = sphere_at<FEATURES>(S, i, time);
            float t;
            bool entering;
            if (hit_sphere(s, o, d, inverse_a, t_min, hit.t, own, t, entering))
            {
                if (SHADOW || any)
                {
                    return true;
                }
                hit = {id, t, entering};
            }
        }
    }
    else if (kind == kind_quad)
    {
        for (int i = start; i < start + count; ++i)
        {
            const int id = S.quad_base + i;
            if (id == from || id == skip)
            {
                continue;
            }
            const quad_v q = load_quad(S.quads, i);
            float t;
            bool front;
            if (hit_quad(q, o, d, t_min, hit.t, t, front))
            {
                if (SHADOW || any)
                {
                    return true;
                }
                hit = {id, t, front};
            }
        }
    }
    else
    {
        const ray_shear shear = shear_of(d);
        for (int i = start; i < start + count; ++i)
        {
            const int id = S.triangle_base + i;
            if (id == from || id == skip)
            {
                continue;
            }
            const triangle_v tr = load_triangle(S.triangles, i);
            float t;
            bool front;
            if (hit_triangle(tr, shear, o, d, t_min, hit.t, t, front))
            {
                if (SHADOW || any)
                {
                    return true;
                }
                hit = {id, t, front};
            }
        }
    }
    return false;
}

// No more nodes to visit (a leaf link never takes this value: its kind field would be 3)
constexpr int traversal_done = traversal_done_link;

// The closest hit in (t_min, t_max) (SHADOW = false; the CPU's world.hit, bvh.cuh:576-706), or whether anything lies
// there (SHADOW = true; shadow.cuh:26-109 occluded, `skip` not tested). The self-intersection rules of the primitive
// the ray leaves, `from`: a quad or a triangle is never hit again (a line meets a plane once); a sphere left outward
// is never hit again, and left inward only at its far root (bvh.cuh:539-575).
//
// The loop is Aila and Laine's speculative while-while (HPG 2009): a lane descends through inner nodes, sets aside the
// first leaf it meets and keeps descending, and the warp leaves the node loop together once every lane holds a leaf;
// then the leaf loop tests them. Node steps and leaf tests so run with the warp's lanes side by side, where a single
// loop would run a node step for some lanes and a leaf test for the others one after the other.
//
// SEARCH: search_any follows the scene's `flat`; search_flat and search_tree compile one of the two searches alone
// (a kernel specialised for one of them keeps no code, registers or stack for the other).
constexpr int search_any = 0;
constexpr int search_flat = 1;
constexpr int search_tree = 2;

template <bool SHADOW, bool COUNT = false, int SEARCH = search_any, bool FEATURES = true>
__device__ __forceinline__ bool traverse(const scene_view& S, float3 o, float3 d, float time, float t_max, int from,
                                         bool inward, int skip, hit_info& hit, fetch_counts* counts = nullptr)
{
    hit.id = -1;
    hit.t = t_max;
    hit.front = false;
    if (S.node_count == 0)
    {
        return false;
    }
    const float inverse_a = 1.0f / length_squared(d);
    if (SEARCH == search_flat || (SEARCH == search_any && S.flat))
    {
        // A small scene of spheres and quads: every primitive tested in order, no tree. The warp's lanes run the same
        // loop over the same records (one broadcast load each), where a tree walk would split them up.
        for (int i = 0; i < S.quad_base; ++i)
        {
            const bool own = i == from;
            if ((own && !inward) || i == skip)
            {
                continue;
            }
            const float4 s = sphere_at<FEATURES>(S, i, time);
            float t;
            bool entering;
            if (hit_sphere(s, o, d, inverse_a, t_min, hit.t, own, t, entering))
            {
                if (SHADOW)
                {
                    return true;
                }
                hit = {i, t, entering};
            }
        }
        const int quads = S.triangle_base - S.quad_base;
        for (int i = 0; i < quads; ++i)
        {
            const int id = S.quad_base + i;
            if (id == from || id == skip)
            {
                continue;
            }
            float t;
            bool front;
            if (hit_quad(load_quad(S.quads, i), o, d, t_min, hit.t, t, front))
            {
                if (SHADOW)
                {
                    return true;
                }
                hit = {id, t, front};
            }
        }
        if (COUNT)
        {
            counts->spheres += S.quad_base;
            counts->quads += quads;
        }
        return hit.id >= 0;
    }
    const float3 inv = make_float3(safe_inverse(d.x), safe_inverse(d.y), safe_inverse(d.z));
    const float3 os = make_float3(o.x * inv.x, o.y * inv.y, o.z * inv.z);
    int2 stack[max_bvh_depth];
    int sp = 0;
    // The next stack entry the ray enters before the closest hit so far, or traversal_done
    const auto pop = [&]() -> int {
        while (sp > 0)
        {
            const int2 e = stack[--sp];
            if (SHADOW || __int_as_float(e.y) < hit.t)
            {
                return e.x;
            }
        }
        return traversal_done;
    };
    int link = 0;
    int leaf = 0; // a leaf set aside (leaf links are negative; 0: none)
    while (link != traversal_done)
    {
        while (link >= 0)
        {
            const float4* np = reinterpret_cast<const float4*>(S.nodes + link);
            const float4 nx = __ldg(np);
            const float4 ny = __ldg(np + 1);
            const float4 nz = __ldg(np + 2);
            const int2 nl = __ldg(reinterpret_cast<const int2*>(np + 3));
            if (COUNT)
            {
                ++counts->nodes;
            }
            const float a0 = fmaf(nx.x, inv.x, -os.x), a1 = fmaf(nx.y, inv.x, -os.x);
            const float b0 = fmaf(ny.x, inv.y, -os.y), b1 = fmaf(ny.y, inv.y, -os.y);
            const float c0 = fmaf(nz.x, inv.z, -os.z), c1 = fmaf(nz.y, inv.z, -os.z);
            const float enter0 = fmaxf(fmaxf(fminf(a0, a1), fminf(b0, b1)), fmaxf(fminf(c0, c1), t_min));
            const float exit0 = fminf(fminf(fmaxf(a0, a1), fmaxf(b0, b1)), fminf(fmaxf(c0, c1), hit.t));
            const float a2 = fmaf(nx.z, inv.x, -os.x), a3 = fmaf(nx.w, inv.x, -os.x);
            const float b2 = fmaf(ny.z, inv.y, -os.y), b3 = fmaf(ny.w, inv.y, -os.y);
            const float c2 = fmaf(nz.z, inv.z, -os.z), c3 = fmaf(nz.w, inv.z, -os.z);
            const float enter1 = fmaxf(fmaxf(fminf(a2, a3), fminf(b2, b3)), fmaxf(fminf(c2, c3), t_min));
            const float exit1 = fminf(fminf(fmaxf(a2, a3), fmaxf(b2, b3)), fminf(fmaxf(c2, c3), hit.t));
            const bool h0 = enter0 <= exit0;
            const bool h1 = enter1 <= exit1;
            if (h0 && h1)
            {
                const bool second_first = enter1 < enter0;
                link = second_first ? nl.y : nl.x;
                stack[sp++] = make_int2(second_first ? nl.x : nl.y, __float_as_int(second_first ? enter0 : enter1));
            }
            else if (h0 || h1)
            {
                link = h0 ? nl.x : nl.y;
            }
            else
            {
                link = pop();
            }
            // A leaf: set it aside and go on descending, unless one is already waiting
            if (link < 0 && link != traversal_done && leaf == 0)
            {
                leaf = link;
                link = pop();
            }
            if (!__any_sync(__activemask(), leaf == 0))
            {
                break; // every lane of the warp holds a leaf: test them together
            }
        }
        while (leaf < 0)
        {
            if (test_leaf<SHADOW, COUNT, FEATURES>(S, leaf, o, d, time, inverse_a, from, inward, skip, hit, counts))
            {
                return true;
            }
            leaf = 0;
            if (link < 0 && link != traversal_done)
            {
                leaf = link;
                link = pop();
            }
        }
    }
    return hit.id >= 0;
}

// ---- the walk of the tree four wide ----------------------------------------------------------------------------
// A ray as the wide nodes are tested: the direction's reciprocals, the origin times them, and where the near bounds of
// an axis lie in a node (lo_x, hi_x, lo_y, ...: the low or the high row by the direction's sign; the far ones 16 bytes
// off), instead of a minimum and a maximum of both: the same numbers, since a multiply-add is monotonic
struct wide_ray
{
    float3 inv, os;
    uint32_t x, y, z;
};

__device__ __forceinline__ wide_ray wide_ray_of(float3 o, float3 d)
{
    wide_ray r;
    r.inv = make_float3(safe_inverse(d.x), safe_inverse(d.y), safe_inverse(d.z));
    r.os = make_float3(o.x * r.inv.x, o.y * r.inv.y, o.z * r.inv.z);
    r.x = r.inv.x < 0.0f ? 16u : 0u;
    r.y = r.inv.y < 0.0f ? 48u : 32u;
    r.z = r.inv.z < 0.0f ? 80u : 64u;
    return r;
}

// One inner node: its children that the ray enters before `limit`, the nearest returned, the others pushed on the
// stack, farthest deepest (pop() where it enters none)
template <class Pop>
__device__ __forceinline__ int wide_step(const bvh4_node* tree, int link, const wide_ray& r, float limit, int2* stack,
                                         int& sp, const Pop& pop)
{
    const char* const node = reinterpret_cast<const char*>(tree + link);
    const auto row = [&](uint32_t at) { return __ldg(reinterpret_cast<const float4*>(node + at)); };
    const float4 nx = row(r.x), fx = row(r.x ^ 16u);
    const float4 ny = row(r.y), fy = row(r.y ^ 16u);
    const float4 nz = row(r.z), fz = row(r.z ^ 16u);
    const int4 nl = __ldg(reinterpret_cast<const int4*>(tree[link].link));
    // each child's entry distance, or infinity where the ray misses it (or the slot is unused)
    const auto entry = [&](float ax, float bx, float ay, float by, float az, float bz, int child) -> float {
        const float enter = fmaxf(fmaxf(fmaf(ax, r.inv.x, -r.os.x), fmaf(ay, r.inv.y, -r.os.y)),
                                  fmaxf(fmaf(az, r.inv.z, -r.os.z), t_min));
        const float exit = fminf(fminf(fmaf(bx, r.inv.x, -r.os.x), fmaf(by, r.inv.y, -r.os.y)),
                                 fminf(fmaf(bz, r.inv.z, -r.os.z), limit));
        return enter <= exit && child != traversal_done ? enter : infinity_f;
    };
    float k0 = entry(nx.x, fx.x, ny.x, fy.x, nz.x, fz.x, nl.x);
    float k1 = entry(nx.y, fx.y, ny.y, fy.y, nz.y, fz.y, nl.y);
    float k2 = entry(nx.z, fx.z, ny.z, fy.z, nz.z, fz.z, nl.z);
    float k3 = entry(nx.w, fx.w, ny.w, fy.w, nz.w, fz.w, nl.w);
    int l0 = nl.x, l1 = nl.y, l2 = nl.z, l3 = nl.w;
    const auto order = [](float& ka, int& la, float& kb, int& lb) {
        if (kb < ka)
        {
            const float k = ka;
            ka = kb;
            kb = k;
            const int l = la;
            la = lb;
            lb = l;
        }
    };
    order(k0, l0, k1, l1);
    order(k2, l2, k3, l3);
    order(k0, l0, k2, l2);
    order(k1, l1, k3, l3);
    order(k1, l1, k2, l2);
    if (k0 == infinity_f)
    {
        return pop();
    }
    if (k3 != infinity_f)
    {
        stack[sp++] = make_int2(l3, __float_as_int(k3));
    }
    if (k2 != infinity_f)
    {
        stack[sp++] = make_int2(l2, __float_as_int(k2));
    }
    if (k1 != infinity_f)
    {
        stack[sp++] = make_int2(l1, __float_as_int(k1));
    }
    return l0;
}

// The closest hit as the walk of the binary tree meets it, called: a query's rare second walk
__device__ __noinline__ void closest_hit_binary(const scene_view& S, float3 o, float3 d, hit_info& hit)
{
    traverse<false, false, search_tree>(S, o, d, 0.0f, infinity_f, -1, false, -1, hit);
}

// The closest hit of one ray per lane (a query of rays that do not follow from one another): the walk's inner nodes and
// leaves by turns, each lane through the whole of its walk. Which of several primitives at one distance (two quads in a
// plane, a mesh's shared edge, a sphere twice in the scene) is the hit follows from the order of the walk, and the order
// of a query's is the binary tree's: a ray that meets a second primitive as near as the nearest to within the boxes' and
// the distances' rounding walks that tree. (The nodes' entries are off by some 2^-24 of the origin times the direction's
// reciprocal; an axis the ray hardly moves along decides no entry near a hit.)
__device__ __forceinline__ void closest_hit_wide(const scene_view& S, float3 o, float3 d, hit_info& hit)
{
    hit = {-1, infinity_f, false};
    const float inverse_a = 1.0f / length_squared(d);
    const wide_ray ray = wide_ray_of(o, d);
    const float steepest = fminf(fminf(fabsf(ray.inv.x), fabsf(ray.inv.y)), fabsf(ray.inv.z));
    const auto reach = [&](float inv, float os) { return fabsf(inv) <= 1024.0f * steepest ? fabsf(os) : 0.0f; };
    const float origin = fmaxf(fmaxf(reach(ray.inv.x, ray.os.x), reach(ray.inv.y, ray.os.y)), reach(ray.inv.z, ray.os.z));
    float as_near = 0.0f; // what lies within this of the closest hit may be as near
    float bound = infinity_f;
    bool tied = false;
    int2 stack[wide_stack];
    int sp = 0;
    int link = 0;
    const auto pop = [&]() -> int {
        while (sp > 0)
        {
            const int2 e = stack[--sp];
            if (__int_as_float(e.y) < bound)
            {
                return e.x;
            }
        }
        return traversal_done;
    };
    while (link != traversal_done)
    {
        while (link >= 0)
        {
            link = wide_step(S.wide_nodes, link, ray, bound, stack, sp, pop);
        }
        if (link != traversal_done)
        {
            // the leaf's own closest hit (its primitives are tested in one order by either walk)
            hit_info found{-1, bound, false};
            test_leaf<false, false, true>(S, link, o, d, 0.0f, inverse_a, -1, false, -1, found, nullptr);
            if (found.id >= 0)
            {
                tied = hit.id >= 0 && found.t >= hit.t - as_near;
                if (hit.id < 0 || found.t < hit.t)
                {
                    hit = found;
                    as_near = 0x1p-18f * (hit.t + origin);
                    bound = hit.t + as_near;
                }
            }
            link = pop();
        }
    }
    if (tied)
    {
        closest_hit_binary(S, o, d, hit);
    }
}

// ---- volumes of smoke (constant_medium.cuh:29-120, camera.cuh:259-284, shadow.cuh:129-165) -------------------------
constexpr int block_media = 4; // max_media volumes: one number each from blocks 4-15 of a vertex

// Where the ray's line crosses the medium's boundary: the sphere's two roots, the sphere where it is at the ray's time,
// kept only if the chord is longer than 0.0001; or the nearest and the farthest plane of the boundary quads the line
// meets inside them
__device__ bool boundary_crossings(const scene_view& S, const medium16& m, float3 o, float3 d, float time,
                                   float inverse_a, float& t_in, float& t_out)
{
    if (m.quad_count == 0)
    {
        const float4 s = make_float4(fmaf(time, m.dx, m.cx), fmaf(time, m.dy, m.cy), fmaf(time, m.dz, m.cz), m.radius);
        return sphere_roots(s, o, d, inverse_a, t_in, t_out) && t_out - t_in > 0.0001f;
    }
    t_in = infinity_f;
    t_out = -infinity_f;
    for (int i = m.first_quad; i < m.first_quad + m.quad_count; ++i)
    {
        float t;
        bool front;
        if (hit_quad(load_quad(S.boundary_quads, i), o, d, -infinity_f, infinity_f, t, front))
        {
            t_in = fminf(t_in, t);
            t_out = fmaxf(t_out, t);
        }
    }
    return t_out - t_in >= 0.0001f;
}

// The stretch [t_in, t_out] of (t_min, t_max) that lies inside the medium, or false: its box first (a ray that misses
// the box misses the volume), then the boundary's crossings
__device__ __forceinline__ bool medium_stretch(const scene_view& S, const medium16& m, float3 o, float3 d, float time,
                                               float inverse_a, float3 inv, float3 os, float t_max, float& t_in,
                                               float& t_out)
{
    const float a0 = fmaf(m.lo_x, inv.x, -os.x), a1 = fmaf(m.hi_x, inv.x, -os.x);
    const float b0 = fmaf(m.lo_y, inv.y, -os.y), b1 = fmaf(m.hi_y, inv.y, -os.y);
    const float c0 = fmaf(m.lo_z, inv.z, -os.z), c1 = fmaf(m.hi_z, inv.z, -os.z);
    const float enter = fmaxf(fmaxf(fminf(a0, a1), fminf(b0, b1)), fmaxf(fminf(c0, c1), t_min));
    const float exit = fminf(fminf(fmaxf(a0, a1), fmaxf(b0, b1)), fminf(fmaxf(c0, c1), t_max));
    if (!(enter <= exit))
    {
        return false;
    }
    float line_in, line_out;
    if (!boundary_crossings(S, m, o, d, time, inverse_a, line_in, line_out))
    {
        return false;
    }
    t_in = fmaxf(line_in, t_min);
    t_out = fminf(line_out, t_max);
    if (!(t_in < t_out))
    {
        return false;
    }
    t_in = fmaxf(t_in, 0.0f);
    return true;
}

// What the ray meets first: the closest surface `hit`, or a particle of smoke in front of it (closest_event,
// camera.cuh:259-284). Each volume, in the list's order, against the closest event so far: a free flight of
// -log(u) / density from where the ray enters it (medium_collision, constant_medium.cuh:86-120), u drawn from the
// vertex's media blocks.
// (Like transmittance and texture_value: only the kernels of scenes with these features call them, so they are
// inlined there; measured 5-10% faster on the second book's scenes than as calls.)
#define RTB_FEATURE_FUNCTION __device__ __forceinline__
RTB_FEATURE_FUNCTION void media_event(const scene_view& S, float3 o, float3 d, float time, const sampler& rng,
                                      int depth,
                            hit_info& hit)
{
    const float inverse_a = 1.0f / length_squared<rounds::flight>(d);
    const float3 inv = make_float3(safe_inverse(d.x), safe_inverse(d.y), safe_inverse(d.z));
    const float3 os = make_float3(o.x * inv.x, o.y * inv.y, o.z * inv.z);
    const float length = sqrtf(length_squared<rounds::flight>(d));
    float4 u = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int k = 0; k < S.medium_count; ++k)
    {
        if ((k & 3) == 0)
        {
            u = rng.draw(depth, block_media + (k >> 2));
        }
        const medium16 m = S.media[k];
        float t_in, t_out;
        if (!medium_stretch(S, m, o, d, time, inverse_a, inv, os, hit.t, t_in, t_out))
        {
            continue;
        }
        const float uk = (k & 3) == 0 ? u.x : (k & 3) == 1 ? u.y : (k & 3) == 2 ? u.z : u.w;
        const float distance = m.neg_inv_density * logf(uk);
        if (distance > (t_out - t_in) * length)
        {
            continue; // through without meeting a particle
        }
        hit = {S.medium_base + k, t_in + distance / length, true};
    }
}

// The chance that (t_min, t_max) of the ray crosses every volume without meeting a particle: the expected value of
// media_event's free-flight test over exactly the stretch it would test (transmittance, shadow.cuh:129-165)
RTB_FEATURE_FUNCTION float transmittance(const scene_view& S, float3 o, float3 d, float time, float t_max)
{
    const float inverse_a = 1.0f / length_squared(d);
    const float3 inv = make_float3(safe_inverse(d.x), safe_inverse(d.y), safe_inverse(d.z));
    const float3 os = make_float3(o.x * inv.x, o.y * inv.y, o.z * inv.z);
    const float length = sqrtf(length_squared(d));
    float exponent = 0.0f;
    for (int k = 0; k < S.medium_count; ++k)
    {
        const medium16 m = S.media[k];
        float t_in, t_out;
        if (medium_stretch(S, m, o, d, time, inverse_a, inv, os, t_max, t_in, t_out))
        {
            exponent += (t_out - t_in) * length / m.neg_inv_density;
        }
    }
    return expf(exponent);
}

// ---- textures (texture.cuh, perlin.cuh: the books' solid, checker, image and marble textures) ------------------
// Perlin noise with Hermite smoothing of the cell's coordinates and the trilinear sum of the eight corners'
// gradient dot products (perlin.ixx noise); turbulence: 7 octaves of it, each at twice the frequency and half the
// weight, absolute value
__device__ float perlin_noise(const noise_table& n, float3 p)
{
    const float fx = floorf(p.x), fy = floorf(p.y), fz = floorf(p.z);
    const int i = static_cast<int>(fx), j = static_cast<int>(fy), k = static_cast<int>(fz);
    const float u = p.x - fx, v = p.y - fy, w = p.z - fz;
    const float uu = u * u * (3.0f - 2.0f * u);
    const float vv = v * v * (3.0f - 2.0f * v);
    const float ww = w * w * (3.0f - 2.0f * w);
    float accum = 0.0f;
#pragma unroll
    for (int di = 0; di < 2; ++di)
    {
        const int px = n.perm_x[(i + di) & 255];
        const float wx = di == 0 ? 1.0f - uu : uu;
#pragma unroll
        for (int dj = 0; dj < 2; ++dj)
        {
            const int py = n.perm_y[(j + dj) & 255];
            const float wy = dj == 0 ? 1.0f - vv : vv;
#pragma unroll
            for (int dk = 0; dk < 2; ++dk)
            {
                const int pz = n.perm_z[(k + dk) & 255];
                const float wz = dk == 0 ? 1.0f - ww : ww;
                const float4 g = n.gradients[px ^ py ^ pz];
                const float dot_g = g.x * (u - static_cast<float>(di)) + g.y * (v - static_cast<float>(dj)) +
                                    g.z * (w - static_cast<float>(dk));
                accum += wx * wy * wz * dot_g;
            }
        }
    }
    return accum;
}

__device__ float turbulence(const noise_table& n, float3 p)
{
    float accum = 0.0f;
    float weight = 1.0f;
    for (int layer = 0; layer < 7; ++layer)
    {
        accum += weight * perlin_noise(n, p);
        weight *= 0.5f;
        p = 2.0f * p;
    }
    return fabsf(accum);
}

// The texture's color at the hit (texture_value, texture.cuh:60-110): a checker is walked down to the texture of the
// point's cube (its textures come before it, so the walk ends); an image is read at (u, v) clamped to [0, 1], v
// flipped, the pixel they fall in; a marble is 0.5 (1 + sin(scale z + 10 turbulence(p))) in every channel
RTB_FEATURE_FUNCTION float3 texture_value(const scene_view& S, int index, float u, float v, float3 p)
{
    texture8 t = S.textures[index];
    while (t.kind == RT_TEXTURE_CHECKER)
    {
        const int x = static_cast<int>(floorf(t.inv_scale * p.x));
        const int y = static_cast<int>(floorf(t.inv_scale * p.y));
        const int z = static_cast<int>(floorf(t.inv_scale * p.z));
        t = S.textures[(x + y + z) % 2 == 0 ? t.even : t.odd];
    }
    if (t.kind == RT_TEXTURE_IMAGE)
    {
        const image_info im = S.images[t.table];
        const float cu = fminf(fmaxf(u, 0.0f), 1.0f);
        const float fv = 1.0f - fminf(fmaxf(v, 0.0f), 1.0f);
        const int column = static_cast<int>(cu * static_cast<float>(im.width));
        const int row = static_cast<int>(fv * static_cast<float>(im.height));
        const int i = column < im.width - 1 ? column : im.width - 1;
        const int j = row < im.height - 1 ? row : im.height - 1;
        const float4 c = __ldg(S.texels + im.offset + j * im.width + i);
        return make_float3(c.x, c.y, c.z);
    }
    if (t.kind == RT_TEXTURE_NOISE)
    {
        const noise_table& n = S.noises[t.table];
        const float gray = 0.5f * (1.0f + sinf(n.scale * p.z + 10.0f * turbulence(n, p)));
        return make_float3(gray, gray, gray);
    }
    return make_float3(t.r, t.g, t.b);
}

// ---- the books' lights list (lights.cuh:49-227) ---------------------------------------------------------------
__device__ __forceinline__ quad_v light_quad(const light24& l)
{
    return {make_float3(l.quad.qx, l.quad.qy, l.quad.qz), make_float3(l.quad.nx, l.quad.ny, l.quad.nz),
            make_float3(l.quad.ax, l.quad.ay, l.quad.az), make_float3(l.quad.bx, l.quad.by, l.quad.bz)};
}

__device__ __forceinline__ float one_minus_cos_theta_max(float radius, float distance_squared)
{
    const float sin_squared = radius * radius / distance_squared;
    return sin_squared / (1.0f + sqrtf(1.0f - sin_squared));
}

// |center - origin|^2 with its multiply-adds written out, so that the density and the sampler decide alike
__device__ __forceinline__ float sphere_distance_squared(float3 v)
{
    return fmaf(v.z, v.z, fmaf(v.x, v.x, __fmul_rn(v.y, v.y)));
}

__device__ float lights_pdf_value(const scene_view& S, float3 origin, float3 direction, int from)
{
    float sum = 0.0f;
    for (int k = 0; k < S.light_count; ++k)
    {
        const light24& l = S.lights[k];
        const bool own = from >= 0 && l.twin == from;
        if (l.kind == RT_LIGHT_QUAD)
        {
            if (own)
            {
                continue;
            }
            float t;
            bool front;
            if (!hit_quad(light_quad(l), origin, direction, t_min, infinity_f, t, front))
            {
                continue;
            }
            const float len2 = length_squared(direction);
            const float distance_squared = t * t * len2;
            const float3 n = make_float3(l.quad.nx, l.quad.ny, l.quad.nz);
            const float cosine = fabsf(dot(direction, n)) * rsqrtf(len2);
            sum += l.weight * (distance_squared / (cosine * l.area));
        }
        else
        {
            const float3 c = make_float3(l.cx, l.cy, l.cz);
            const float3 to_center = c - origin;
            const float distance_squared = sphere_distance_squared(to_center);
            if (distance_squared < l.radius * l.radius)
            {
                sum += l.weight * uniform_sphere_density;
                continue;
            }
            if (own && !(dot(direction, to_center) > 0.0f))
            {
                continue;
            }
            float t;
            bool entering;
            if (!hit_sphere(make_float4(c.x, c.y, c.z, l.radius), origin, direction, 1.0f / length_squared(direction),
                            t_min, infinity_f, own, t, entering))
            {
                continue;
            }
            sum += l.weight * (1.0f / (2.0f * pi_f * one_minus_cos_theta_max(l.radius, distance_squared)));
        }
    }
    return sum;
}

// lights_random: the running sums pick a light with `pick`; (a, b) draw its point or direction
__device__ float3 lights_random(const scene_view& S, float3 origin, float pick, float a, float b)
{
    int k = 0;
    while (k < S.light_count - 1 && !(pick < S.lights[k].cdf))
    {
        ++k;
    }
    const light24& l = S.lights[k];
    if (l.kind == RT_LIGHT_QUAD)
    {
        const float3 q = make_float3(l.quad.qx, l.quad.qy, l.quad.qz);
        return unit_vector((q - origin) + a * make_float3(l.ux, l.uy, l.uz) + b * make_float3(l.vx, l.vy, l.vz));
    }
    const float3 to_center = make_float3(l.cx, l.cy, l.cz) - origin;
    const float distance_squared = sphere_distance_squared(to_center);
    if (distance_squared < l.radius * l.radius)
    {
        return random_unit_vector(a, b);
    }
    const float one_minus_cos_max = one_minus_cos_theta_max(l.radius, distance_squared);
    float s, c;
    sincospif(2.0f * a, &s, &c);
    const float one_minus_z = b * one_minus_cos_max;
    const float sin_theta = sqrtf(one_minus_z * (2.0f - one_minus_z));
    return around(rsqrtf(distance_squared) * to_center,
                  make_float3(c * sin_theta, s * sin_theta, 1.0f - one_minus_z));
}

// ---- the NEE/MIS integrator's lamps and weights (lamps.cuh, light_sampler.cuh, mis.cuh) ------------------------
__device__ __forceinline__ float power_weight(float self, float other)
{
    if (!(self > 0.0f))
    {
        return 0.0f;
    }
    const float r = other / self;
    const float w = 1.0f / fmaf(r, r, 1.0f);
    return w == w ? w : 0.0f;
}

__device__ __forceinline__ float light_weight(int c, float p_light, float p_bsdf)
{
    return c == RT_COMBINE_POWER_HEURISTIC ? power_weight(p_light, p_bsdf) : 1.0f;
}

__device__ __forceinline__ float bsdf_weight(int c, float p_bsdf, float p_light)
{
    if (c == RT_COMBINE_BSDF_ONLY || !(p_bsdf > 0.0f) || !(p_light > 0.0f))
    {
        return 1.0f;
    }
    return c == RT_COMBINE_POWER_HEURISTIC ? power_weight(p_bsdf, p_light) : 0.0f;
}

struct lamp_sample
{
    float3 wi;
    float distance;
    float pdf;
};

// sample_lamp (lamps.cuh:81-131): two numbers; false for the back of a quad or a point inside a sphere
__device__ bool sample_lamp(const emitter20& e, float3 x, float a, float b, lamp_sample& out)
{
    const float3 corner = make_float3(e.cx, e.cy, e.cz);
    if (e.kind == RT_LIGHT_QUAD)
    {
        const float3 to = (corner - x) + a * make_float3(e.ux, e.uy, e.uz) + b * make_float3(e.vx, e.vy, e.vz);
        const float distance_squared = length_squared<rounds::lamp_distance>(to);
        const float inverse_distance = rsqrtf(distance_squared);
        out.wi = inverse_distance * to;
        out.distance = distance_squared * inverse_distance;
        const float cos_light = -dot<rounds::lamp_cosine>(out.wi, make_float3(e.nx, e.ny, e.nz));
        if (!(cos_light > 0.0f))
        {
            return false;
        }
        out.pdf = distance_squared / (cos_light * e.size);
        return true;
    }
    const float3 to_center = corner - x;
    const float distance_squared = sphere_distance_squared(to_center);
    const float radius_squared = e.size * e.size;
    if (!(distance_squared > radius_squared))
    {
        return false;
    }
    const float one_minus_cos_max = one_minus_cos_theta_max(e.size, distance_squared);
    float s, c;
    sincospif(2.0f * a, &s, &c);
    const float one_minus_z = b * one_minus_cos_max;
    const float sin_squared = one_minus_z * (2.0f - one_minus_z);
    const float sin_theta = sqrtf(sin_squared);
    const float cos_theta = 1.0f - one_minus_z;
    const float inverse_distance = rsqrtf(distance_squared);
    out.wi = around(inverse_distance * to_center, make_float3(c * sin_theta, s * sin_theta, cos_theta));
    const float distance = distance_squared * inverse_distance;
    out.distance = distance * cos_theta - sqrtf(fmaxf(0.0f, fmaf(-distance_squared, sin_squared, radius_squared)));
    out.pdf = 1.0f / (2.0f * pi_f * one_minus_cos_max);
    return true;
}

// lamp_pdf (lamps.cuh:136-146), for a ray from x that hit lamp e at `distance`
__device__ float lamp_pdf(const emitter20& e, float3 x, float3 unit_dir, float distance)
{
    if (e.kind == RT_LIGHT_QUAD)
    {
        const float cos_light = -dot(unit_dir, make_float3(e.nx, e.ny, e.nz));
        return cos_light > 0.0f ? distance * distance / (cos_light * e.size) : 0.0f;
    }
    const float distance_squared = sphere_distance_squared(make_float3(e.cx, e.cy, e.cz) - x);
    return distance_squared > e.size * e.size
               ? 1.0f / (2.0f * pi_f * one_minus_cos_theta_max(e.size, distance_squared))
               : 0.0f;
}

// ---- the camera (camera.cuh:53-107) -----------------------------------------------------------------------------
__device__ __forceinline__ void camera_ray(const camera_params& cam, int i, int j, int s_i, int s_j, float4 u,
                                           float3& origin, float3& direction)
{
    const float dx = (static_cast<float>(s_i) + u.x) * cam.recip_sqrt_spp - 0.5f;
    const float dy = (static_cast<float>(s_j) + u.y) * cam.recip_sqrt_spp - 0.5f;
    const float3 to_sample = f3v(cam.center_to_pixel00) + (static_cast<float>(i) + dx) * f3v(cam.delta_u) +
                             (static_cast<float>(j) + dy) * f3v(cam.delta_v);
    origin = f3v(cam.center);
    direction = to_sample;
    if (cam.defocus)
    {
        // A uniform point of the unit disk: r = sqrt(u), angle 2 pi v (random.cuh:110-120)
        const float r = sqrtf(u.z);
        float s, c;
        sincospif(2.0f * u.w, &s, &c);
        const float3 lens = (r * c) * f3v(cam.disk_u) + (r * s) * f3v(cam.disk_v);
        origin = origin + lens;
        direction = to_sample - lens;
    }
}

__device__ __forceinline__ float3 sky(const camera_params& cam, float3 direction)
{
    const float a = 0.5f * (unit_vector<rounds::sky>(direction).y + 1.0f);
    return (1.0f - a) * f3v(cam.sky_bottom) + a * f3v(cam.sky_top);
}

__device__ __forceinline__ double without_nan(float x) { return static_cast<double>(x == x ? x : 0.0f); }

// ---- one path: its state between segments ----------------------------------------------------------------------
struct path_state
{
    float3 o, d;
    float3 throughput;
    float3 radiance; // the NEE/MIS integrator's light found so far
    float bsdf_pdf;  // the density of d at a vertex that took a light sample; 0 otherwise
    bool specular;   // d left the camera or a delta vertex: an escape sees the map filtered
    int rays_left;
    int depth;       // rays traced so far in this sample (the next vertex's depth in the RNG counter)
    int from;
    bool inward;
    float time;      // the moment in the shutter the sample's rays are at (0 in a scene where nothing moves)
};

// The hit as the shading needs it: point, outward normal, material, the hit's side
struct surface
{
    float3 p;
    float3 outward;
    float3 normal;
    float3 color; // the material's color here: its texture read at the hit, or its one solid color
    int material;
    int from;     // the next ray's `from`: the hit primitive, or -1 after a particle of smoke (which has no surface)
};

// The texture coordinates of a point of a sphere (sphere.cuh:119-135): the longitude and latitude of its outward
// normal turned back by the instances' turn, u from -x around y, v from the south pole
__device__ __forceinline__ void sphere_uv(float3 outward, const sphere_frame& f, float& u, float& v)
{
    const float nx = f.cos_theta * outward.x - f.sin_theta * outward.z;
    const float nz = f.sin_theta * outward.x + f.cos_theta * outward.z;
    const float phi = atan2f(-nz, nx) + pi_f;
    const float theta = acosf(fminf(fmaxf(-outward.y, -1.0f), 1.0f));
    u = phi * (0.5f * inverse_pi_f);
    v = theta * inverse_pi_f;
}

// The hit point moved onto the sphere by one Newton step along the outward normal, for a checker to read
// (onto_sphere, sphere.cuh:137-168): f = |p|^2 - 2 p.c + k with k = |c|^2 - r^2 from the host, taken only while its
// rounding bound stays below the frame's limit 2 r |c|
__device__ __forceinline__ float3 onto_sphere(float3 p, float3 outward, float4 ball, const sphere_frame& f)
{
    const float3 c = make_float3(ball.x, ball.y, ball.z);
    const float p_p = dot(p, p);
    const float p_c = dot(p, c);
    if (!(p_p + 2.0f * fabsf(p_c) + fabsf(f.k) < f.limit))
    {
        return p;
    }
    const float value = p_p - 2.0f * p_c + f.k;
    return p - (value / (2.0f * fabsf(ball.w))) * outward;
}

// The hit as the shading needs it (surface_at, camera.cuh:171-253), and the material there with its color
template <bool FEATURES = true>
__device__ __forceinline__ surface surface_at(const scene_view& S, const path_state& ps, const hit_info& h,
                                              material12& m)
{
    surface s;
    s.from = h.id;
    float u = 0.0f, v = 0.0f;
    float4 ball = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    bool on_sphere = false;
    if (FEATURES && h.id >= S.medium_base)
    {
        // A particle of smoke (constant_medium::hit): any normal and side will do, the CPU's (1, 0, 0) and the front
        s.p = ps.o + h.t * ps.d;
        s.outward = make_float3(1.0f, 0.0f, 0.0f);
        s.normal = s.outward;
        s.material = S.media[h.id - S.medium_base].material;
        s.from = -1;
        m = S.materials[s.material];
    }
    else
    {
        s.material = __ldg(S.prim_material + h.id);
        m = S.materials[s.material];
        if (h.id < S.quad_base)
        {
            ball = sphere_at<FEATURES>(S, h.id, ps.time);
            on_sphere = true;
            s.p = ps.o + h.t * ps.d;
            s.outward = (1.0f / fabsf(ball.w)) * (s.p - make_float3(ball.x, ball.y, ball.z));
        }
        else if (h.id < S.triangle_base)
        {
            // The quad's point as the CPU computes it, t * d rounded, then the sum (camera.cuh:175-195 at_unfused)
            const quad_v q = load_quad(S.quads, h.id - S.quad_base);
            s.p = make_float3(__fadd_rn(ps.o.x, __fmul_rn(h.t, ps.d.x)), __fadd_rn(ps.o.y, __fmul_rn(h.t, ps.d.y)),
                              __fadd_rn(ps.o.z, __fmul_rn(h.t, ps.d.z)));
            s.outward = q.n;
            if (FEATURES && m.texture >= 0 && (m.texture_needs & texture_needs_uv) != 0)
            {
                // quad_uv (quad.cuh:86-94): alpha and beta of the point, from hit_quad's expressions
                const float3 rel = h.t * ps.d - (q.q - ps.o);
                u = dot(rel, q.a);
                v = dot(rel, q.b);
            }
        }
        else
        {
            const triangle_v tr = load_triangle(S.triangles, h.id - S.triangle_base);
            s.p = ps.o + h.t * ps.d;
            s.outward = unit_vector(cross(tr.b - tr.a, tr.c - tr.a));
        }
        s.normal = h.front ? s.outward : -s.outward;
    }
    s.color = make_float3(m.r, m.g, m.b);
    if (FEATURES && m.texture >= 0)
    {
        float3 point = s.p;
        if (on_sphere && (m.texture_needs & (texture_needs_uv | texture_needs_point)) != 0)
        {
            const sphere_frame f = S.sphere_frames[h.id];
            if (m.texture_needs & texture_needs_uv)
            {
                sphere_uv(s.outward, f, u, v);
            }
            if (m.texture_needs & texture_needs_point)
            {
                point = onto_sphere(s.p, s.outward, ball, f);
            }
        }
        s.color = texture_value(S, m.texture, u, v, point);
    }
    return s;
}

enum class step_result
{
    go_on,
    done,
};

// One segment of a books' path (camera.cuh:364-437 trace_ray with diffuse_bounce 304-359 and scatter
// material.cuh:84-126), after its closest hit
template <bool FEATURES = true>
__device__ __forceinline__ step_result shade_books(const scene_view& S, const camera_params& cam, const sampler& rng,
                                                   path_state& ps, const hit_info& h, float3& sample)
{
    if (h.id < 0)
    {
        sample = ps.throughput * sky(cam, ps.d);
        return step_result::done;
    }
    material12 m;
    const surface s = surface_at<FEATURES>(S, ps, h, m);
    const float3 albedo = s.color;
    float3 direction;
    if (m.kind == RT_DIFFUSE_LIGHT)
    {
        sample = h.front ? ps.throughput * albedo : make_float3(0.0f, 0.0f, 0.0f);
        return step_result::done;
    }
    const float4 u = rng.draw(ps.depth, block_material);
    if (m.kind == RT_LAMBERTIAN || m.kind == RT_ISOTROPIC)
    {
        // A diffuse bounce (diffuse_bounce, camera.cuh:300-359): a matte surface, or a particle of smoke, which keeps
        // its own density (1/(4 pi) everywhere) except under the lights strategy (isotropic::mixes_in_lights is false)
        const bool matte = m.kind == RT_LAMBERTIAN;
        int strategy = cam.sampling;
        if (!matte && strategy != RT_SAMPLING_LIGHTS)
        {
            strategy = RT_SAMPLING_MATERIAL;
        }
        if (strategy == RT_SAMPLING_MATERIAL)
        {
            direction = matte ? around(s.normal, random_cosine_direction(u.x, u.y)) : random_unit_vector(u.x, u.y);
            if (matte && !(dot(s.normal, direction) > 0.0f))
            {
                sample = make_float3(0.0f, 0.0f, 0.0f);
                return step_result::done;
            }
            ps.throughput = ps.throughput * albedo;
        }
        else
        {
            bool toward_lights = strategy == RT_SAMPLING_LIGHTS;
            if (strategy == RT_SAMPLING_MIXTURE)
            {
                toward_lights = u.z < 0.5f;
            }
            if (toward_lights)
            {
                direction = lights_random(S, s.p, u.w, u.x, u.y);
            }
            else
            {
                direction = strategy == RT_SAMPLING_UNIFORM ? random_unit_vector(u.x, u.y)
                                                            : around(s.normal, random_cosine_direction(u.x, u.y));
            }
            const float p_scatter = matte ? cosine_density(s.normal, direction) : uniform_sphere_density;
            float p = uniform_sphere_density;
            if (strategy != RT_SAMPLING_UNIFORM)
            {
                const float p_lights = lights_pdf_value(S, s.p, direction, s.from);
                p = strategy == RT_SAMPLING_LIGHTS ? p_lights : 0.5f * p_lights + 0.5f * p_scatter;
            }
            if (!(p > 0.0f) || !(p_scatter > 0.0f))
            {
                sample = make_float3(0.0f, 0.0f, 0.0f);
                return step_result::done;
            }
            ps.throughput = (p_scatter / p) * (ps.throughput * albedo);
        }
    }
    else if (m.kind == RT_METAL)
    {
        direction = unit_vector(reflect(ps.d, s.normal)) + m.fuzz * random_unit_vector(u.x, u.y);
        if (dot(direction, s.normal) <= 0.0f)
        {
            sample = make_float3(0.0f, 0.0f, 0.0f);
            return step_result::done;
        }
        ps.throughput = ps.throughput * albedo;
    }
    else // dielectric
    {
        const float ri = h.front ? 1.0f / m.ior : m.ior;
        const float3 ud = unit_vector<rounds::dielectric_unit>(ps.d);
        const float cos_theta = fminf(dot<rounds::dielectric_cosine>(-ud, s.normal), 1.0f);
        const float sin_theta = sqrtf(1.0f - cos_theta * cos_theta);
        const bool cannot_refract = ri * sin_theta > 1.0f;
        direction = cannot_refract || reflectance(cos_theta, ri) > u.z ? reflect<rounds::dielectric_reflect>(ud, s.normal)
                                                                       : refract(ud, s.normal, ri);
    }
    if (--ps.rays_left == 0)
    {
        sample = make_float3(0.0f, 0.0f, 0.0f);
        return step_result::done;
    }
    ps.o = s.p;
    ps.d = direction;
    ps.from = s.from;
    ps.inward = dot(direction, s.outward) < 0.0f;
    return step_result::go_on;
}

// ---- GGX (ggx.cuh: Walter et al. 2007, Heitz 2014 and 2018, Dupuy & Benyoub 2023, Turquin 2019) --------------
constexpr float min_ggx_alpha = 1e-3f; // below it, the perfect mirror with Schlick's F (ggx.cuh:37)

__constant__ float ggx_energy_table[32 * 32] = {RTB_GGX_ENERGY_TABLE};

__device__ __forceinline__ float smith_a(float c, float alpha2) { return sqrtf(fmaf(c * c, 1.0f - alpha2, alpha2)); }

// D(h) = alpha^2 / (pi (alpha^2 c^2 + sin^2)^2), sin^2 from |n x h|^2 (exact near the peak)
__device__ __forceinline__ float ggx_d(float3 n, float3 h, float alpha2)
{
    const float c = dot(n, h);
    if (!(c > 0.0f))
    {
        return 0.0f;
    }
    const float3 s = cross(n, h);
    const float d = fmaf(alpha2 * c, c, dot(s, s));
    return alpha2 * inverse_pi_f / (d * d);
}

__device__ __forceinline__ float3 schlick(float3 f0, float cosine)
{
    const float x = fmaxf(0.0f, 1.0f - cosine);
    const float x2 = x * x;
    const float x5 = x2 * x2 * x;
    return make_float3(fmaf(1.0f - f0.x, x5, f0.x), fmaf(1.0f - f0.y, x5, f0.y), fmaf(1.0f - f0.z, x5, f0.z));
}

// f * cos(theta_l) = F D cl / (2 (cl A_v + cv A_l)) and the visible-normal density D / (2 (cv + A_v))
template <rounding LENGTH, rounding LIGHT = rounds::other>
__device__ float3 ggx_eval(float3 n, float3 v, float3 l, float alpha, float3 f0, float& pdf)
{
    pdf = 0.0f;
    const float cv = dot<rounds::ggx_eval_view>(n, v);
    const float cl = dot<LIGHT>(n, l);
    const float3 sum = v + l;
    const float len2 = length_squared<LENGTH>(sum);
    if (!(cv > 0.0f) || !(cl > 0.0f) || !(len2 > 0.0f))
    {
        return make_float3(0.0f, 0.0f, 0.0f);
    }
    const float3 h = rsqrtf(len2) * sum;
    const float alpha2 = alpha * alpha;
    const float d = ggx_d(n, h, alpha2);
    const float av = smith_a(cv, alpha2);
    const float al = smith_a(cl, alpha2);
    pdf = d / (2.0f * (cv + av));
    return (d * cl / (2.0f * (cl * av + cv * al))) * schlick(f0, dot<rounds::ggx_eval_half>(v, h));
}

// A direction by the visible normals with spherical caps: u1 the azimuth, u2 the height in the cap; weight
// F G2/G1 (at most F); false: absorbed
__device__ bool ggx_sample(float3 n, float3 v, float alpha, float3 f0, float u1, float u2, float3& l, float3& weight,
                           float& pdf)
{
    const float cv = dot<rounds::ggx_sample_view>(n, v);
    if (!(cv > 0.0f))
    {
        return false;
    }
    const float3 vs = unit_vector(alpha * (v - cv * n) + cv * n);
    const float zs = dot(n, vs);
    const float z = fmaf(1.0f - u2, 1.0f + zs, -zs);
    const float sin_theta = sqrtf(fmaxf(0.0f, 1.0f - z * z));
    float s, c;
    sincospif(2.0f * u1, &s, &c);
    const float3 cap = around(n, make_float3(sin_theta * c, sin_theta * s, z));
    const float3 hs = cap + vs;
    const float hn = dot(n, hs);
    const float3 m = alpha * (hs - hn * n) + fmaxf(0.0f, hn) * n;
    const float m2 = length_squared(m);
    if (!(m2 > 0.0f))
    {
        return false;
    }
    const float3 h = rsqrtf(m2) * m;
    const float vh = dot<rounds::ggx_sample_half>(v, h);
    l = (2.0f * vh) * h - v;
    const float cl = dot(n, l);
    if (!(cl > 0.0f) || !(vh > 0.0f))
    {
        return false;
    }
    const float alpha2 = alpha * alpha;
    const float av = smith_a(cv, alpha2);
    const float al = smith_a(cl, alpha2);
    weight = (cl * (cv + av) / (cl * av + cv * al)) * schlick(f0, vh);
    pdf = ggx_d(n, h, alpha2) / (2.0f * (cv + av));
    return true;
}

// Turquin's factor 1 + F0 (1 - E) / E, E from the energy table (bilinear; nodes sqrt(mu) = i/31, r = j/31)
__device__ float3 ggx_compensation(float3 f0, float cos_v, float roughness)
{
    constexpr int last = 31;
    const float x = sqrtf(fminf(fmaxf(cos_v, 0.0f), 1.0f)) * static_cast<float>(last);
    const float y = fminf(fmaxf(roughness, 0.0f), 1.0f) * static_cast<float>(last);
    const int i = min(static_cast<int>(x), last - 1);
    const int j = min(static_cast<int>(y), last - 1);
    const float fx = x - static_cast<float>(i);
    const float fy = y - static_cast<float>(j);
    const float* row = ggx_energy_table + j * 32 + i;
    const float below = (1.0f - fx) * row[0] + fx * row[1];
    const float above = (1.0f - fx) * row[32] + fx * row[33];
    const float e = fminf((1.0f - fy) * below + fy * above, 1.0f);
    const float lost = (1.0f - e) / e;
    return make_float3(fmaf(f0.x, lost, 1.0f), fmaf(f0.y, lost, 1.0f), fmaf(f0.z, lost, 1.0f));
}

constexpr float gloss_coat_f0 = 0.04f;
constexpr float gloss_diffuse_scale = 0.37200738f; // 28 / (23 pi) * (1 - 0.04)

__device__ __forceinline__ float gloss_crossing(float c)
{
    const float x = 1.0f - 0.5f * c;
    const float x2 = x * x;
    return 1.0f - x2 * x2 * x;
}

// The coat over a matte base of color rho: GGX with F0 0.04 plus the coupled diffuse term; pdf the half-and-half
// mixture of the two lobes' densities
template <rounding LENGTH, rounding LIGHT = rounds::other>
__device__ float3 gloss_eval(float3 n, float3 v, float3 l, float alpha, float3 rho, float& pdf)
{
    pdf = 0.0f;
    const float cv = dot<rounds::ggx_eval_view>(n, v);
    const float cl = dot<LIGHT>(n, l);
    if (!(cv > 0.0f) || !(cl > 0.0f))
    {
        return make_float3(0.0f, 0.0f, 0.0f);
    }
    float coat_pdf;
    const float3 coat = ggx_eval<LENGTH, LIGHT>(n, v, l, alpha, make_float3(gloss_coat_f0, gloss_coat_f0, gloss_coat_f0), coat_pdf);
    pdf = 0.5f * (coat_pdf + cl * inverse_pi_f);
    const float base = gloss_diffuse_scale * (gloss_crossing(cl) * gloss_crossing(cv)) * cl;
    return coat + base * rho;
}

// ---- the environment map (environment.cuh, background.cuh) ---------------------------------------------------
__device__ __forceinline__ float3 to_map(const environment_view& e, float3 d)
{
    return make_float3(e.cos_yaw * d.x + e.sin_yaw * d.z, d.y, -e.sin_yaw * d.x + e.cos_yaw * d.z);
}

__device__ __forceinline__ float3 from_map(const environment_view& e, float3 d)
{
    return make_float3(e.cos_yaw * d.x - e.sin_yaw * d.z, d.y, e.sin_yaw * d.x + e.cos_yaw * d.z);
}

// u = 0.5 + atan2(z, x) / (2 pi) across, t = atan2(sqrt(x^2 + z^2), y) / pi down: +y up, seen from inside
__device__ __forceinline__ void map_coordinates(float3 m, float& u, float& t)
{
    u = 0.5f + atan2f(m.z, m.x) * (0.5f * inverse_pi_f);
    t = atan2f(sqrtf(m.x * m.x + m.z * m.z), m.y) * inverse_pi_f;
}

__device__ __forceinline__ int clamp_index(int k, int n) { return k < 0 ? 0 : (k < n ? k : n - 1); }

// The one map from a direction to its cell, used by escapes and light samples alike
__device__ __forceinline__ int env_cell(const environment_view& e, float3 world)
{
    float u, t;
    map_coordinates(to_map(e, world), u, t);
    const int i = clamp_index(static_cast<int>(u * static_cast<float>(e.width)), e.width);
    const int j = clamp_index(static_cast<int>(t * static_cast<float>(e.height)), e.height);
    return j * e.width + i;
}

__device__ __forceinline__ float3 env_radiance(const environment_view& e, float3 dir, float& pdf)
{
    const env_texel texel = e.texels[env_cell(e, dir)];
    pdf = texel.pdf;
    return e.scale * make_float3(texel.r, texel.g, texel.b);
}

__device__ float3 env_radiance_filtered(const environment_view& e, float3 dir)
{
    float u, t;
    map_coordinates(to_map(e, dir), u, t);
    const float x = u * static_cast<float>(e.width) - 0.5f;
    const float y = t * static_cast<float>(e.height) - 0.5f;
    const float x0 = floorf(x);
    const float y0 = floorf(y);
    const float fx = x - x0;
    const float fy = y - y0;
    const int i = static_cast<int>(x0);
    const int i0 = i < 0 ? i + e.width : i;
    const int i1 = i0 + 1 < e.width ? i0 + 1 : 0;
    const int j = static_cast<int>(y0);
    const int j0 = clamp_index(j, e.height) * e.width;
    const int j1 = clamp_index(j + 1, e.height) * e.width;
    const auto texel = [&](int k) {
        const env_texel t4 = e.texels[k];
        return make_float3(t4.r, t4.g, t4.b);
    };
    const float3 a = texel(j0 + i0);
    const float3 b = texel(j0 + i1);
    const float3 c = texel(j1 + i0);
    const float3 d = texel(j1 + i1);
    const float3 top = a + fx * (b - a);
    const float3 bottom = c + fx * (d - c);
    return e.scale * (top + fy * (bottom - top));
}

// A cell from the alias table (the bin from the top bits of `bits`, then its coin), then a direction uniform over
// the cell's solid angle; the radiance and density of the cell the direction lands in
__device__ bool sample_environment(const environment_view& e, uint32_t bits, float coin, float s_theta, float s_phi,
                                   float3& wi, float3& le, float& pdf)
{
    const int bin = static_cast<int>(bits >> (32 - e.log2_bins));
    const alias_bin b = e.bins[bin];
    const int cell = coin < b.q ? bin : b.alias;
    const int j = cell / e.width;
    const int i = cell - j * e.width;
    const float top = e.row_cos[j];
    const float bottom = e.row_cos[j + 1];
    const float cos_theta = top - s_theta * (top - bottom);
    const float sin_theta = sqrtf(fmaxf(0.0f, (1.0f - cos_theta) * (1.0f + cos_theta)));
    float sp, cp;
    sincospif(2.0f * (static_cast<float>(i) + s_phi) / static_cast<float>(e.width) - 1.0f, &sp, &cp);
    wi = from_map(e, make_float3(sin_theta * cp, cos_theta, sin_theta * sp));
    le = env_radiance(e, wi, pdf);
    return pdf > 0.0f;
}

// ---- the NEE/MIS step (quality_path.cuh:83-188, bsdf.cuh:30-201, light_sampler.cuh:40-103) -------------------
enum lobe_id : int
{
    lobe_lambertian,
    lobe_isotropic,
    lobe_conductor,
    lobe_gloss,
    lobe_smooth_conductor, // from here on: delta lobes (no density)
    lobe_books_delta,
};

__device__ __forceinline__ int lobe_of(const material12& m)
{
    if (m.lobe == RT_MICROFACET_CONDUCTOR)
    {
        return m.alpha >= min_ggx_alpha ? lobe_conductor : lobe_smooth_conductor;
    }
    if (m.lobe == RT_MICROFACET_GLOSS)
    {
        return lobe_gloss;
    }
    return m.kind == RT_LAMBERTIAN ? lobe_lambertian : m.kind == RT_ISOTROPIC ? lobe_isotropic : lobe_books_delta;
}

// eval_bsdf: f * |cos| of a light sample's unit direction, and the lobe's density of it (0 for delta lobes)
__device__ float3 eval_lobe(int lobe, const material12& m, float3 albedo, float3 n, float3 wo, float3 wi, float& pdf)
{
    if (lobe == lobe_lambertian)
    {
        pdf = cosine_density(n, wi);
        return pdf * albedo;
    }
    if (lobe == lobe_isotropic)
    {
        pdf = uniform_sphere_density;
        return uniform_sphere_density * albedo;
    }
    if (lobe == lobe_conductor)
    {
        const float3 single = ggx_eval<rounds::ggx_light_length>(n, wo, wi, m.alpha, albedo, pdf);
        return ggx_compensation(albedo, dot<rounds::energy>(n, wo), m.roughness) * single;
    }
    if (lobe == lobe_gloss)
    {
        return gloss_eval<rounds::ggx_light_length>(n, wo, wi, m.alpha, albedo, pdf);
    }
    pdf = 0.0f;
    return make_float3(0.0f, 0.0f, 0.0f);
}

// A shadow ray handed back to the caller instead of traced (the wavefront's trace kernel walks it): the ray, and the
// light it brings to the path's radiance if nothing blocks it
struct shadow_query
{
    float3 o, d;
    float3 contribution;
    float t_max;
    int from;
    int skip;
    bool inward;
    bool lit;
};

// One segment of an NEE/MIS path after its closest hit; the shadow ray is traced here, or with DEFER handed back in
// `deferred` (lit set) with the path's radiance left without it: a `done` sample then is the radiance once the
// caller has added the light
template <bool COUNT, int SEARCH = search_any, bool FEATURES = true, bool DEFER = false>
__device__ __forceinline__ step_result shade_quality(const scene_view& S, const camera_params& cam,
                                                     const sampler& rng, path_state& ps, const hit_info& h,
                                                     float3& sample, uint32_t& shadow_rays, fetch_counts* counts,
                                                     shadow_query* deferred = nullptr)
{
    if (h.id < 0)
    {
        // The environment (filtered after the camera and delta vertices, the nearest texel with its density
        // otherwise), or the camera's sky
        if (!S.has_environment)
        {
            sample = ps.radiance + ps.throughput * sky(cam, ps.d);
            return step_result::done;
        }
        if (ps.specular)
        {
            sample = ps.radiance + ps.throughput * env_radiance_filtered(S.env, ps.d);
            return step_result::done;
        }
        float density;
        const float3 le = env_radiance(S.env, ps.d, density);
        const float p_light = S.env.sampled ? S.light_pmf * density : 0.0f;
        const float w = ps.bsdf_pdf > 0.0f ? bsdf_weight(S.combination, ps.bsdf_pdf, p_light) : 1.0f;
        sample = ps.radiance + w * (ps.throughput * le);
        return step_result::done;
    }
    material12 m;
    const surface s = surface_at<FEATURES>(S, ps, h, m);
    const float3 albedo = s.color;
    if (m.kind == RT_DIFFUSE_LIGHT)
    {
        float w = 1.0f;
        if (ps.bsdf_pdf > 0.0f)
        {
            const int k = S.lamp_count > 0 ? __ldg(S.lamp_of + h.id) : -1;
            float p_light = 0.0f;
            if (k >= 0)
            {
                const float distance = h.t * sqrtf(length_squared<rounds::lamp_hit>(ps.d));
                p_light = S.light_pmf * lamp_pdf(S.lamps[k], ps.o, unit_vector<rounds::lamp_hit>(ps.d), distance);
            }
            w = bsdf_weight(S.combination, ps.bsdf_pdf, p_light);
        }
        sample = ps.radiance + w * (h.front ? ps.throughput * albedo : make_float3(0.0f, 0.0f, 0.0f));
        return step_result::done;
    }
    const int lobe = lobe_of(m);
    const bool delta = lobe >= lobe_smooth_conductor;
    const float3 wo = -unit_vector<rounds::view>(ps.d);
    const int lights = S.lamp_count + (S.env.sampled ? 1 : 0);
    const bool nee = S.combination != RT_COMBINE_BSDF_ONLY && ps.rays_left > 1 && !delta && lights > 0 &&
                     largest_channel(ps.throughput) > 0.0f;
    bool lit = false;
    float3 contribution = make_float3(0.0f, 0.0f, 0.0f);
    float3 light_dir = make_float3(0.0f, 0.0f, 0.0f);
    float light_distance = infinity_f;
    int skip = -1;
    if (nee)
    {
        // One number picks a light, the lamps first and the map last (light_sampler.cuh:40-75)
        const uint4 bits = rng.draw_bits(ps.depth, block_nee);
        const float pick = to_unit(bits.x);
        int k = static_cast<int>(pick * static_cast<float>(lights));
        k = k < lights ? k : lights - 1;
        bool drawn = false;
        float3 le;
        float p_light = 0.0f;
        if (k < S.lamp_count)
        {
            const emitter20 e = S.lamps[k];
            lamp_sample ls;
            if (sample_lamp(e, s.p, to_unit(bits.y), to_unit(bits.z), ls))
            {
                drawn = true;
                light_dir = ls.wi;
                light_distance = ls.distance;
                le = make_float3(e.er, e.eg, e.eb);
                p_light = S.light_pmf * ls.pdf;
                skip = e.primitive;
            }
        }
        else
        {
            float density;
            const float s_phi = rng.draw(ps.depth, block_nee + 1).x;
            if (sample_environment(S.env, bits.y, to_unit(bits.z), to_unit(bits.w), s_phi, light_dir, le, density))
            {
                drawn = true;
                p_light = S.light_pmf * density;
            }
        }
        if (drawn)
        {
            float p_bsdf;
            const float3 f = eval_lobe(lobe, m, albedo, s.normal, wo, light_dir, p_bsdf);
            if (p_light > 0.0f && largest_channel(f) > 0.0f)
            {
                contribution =
                    (light_weight(S.combination, p_light, p_bsdf) / p_light) * (ps.throughput * (f * le));
                const float sum = contribution.x + contribution.y + contribution.z;
                lit = sum > 0.0f && sum < infinity_f;
            }
        }
    }
    // The material's own sample: the path's next ray
    const float4 u = rng.draw(ps.depth, block_material);
    float3 wi = make_float3(0.0f, 0.0f, 0.0f);
    float3 weight = albedo;
    float pdf = 0.0f;
    bool scattered = true;
    if (lobe == lobe_lambertian)
    {
        wi = around(s.normal, random_cosine_direction(u.x, u.y));
        scattered = dot(s.normal, wi) > 0.0f;
        pdf = cosine_density(s.normal, wi);
    }
    else if (lobe == lobe_isotropic)
    {
        wi = random_unit_vector(u.x, u.y);
        pdf = uniform_sphere_density;
    }
    else if (lobe == lobe_conductor)
    {
        scattered = ggx_sample(s.normal, wo, m.alpha, albedo, u.x, u.y, wi, weight, pdf);
        if (scattered)
        {
            weight = weight * ggx_compensation(albedo, dot<rounds::energy>(s.normal, wo), m.roughness);
        }
    }
    else if (lobe == lobe_gloss)
    {
        // The coat or the base, half the time each, then the mixture's weight and density (ggx.cuh:300-324)
        if (u.z < 0.5f)
        {
            float3 coat_weight;
            float coat_pdf;
            scattered = ggx_sample(s.normal, wo, m.alpha, make_float3(gloss_coat_f0, gloss_coat_f0, gloss_coat_f0),
                                   u.x, u.y, wi, coat_weight, coat_pdf);
        }
        else
        {
            wi = around(s.normal, random_cosine_direction(u.x, u.y));
            scattered = dot(s.normal, wi) > 0.0f;
        }
        if (scattered)
        {
            const float3 f = gloss_eval<rounds::ggx_gloss_length, rounds::ggx_gloss_light>(s.normal, wo, wi, m.alpha, albedo, pdf);
            scattered = pdf > 0.0f;
            weight = (1.0f / pdf) * f;
        }
    }
    else if (lobe == lobe_smooth_conductor)
    {
        // The mirror with Schlick's F: no random number (bsdf.cuh:153-166)
        scattered = dot<rounds::mirror_cosine>(s.normal, wo) > 0.0f;
        wi = unit_vector(reflect<rounds::mirror_reflect>(-wo, s.normal));
        weight = schlick(albedo, dot<rounds::mirror_cosine>(s.normal, wo));
    }
    else if (m.kind == RT_METAL)
    {
        wi = unit_vector(reflect(ps.d, s.normal)) + m.fuzz * random_unit_vector(u.x, u.y);
        scattered = dot(wi, s.normal) > 0.0f;
    }
    else // dielectric
    {
        const float ri = h.front ? 1.0f / m.ior : m.ior;
        const float3 ud = unit_vector<rounds::dielectric_unit>(ps.d);
        const float cos_theta = fminf(dot<rounds::dielectric_cosine>(-ud, s.normal), 1.0f);
        const float sin_theta = sqrtf(1.0f - cos_theta * cos_theta);
        wi = ri * sin_theta > 1.0f || reflectance(cos_theta, ri) > u.z ? reflect<rounds::dielectric_reflect>(ud, s.normal)
                                                                       : refract(ud, s.normal, ri);
        weight = make_float3(1.0f, 1.0f, 1.0f);
    }
    if (DEFER)
    {
        deferred->lit = lit;
        if (lit)
        {
            ++shadow_rays;
            *deferred = {s.p, light_dir, contribution, light_distance, s.from, skip, dot(light_dir, s.outward) < 0.0f,
                         true};
        }
    }
    else if (lit)
    {
        ++shadow_rays;
        hit_info blocker;
        const bool blocked = traverse<true, COUNT, SEARCH, FEATURES>(
            S, s.p, light_dir, ps.time, light_distance, s.from, dot(light_dir, s.outward) < 0.0f, skip, blocker, counts);
        if (!blocked)
        {
            // through smoke, the light arrives with the chance of crossing it (its expected value, not a draw)
            const float through =
                FEATURES && S.medium_count > 0 ? transmittance(S, s.p, light_dir, ps.time, light_distance) : 1.0f;
            ps.radiance = ps.radiance + through * contribution;
        }
    }
    if (!scattered)
    {
        sample = ps.radiance;
        return step_result::done;
    }
    ps.throughput = ps.throughput * weight;
    ps.bsdf_pdf = nee ? pdf : 0.0f;
    ps.specular = delta;
    if (S.combination != RT_COMBINE_BSDF_ONLY && ps.throughput.x == 0.0f && ps.throughput.y == 0.0f &&
        ps.throughput.z == 0.0f)
    {
        sample = ps.radiance;
        return step_result::done;
    }
    if (--ps.rays_left == 0)
    {
        sample = ps.radiance;
        return step_result::done;
    }
    ps.o = s.p;
    ps.d = wi;
    ps.from = s.from;
    ps.inward = dot(wi, s.outward) < 0.0f;
    return step_result::go_on;
}

// Where sample number `local` of a launch (or of a batch job) lies: pass-major, then the pixels in 8x4 tiles (a
// warp's worth); x may fall past the image's right edge or y past its bottom in the last tiles
struct sample_place
{
    int64_t pass;
    int x, y;
};

// (uses the camera's divisors: cam.div_padded and cam.div_tiles_x; a number of 2^32 or more, which only a served
// request's numbering reaches, takes the 64-bit division; `first_pixel`: of a job rendered in bands)
__device__ __forceinline__ sample_place place_of(int64_t local, const camera_params& cam, int64_t pass_begin,
                                                 int first_pixel = 0)
{
    const uint32_t padded = cam.div_padded.d;
    int64_t j;
    int q;
    if (local < (int64_t{1} << 32))
    {
        const auto n = static_cast<uint32_t>(local);
        const uint32_t jj = quotient(n, cam.div_padded);
        j = jj;
        q = static_cast<int>(n - jj * padded);
    }
    else
    {
        j = local / padded;
        q = static_cast<int>(local - j * padded);
    }
    const int tile = (first_pixel + q) >> 5;
    const int l = q & 31;
    const auto ty = static_cast<int>(quotient(static_cast<uint32_t>(tile), cam.div_tiles_x));
    const int tx = tile - ty * static_cast<int>(cam.div_tiles_x.d);
    return {pass_begin + j, tx * 8 + (l & 7), ty * 4 + (l >> 3)};
}

// A pass's round of strata and its pass within the round (cam.div_round_passes)
__device__ __forceinline__ int64_t round_of(int64_t pass, const camera_params& cam)
{
    return pass < (int64_t{1} << 32) ? static_cast<int64_t>(quotient(static_cast<uint32_t>(pass), cam.div_round_passes))
                                     : pass / static_cast<int64_t>(cam.div_round_passes.d);
}

// A sample's random-number stream: its pixel, its pass within its round of strata, and the round's key
// (seed + round * 2^32), as the persistent kernel sets them when it starts the sample
__device__ __forceinline__ int sample_rng(const sample_place& at, const camera_params& cam, uint64_t seed, sampler& rng)
{
    const int64_t round = round_of(at.pass, cam);
    const int round_pass = static_cast<int>(at.pass - round * static_cast<int64_t>(cam.div_round_passes.d));
    const uint64_t key = seed + (static_cast<uint64_t>(round) << 32);
    rng.key = make_uint2(static_cast<uint32_t>(key), static_cast<uint32_t>(key >> 32));
    rng.pass = static_cast<uint32_t>(round_pass);
    rng.pixel = static_cast<uint32_t>(at.y) * static_cast<uint32_t>(cam.width) + static_cast<uint32_t>(at.x);
    return round_pass;
}

// The job of jobs [first, end) whose range of the batch's item (or pixel) space holds `index`: a binary search over
// the jobs' starts
constexpr int job_items = 0;   // find_job by item_begin
constexpr int job_pixels = 1;  // by pixel_begin
constexpr int job_samples = 2; // by sample_begin (a wavefront group's sample space)

template <int SPACE>
__device__ __forceinline__ int find_job(const batch_job* jobs, int first, int end, int64_t index, int mask = 0)
{
    int lo = first;
    int hi = end - 1;
    while (lo < hi)
    {
        const int mid = (lo + hi + 1) >> 1;
        const batch_job& j = jobs[mask != 0 ? (mid & mask) : mid]; // a stream run's ring: [first, end) unwrapped
        const int64_t begin = SPACE == job_pixels    ? j.pixel_begin
                              : SPACE == job_samples ? j.sample_begin
                                                     : j.item_begin;
        if (begin <= index)
        {
            lo = mid;
        }
        else
        {
            hi = mid - 1;
        }
    }
    return lo;
}

constexpr unsigned full_warp = 0xffffffffu;

// The slots, queries, answers and samples pass through L2 once per step: loaded and stored evict-first (.cs), so that
// they do not push the tree and the primitives, which every walk reads, out of L2
#ifndef RTB_WAVE_STREAMING
#define RTB_WAVE_STREAMING 1
#endif
template <class T>
__device__ __forceinline__ T stream_load(const T* p)
{
#if RTB_WAVE_STREAMING
    return __ldcs(p);
#else
    return *p;
#endif
}
template <class T>
__device__ __forceinline__ void stream_store(T* p, T v)
{
#if RTB_WAVE_STREAMING
    __stcs(p, v);
#else
    *p = v;
#endif
}

// A flat-searched scene's query in the wavefront: every sphere, then every quad, in order (the persistent kernel's
// flat search, the same tests and self-intersection rules); `any` (a shadow ray) stops at the first hit
template <bool FEATURES>
__device__ __forceinline__ void flat_search(const scene_view& S, float3 o, float3 d, float time, int from, bool inward,
                                            int skip, bool any, hit_info& hit)
{
    const float inverse_a = 1.0f / length_squared<rounds::walk_flat>(d);
    for (int i = 0; i < S.quad_base; ++i)
    {
        const bool own = i == from;
        if ((own && !inward) || i == skip)
        {
            continue;
        }
        const float4 s = sphere_at<FEATURES>(S, i, time);
        float t;
        bool entering;
        if (hit_sphere(s, o, d, inverse_a, t_min, hit.t, own, t, entering))
        {
            hit = {i, t, entering};
            if (any)
            {
                return;
            }
        }
    }
    const int quads = S.triangle_base - S.quad_base;
    for (int i = 0; i < quads; ++i)
    {
        const int id = S.quad_base + i;
        if (id == from || id == skip)
        {
            continue;
        }
        float t;
        bool front;
        if (hit_quad(load_quad(S.quads, i), o, d, t_min, hit.t, t, front))
        {
            hit = {id, t, front};
            if (any)
            {
                return;
            }
        }
    }
}

// The same, called rather than inlined: a walk compiled with the flat search inlined beside its own leaf tests rounds
// differently (the shared tests are contracted differently), and the walk must give a session's hits bit for bit
template <bool FEATURES>
__device__ __noinline__ void flat_search_call(const scene_view& S, float3 o, float3 d, float time, int from,
                                              bool inward, int skip, bool any, hit_info& hit)
{
    flat_search<FEATURES>(S, o, d, time, from, inward, skip, any, hit);
}
