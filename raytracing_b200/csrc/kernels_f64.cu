// The books' integrator in double: the reference's precision::float64 (renderer.h:402-409), its all_books_kernel<double>
// and first_book_kernel<double> (renderer.cu:417-451), a mode "there to compare with" rather than a fast path.
//
// It renders what the reference renders in float64: the three books' scenes (spheres, moving spheres, quads, smoke,
// the solid, checker, image and marble textures) under the books' four strategies (camera.cuh:304-437, lights.cuh);
// the NEE/MIS integrator and triangle meshes compute in float only, there as here. Every number of a path is a
// double: rays, hits, normals, throughput, the random numbers (53-bit uniforms, as random_real<double> draws).
//
// The B200 form is the float pool kernel's (pool_kernel.cuh): persistent warps that keep their paths in shared memory and
// walk, shade and start them a warp's worth at a time. A finished sample's value goes to its place in a buffer, and a
// reduction of its own adds them in pass order, chunk by chunk, in the FP64 sums, so the grouping of passes into launches
// does not change the image, as in float; an image whose samples would not fit the buffer is rendered in bands of tiles.
// The tree is the float tables' (its boxes rounded outward in float); a double primitive can stand out of its float box by
// the rounding of its float copy, so every node bound is widened by the scene's box_margin, and the walk, four wide with
// its boxes tested in float, sets them out by its own rounding too (float_ray): it meets every primitive the ray meets.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.cuh"
#include "philox.cuh"
#include "rounding.cuh"
#include "rt_b200.h"

namespace rtb
{
namespace
{
using v3 = double3;

__device__ __forceinline__ v3 operator+(v3 a, v3 b) { return make_double3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ v3 operator-(v3 a, v3 b) { return make_double3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ v3 operator-(v3 a) { return make_double3(-a.x, -a.y, -a.z); }
__device__ __forceinline__ v3 operator*(double t, v3 v) { return make_double3(t * v.x, t * v.y, t * v.z); }
__device__ __forceinline__ v3 operator*(v3 a, v3 b) { return make_double3(a.x * b.x, a.y * b.y, a.z * b.z); }
// The dot products' roundings are written out (rounding.cuh), so that an image does not depend on what the compiler makes
// of a product's surroundings: path after path of mirrors and glass would grow a last bit into another image. (A
// mirror's is left to it: none of the written forms is the one its images have been rendered with.)
template <rounding R = rounding::x>
__device__ __forceinline__ double dot(v3 a, v3 b)
{
    if constexpr (R == rounding::x)
    {
        return __fma_rn(a.z, b.z, __fma_rn(a.x, b.x, __dmul_rn(a.y, b.y)));
    }
    else if constexpr (R == rounding::y)
    {
        return __fma_rn(a.z, b.z, __fma_rn(a.y, b.y, __dmul_rn(a.x, b.x)));
    }
    else if constexpr (R == rounding::yz)
    {
        return __dadd_rn(__dmul_rn(a.z, b.z), __fma_rn(a.y, b.y, __dmul_rn(a.x, b.x)));
    }
    else
    {
        return a.x * b.x + a.y * b.y + a.z * b.z;
    }
}
template <rounding R = rounding::x>
__device__ __forceinline__ double length_squared(v3 v)
{
    return dot<R>(v, v);
}
template <rounding R = rounding::x>
__device__ __forceinline__ v3 unit_vector(v3 v)
{
    return (1.0 / sqrt(length_squared<R>(v))) * v;
}
template <rounding R = rounding::x>
__device__ __forceinline__ v3 reflect(v3 v, v3 n)
{
    return v - (2.0 * dot<R>(v, n)) * n;
}
__device__ __forceinline__ v3 refract(v3 uv, v3 n, double etai_over_etat) // vec3.cuh refract
{
    const double cos_theta = fmin(dot<rounding::yz>(-uv, n), 1.0);
    const v3 r_out_perp = etai_over_etat * (uv + cos_theta * n);
    const v3 r_out_parallel = -sqrt(fabs(1.0 - length_squared(r_out_perp))) * n;
    return r_out_perp + r_out_parallel;
}
__device__ __forceinline__ v3 vec(const double* p) { return make_double3(p[0], p[1], p[2]); }

constexpr double pi_d = 3.14159265358979323846;
constexpr double uniform_sphere_density = 1.0 / (4.0 * pi_d);
constexpr double infinity_d = __builtin_huge_val();
constexpr double t_min = 0.001;

// ---- random numbers: Philox4x32-10 on the float kernel's counter, 53 bits a uniform ----------------------------------
// 53 random bits as a double in [0, 1 - 2^-53], every value k / 2^53 exactly, as random_real<double> (random.cuh:79-93)
__device__ __forceinline__ double to_unit53(uint32_t hi, uint32_t lo)
{
    return static_cast<double>((static_cast<uint64_t>(hi >> 11) << 32) | lo) * 0x1p-53;
}

struct uniforms
{
    double x, y, z, w;
};

struct sampler
{
    uint2 key;
    uint32_t pixel;
    uint32_t pass;

    // Four uniforms for dimension block `block` of the vertex at depth `depth`: two Philox blocks, the counter of the
    // float kernel's draw and the same with the job word's top bit set (a plain render's job word is 0)
    __device__ __forceinline__ uniforms draw(int depth, int block) const
    {
        const uint32_t c = (static_cast<uint32_t>(depth) << 4) | static_cast<uint32_t>(block);
        const uint4 a = philox4x32_10(make_uint4(pixel, pass, c, 0u), key);
        const uint4 b = philox4x32_10(make_uint4(pixel, pass, c, 0x80000000u), key);
        return {to_unit53(a.x, a.y), to_unit53(a.z, a.w), to_unit53(b.x, b.y), to_unit53(b.z, b.w)};
    }
};

// The float kernel's dimension blocks: 0 the material's sample (at depth 0 the camera ray's), 1 the ray's time,
// 4-15 the free flights through the volumes of smoke, four volumes a block
constexpr int block_material = 0;
constexpr int block_time = 1;
constexpr int block_media = 4;

// ---- directions (random.cuh:95-140, material.cuh:55-64, pdf.cuh:21-26) -------------------------------------------
__device__ __forceinline__ v3 random_unit_vector(double u, double v)
{
    double s, c;
    sincospi(2.0 * v, &s, &c);
    const double r = 2.0 * sqrt(u * (1.0 - u));
    return make_double3(r * c, r * s, 1.0 - 2.0 * u);
}

__device__ __forceinline__ v3 random_cosine_direction(double r1, double r2)
{
    double s, c;
    sincospi(2.0 * r1, &s, &c);
    const double sin_theta = sqrt(r2);
    return make_double3(c * sin_theta, s * sin_theta, sqrt(1.0 - r2));
}

// v in a basis whose z axis is the unit vector n (Duff et al., "Building an Orthonormal Basis, Revisited", JCGT 2017)
__device__ __forceinline__ v3 around(v3 n, v3 v)
{
    const double sign = copysign(1.0, n.z);
    const double a = -1.0 / (sign + n.z);
    const double b = n.x * n.y * a;
    const v3 x_axis = make_double3(1.0 + sign * n.x * n.x * a, sign * b, -sign * n.x);
    const v3 y_axis = make_double3(b, sign + n.y * n.y * a, -n.y);
    return v.x * x_axis + v.y * y_axis + v.z * n;
}

__device__ __forceinline__ double cosine_density(v3 unit_normal, v3 direction)
{
    const double cosine = dot(unit_normal, direction) / sqrt(length_squared(direction));
    return cosine > 0.0 ? cosine / pi_d : 0.0;
}

// Schlick's reflectance (material.cuh:67-76)
__device__ __forceinline__ double reflectance(double cosine, double ri)
{
    double r0 = (1.0 - ri) / (1.0 + ri);
    r0 = r0 * r0;
    const double x = 1.0 - cosine;
    const double x2 = x * x;
    return r0 + (1.0 - r0) * (x2 * x2 * x);
}

// ---- primitive tests -----------------------------------------------------------------------------------------------
// 1 / x, never infinite (bvh.cuh:475-488): |x| below 2^-80 moves out to +-2^-80
__device__ __forceinline__ double safe_inverse(double x)
{
    const double tiny = 0x1p-80;
    return 1.0 / (fabs(x) > tiny ? x : copysign(tiny, x));
}

// The line's two roots with a sphere in the l-vector form (sphere.cuh:70-97): (h/a) -+ sqrt(r^2 - |l|^2)/sqrt(a), the
// three squares taken from r^2 by fused multiply-adds
__device__ __forceinline__ bool sphere_roots(const sphere_d& s, v3 o, v3 d, double inverse_a, double& near,
                                             double& far)
{
    const v3 oc = make_double3(s.x - o.x, s.y - o.y, s.z - o.z);
    const double h_over_a = dot(d, oc) * inverse_a;
    const v3 l = oc - h_over_a * d;
    const double disc = fma(-l.x, l.x, fma(-l.y, l.y, fma(-l.z, l.z, s.w * s.w)));
    if (disc < 0.0)
    {
        return false;
    }
    const double half_chord = sqrt(disc * inverse_a);
    near = h_over_a - half_chord;
    far = h_over_a + half_chord;
    return true;
}

// hit_sphere (sphere.cuh:99-117): the nearest root in (t_min, t_max); far_only for the sphere the ray leaves inward
__device__ __forceinline__ bool hit_sphere(const sphere_d& s, v3 o, v3 d, double inverse_a, double lo, double hi,
                                           bool far_only, double& t, bool& entering)
{
    double near, far;
    if (!sphere_roots(s, o, d, inverse_a, near, far))
    {
        return false;
    }
    t = near;
    entering = !far_only && t > lo;
    if (!entering)
    {
        t = far;
    }
    return lo < t && t < hi;
}

struct quad_v
{
    v3 q, n, a, b;
};

__device__ __forceinline__ quad_v load_quad(const quad_d& r)
{
    return {vec(r.q), vec(r.n), vec(r.a), vec(r.b)};
}

// hit_quad (quad.cuh:60-84): t in [lo, hi], alpha and beta in [0, 1], closed; NaNs fail every comparison
__device__ __forceinline__ bool hit_quad(const quad_v& s, v3 o, v3 d, double lo, double hi, double& t, bool& front)
{
    const double denominator = dot(s.n, d);
    if (!(fabs(denominator) >= 1e-8))
    {
        return false;
    }
    const v3 origin_to_q = s.q - o;
    t = dot<rounding::y>(s.n, origin_to_q) / denominator;
    if (!(lo <= t && t <= hi))
    {
        return false;
    }
    const v3 p = t * d - origin_to_q;
    const double alpha = dot(p, s.a);
    const double beta = dot(p, s.b);
    if (!(0.0 <= alpha && alpha <= 1.0 && 0.0 <= beta && beta <= 1.0))
    {
        return false;
    }
    front = denominator < 0.0;
    return true;
}

struct hit_info
{
    int id; // global id, -1 for none
    double t;
    bool front;
};

// Sphere i (leaf order) where it is at the ray's time
__device__ __forceinline__ sphere_d sphere_at(const scene_view_f64& S, int i, double time)
{
    sphere_d s = S.spheres[i];
    if (S.has_motion)
    {
        const motion_d m = S.sphere_motion[i];
        s.x = fma(time, m.x, s.x);
        s.y = fma(time, m.y, s.y);
        s.z = fma(time, m.z, s.z);
    }
    return s;
}

// The leaf's primitives against the ray (spheres or quads: a float64 scene has no triangles), shrinking hit.t
__device__ __forceinline__ void test_leaf(const scene_view_f64& S, int link, v3 o, v3 d, double time,
                                          double inverse_a, int from, bool inward, hit_info& hit)
{
    const int kind = leaf_kind(link);
    const int count = leaf_count(link);
    const int start = leaf_start(link);
    if (kind == kind_sphere)
    {
        for (int i = start; i < start + count; ++i)
        {
            const bool own = i == from;
            if (own && !inward)
            {
                continue;
            }
            double t;
            bool entering;
            if (hit_sphere(sphere_at(S, i, time), o, d, inverse_a, t_min, hit.t, own, t, entering))
            {
                hit = {i, t, entering};
            }
        }
    }
    else
    {
        for (int i = start; i < start + count; ++i)
        {
            const int id = S.quad_base + i;
            if (id == from)
            {
                continue;
            }
            double t;
            bool front;
            if (hit_quad(load_quad(S.quads[i]), o, d, t_min, hit.t, t, front))
            {
                hit = {id, t, front};
            }
        }
    }
}

// The entry distance of the ray into a float box widened by `margin`, or +infinity if it misses it before `limit`
__device__ __forceinline__ double box_entry(float lo_x, float hi_x, float lo_y, float hi_y, float lo_z, float hi_z,
                                            double margin, v3 o, v3 inv, double limit)
{
    const double a0 = (static_cast<double>(lo_x) - margin - o.x) * inv.x;
    const double a1 = (static_cast<double>(hi_x) + margin - o.x) * inv.x;
    const double b0 = (static_cast<double>(lo_y) - margin - o.y) * inv.y;
    const double b1 = (static_cast<double>(hi_y) + margin - o.y) * inv.y;
    const double c0 = (static_cast<double>(lo_z) - margin - o.z) * inv.z;
    const double c1 = (static_cast<double>(hi_z) + margin - o.z) * inv.z;
    const double enter = fmax(fmax(fmin(a0, a1), fmin(b0, b1)), fmax(fmin(c0, c1), t_min));
    const double exit = fmin(fmin(fmax(a0, a1), fmax(b0, b1)), fmin(fmax(c0, c1), limit));
    return enter <= exit ? enter : infinity_d;
}

// The closest hit in (t_min, +inf) with the self-intersection rules of the primitive the ray leaves (bvh.cuh:539-575,
// 576-706): every primitive in turn for a flat scene, else a walk of the tree, nearer child first, with a stack of
// (node, entry distance) in local memory
__device__ hit_info closest_hit(const scene_view_f64& S, v3 o, v3 d, double time, int from, bool inward)
{
    hit_info hit{-1, infinity_d, false};
    if (S.node_count == 0)
    {
        return hit;
    }
    const double inverse_a = 1.0 / length_squared<rounding::y>(d);
    if (S.flat)
    {
        for (int i = 0; i < S.quad_base; ++i)
        {
            const bool own = i == from;
            if (own && !inward)
            {
                continue;
            }
            double t;
            bool entering;
            if (hit_sphere(sphere_at(S, i, time), o, d, inverse_a, t_min, hit.t, own, t, entering))
            {
                hit = {i, t, entering};
            }
        }
        for (int i = 0; i < S.prim_count - S.quad_base; ++i)
        {
            const int id = S.quad_base + i;
            if (id == from)
            {
                continue;
            }
            double t;
            bool front;
            if (hit_quad(load_quad(S.quads[i]), o, d, t_min, hit.t, t, front))
            {
                hit = {id, t, front};
            }
        }
        return hit;
    }
    const v3 inv = make_double3(safe_inverse(d.x), safe_inverse(d.y), safe_inverse(d.z));
    const double m = S.box_margin;
    int links[max_bvh_depth];
    double entries[max_bvh_depth];
    int sp = 0;
    int link = 0;
    while (true)
    {
        if (link >= 0)
        {
            const bvh_node& n = S.nodes[link];
            const double e0 = box_entry(n.x[0], n.x[1], n.y[0], n.y[1], n.z[0], n.z[1], m, o, inv, hit.t);
            const double e1 = box_entry(n.x[2], n.x[3], n.y[2], n.y[3], n.z[2], n.z[3], m, o, inv, hit.t);
            const bool h0 = e0 != infinity_d;
            const bool h1 = e1 != infinity_d;
            if (h0 && h1)
            {
                const bool second_first = e1 < e0;
                link = second_first ? n.link[1] : n.link[0];
                links[sp] = second_first ? n.link[0] : n.link[1];
                entries[sp] = second_first ? e0 : e1;
                ++sp;
                continue;
            }
            if (h0 || h1)
            {
                link = h0 ? n.link[0] : n.link[1];
                continue;
            }
        }
        else
        {
            test_leaf(S, link, o, d, time, inverse_a, from, inward, hit);
        }
        // The next stack entry the ray enters before the closest hit so far
        link = traversal_done_link;
        while (sp > 0)
        {
            --sp;
            if (entries[sp] < hit.t)
            {
                link = links[sp];
                break;
            }
        }
        if (link == traversal_done_link)
        {
            return hit;
        }
    }
}

// ---- volumes of smoke (constant_medium.cuh:29-120, camera.cuh:259-284) -----------------------------------------------
// Where the ray's line crosses the medium's boundary: the sphere's roots where it is at the ray's time, kept if the
// chord is longer than 0.0001; or the nearest and the farthest plane of the boundary quads the line meets inside them
__device__ bool boundary_crossings(const scene_view_f64& S, const medium_d& m, v3 o, v3 d, double time,
                                   double inverse_a, double& t_in, double& t_out)
{
    if (m.quad_count == 0)
    {
        const sphere_d s{fma(time, m.dm[0], m.c[0]), fma(time, m.dm[1], m.c[1]), fma(time, m.dm[2], m.c[2]), m.radius};
        return sphere_roots(s, o, d, inverse_a, t_in, t_out) && t_out - t_in > 0.0001;
    }
    t_in = infinity_d;
    t_out = -infinity_d;
    for (int i = m.first_quad; i < m.first_quad + m.quad_count; ++i)
    {
        double t;
        bool front;
        if (hit_quad(load_quad(S.boundary_quads[i]), o, d, -infinity_d, infinity_d, t, front))
        {
            t_in = fmin(t_in, t);
            t_out = fmax(t_out, t);
        }
    }
    return t_out - t_in >= 0.0001;
}

// The stretch [t_in, t_out] of (t_min, t_max) inside the medium: its box first, then the boundary's crossings
__device__ bool medium_stretch(const scene_view_f64& S, const medium_d& m, v3 o, v3 d, double time, double inverse_a,
                               v3 inv, double t_max, double& t_in, double& t_out)
{
    const double a0 = (m.lo[0] - o.x) * inv.x, a1 = (m.hi[0] - o.x) * inv.x;
    const double b0 = (m.lo[1] - o.y) * inv.y, b1 = (m.hi[1] - o.y) * inv.y;
    const double c0 = (m.lo[2] - o.z) * inv.z, c1 = (m.hi[2] - o.z) * inv.z;
    const double enter = fmax(fmax(fmin(a0, a1), fmin(b0, b1)), fmax(fmin(c0, c1), t_min));
    const double exit = fmin(fmin(fmax(a0, a1), fmax(b0, b1)), fmin(fmax(c0, c1), t_max));
    if (!(enter <= exit))
    {
        return false;
    }
    double line_in, line_out;
    if (!boundary_crossings(S, m, o, d, time, inverse_a, line_in, line_out))
    {
        return false;
    }
    t_in = fmax(line_in, t_min);
    t_out = fmin(line_out, t_max);
    if (!(t_in < t_out))
    {
        return false;
    }
    t_in = fmax(t_in, 0.0);
    return true;
}

// A particle of smoke in front of the closest surface (closest_event, camera.cuh:259-284): each volume in turn against
// the closest event so far, a free flight of -log(u) / density from where the ray enters it
__device__ void media_event(const scene_view_f64& S, v3 o, v3 d, double time, const sampler& rng, int depth,
                            hit_info& hit)
{
    const double inverse_a = 1.0 / length_squared<rounding::y>(d);
    const v3 inv = make_double3(safe_inverse(d.x), safe_inverse(d.y), safe_inverse(d.z));
    const double length = sqrt(length_squared<rounding::y>(d));
    uniforms u{};
    for (int k = 0; k < S.medium_count; ++k)
    {
        if ((k & 3) == 0)
        {
            u = rng.draw(depth, block_media + (k >> 2));
        }
        const medium_d& m = S.media[k];
        double t_in, t_out;
        if (!medium_stretch(S, m, o, d, time, inverse_a, inv, hit.t, t_in, t_out))
        {
            continue;
        }
        const double uk = (k & 3) == 0 ? u.x : (k & 3) == 1 ? u.y : (k & 3) == 2 ? u.z : u.w;
        const double distance = m.neg_inv_density * log(uk);
        if (distance > (t_out - t_in) * length)
        {
            continue;
        }
        hit = {S.medium_base + k, t_in + distance / length, true};
    }
}

// ---- textures (texture.cuh, perlin.cuh) ---------------------------------------------------------------------------
// Perlin noise (perlin.ixx noise): Hermite-smoothed cell coordinates, the trilinear sum of the corners' gradient dot
// products; turbulence: 7 octaves, each at twice the frequency and half the weight, absolute value
__device__ double perlin_noise(const noise_d& n, v3 p)
{
    const double fx = floor(p.x), fy = floor(p.y), fz = floor(p.z);
    const int i = static_cast<int>(fx), j = static_cast<int>(fy), k = static_cast<int>(fz);
    const double u = p.x - fx, v = p.y - fy, w = p.z - fz;
    const double uu = u * u * (3.0 - 2.0 * u);
    const double vv = v * v * (3.0 - 2.0 * v);
    const double ww = w * w * (3.0 - 2.0 * w);
    double accum = 0.0;
    for (int di = 0; di < 2; ++di)
    {
        const int px = n.perm_x[(i + di) & 255];
        const double wx = di == 0 ? 1.0 - uu : uu;
        for (int dj = 0; dj < 2; ++dj)
        {
            const int py = n.perm_y[(j + dj) & 255];
            const double wy = dj == 0 ? 1.0 - vv : vv;
            for (int dk = 0; dk < 2; ++dk)
            {
                const int pz = n.perm_z[(k + dk) & 255];
                const double wz = dk == 0 ? 1.0 - ww : ww;
                const d4& g = n.gradients[px ^ py ^ pz];
                const double dot_g = g.x * (u - di) + g.y * (v - dj) + g.z * (w - dk);
                accum += wx * wy * wz * dot_g;
            }
        }
    }
    return accum;
}

__device__ double turbulence(const noise_d& n, v3 p)
{
    double accum = 0.0;
    double weight = 1.0;
    for (int layer = 0; layer < 7; ++layer)
    {
        accum += weight * perlin_noise(n, p);
        weight *= 0.5;
        p = 2.0 * p;
    }
    return fabs(accum);
}

// The texture's color at the hit (texture_value, texture.cuh:60-110): a checker walked down to its point's cube, an
// image read at (u, v) clamped with v flipped, a marble 0.5 (1 + sin(scale z + 10 turbulence(p)))
__device__ v3 texture_value(const scene_view_f64& S, int index, double u, double v, v3 p)
{
    texture_d t = S.textures[index];
    while (t.kind == RT_TEXTURE_CHECKER)
    {
        const int x = static_cast<int>(floor(t.inv_scale * p.x));
        const int y = static_cast<int>(floor(t.inv_scale * p.y));
        const int z = static_cast<int>(floor(t.inv_scale * p.z));
        t = S.textures[(x + y + z) % 2 == 0 ? t.even : t.odd];
    }
    if (t.kind == RT_TEXTURE_IMAGE)
    {
        const image_info im = S.images[t.table];
        const double cu = fmin(fmax(u, 0.0), 1.0);
        const double fv = 1.0 - fmin(fmax(v, 0.0), 1.0);
        const int column = static_cast<int>(cu * im.width);
        const int row = static_cast<int>(fv * im.height);
        const int i = column < im.width - 1 ? column : im.width - 1;
        const int j = row < im.height - 1 ? row : im.height - 1;
        const float4 c = S.texels[im.offset + j * im.width + i];
        return make_double3(c.x, c.y, c.z);
    }
    if (t.kind == RT_TEXTURE_NOISE)
    {
        const noise_d& n = S.noises[t.table];
        const double gray = 0.5 * (1.0 + sin(n.scale * p.z + 10.0 * turbulence(n, p)));
        return make_double3(gray, gray, gray);
    }
    return make_double3(t.r, t.g, t.b);
}

// ---- the books' lights list (lights.cuh:49-227) --------------------------------------------------------------------
__device__ __forceinline__ double one_minus_cos_theta_max(double radius, double distance_squared)
{
    const double sin_squared = radius * radius / distance_squared;
    return sin_squared / (1.0 + sqrt(1.0 - sin_squared));
}

__device__ double lights_pdf_value(const scene_view_f64& S, v3 origin, v3 direction, int from)
{
    double sum = 0.0;
    for (int k = 0; k < S.light_count; ++k)
    {
        const light_d& l = S.lights[k];
        const bool own = from >= 0 && l.twin == from;
        if (l.kind == RT_LIGHT_QUAD)
        {
            if (own)
            {
                continue; // a ray never hits the quad it leaves (the twin rule, lights.cuh:175-187)
            }
            double t;
            bool front;
            if (!hit_quad(load_quad(l.quad), origin, direction, t_min, infinity_d, t, front))
            {
                continue;
            }
            const double len2 = length_squared(direction);
            const double distance_squared = t * t * len2;
            const double cosine = fabs(dot(direction, vec(l.quad.n))) / sqrt(len2);
            sum += l.weight * (distance_squared / (cosine * l.area));
        }
        else
        {
            const v3 c = vec(l.c);
            const v3 to_center = c - origin;
            const double distance_squared = length_squared(to_center);
            if (distance_squared < l.radius * l.radius)
            {
                sum += l.weight * uniform_sphere_density;
                continue;
            }
            if (own && !(dot(direction, to_center) > 0.0))
            {
                continue;
            }
            double t;
            bool entering;
            if (!hit_sphere(sphere_d{c.x, c.y, c.z, l.radius}, origin, direction, 1.0 / length_squared(direction),
                            t_min, infinity_d, own, t, entering))
            {
                continue;
            }
            sum += l.weight * (1.0 / (2.0 * pi_d * one_minus_cos_theta_max(l.radius, distance_squared)));
        }
    }
    return sum;
}

// lights_random: the running sums pick a light with `pick`; (a, b) draw its point or direction
__device__ v3 lights_random(const scene_view_f64& S, v3 origin, double pick, double a, double b)
{
    int k = 0;
    while (k < S.light_count - 1 && !(pick < S.lights[k].cdf))
    {
        ++k;
    }
    const light_d& l = S.lights[k];
    if (l.kind == RT_LIGHT_QUAD)
    {
        return unit_vector((vec(l.quad.q) - origin) + a * vec(l.u) + b * vec(l.v));
    }
    const v3 to_center = vec(l.c) - origin;
    const double distance_squared = length_squared(to_center);
    if (distance_squared < l.radius * l.radius)
    {
        return random_unit_vector(a, b);
    }
    const double one_minus_cos_max = one_minus_cos_theta_max(l.radius, distance_squared);
    double s, c;
    sincospi(2.0 * a, &s, &c);
    const double one_minus_z = b * one_minus_cos_max;
    const double sin_theta = sqrt(one_minus_z * (2.0 - one_minus_z));
    return around((1.0 / sqrt(distance_squared)) * to_center,
                  make_double3(c * sin_theta, s * sin_theta, 1.0 - one_minus_z));
}

// ---- the camera (camera.cuh:53-107) ---------------------------------------------------------------------------------
__device__ __forceinline__ void camera_ray(const camera_d& cam, int i, int j, int s_i, int s_j, const uniforms& u,
                                           v3& origin, v3& direction)
{
    const double dx = (s_i + u.x) * cam.recip_sqrt_spp - 0.5;
    const double dy = (s_j + u.y) * cam.recip_sqrt_spp - 0.5;
    const v3 to_sample = vec(cam.to_pixel00) + (i + dx) * vec(cam.delta_u) + (j + dy) * vec(cam.delta_v);
    origin = vec(cam.center);
    direction = to_sample;
    if (cam.defocus)
    {
        const double r = sqrt(u.z);
        double s, c;
        sincospi(2.0 * u.w, &s, &c);
        const v3 lens = (r * c) * vec(cam.disk_u) + (r * s) * vec(cam.disk_v);
        origin = origin + lens;
        direction = to_sample - lens;
    }
}

__device__ __forceinline__ v3 sky(const camera_d& cam, v3 direction)
{
    const double a = 0.5 * (unit_vector<rounding::y>(direction).y + 1.0);
    return (1.0 - a) * vec(cam.sky_bottom) + a * vec(cam.sky_top);
}

__device__ __forceinline__ double without_nan(double x) { return x == x ? x : 0.0; }

struct path_state
{
    v3 o, d;
    v3 throughput;
    int rays_left;
    int depth;
    int from;
    bool inward;
    double time;
};

struct surface
{
    v3 p;
    v3 outward;
    v3 normal;
    v3 color;
    int material;
    int from;
};

// A sphere point's texture coordinates (sphere.cuh:119-135): its outward normal turned back by the instances' turn,
// u from -x around y, v from the south pole
__device__ __forceinline__ void sphere_uv(v3 outward, const frame_d& f, double& u, double& v)
{
    const double nx = f.x * outward.x - f.y * outward.z;
    const double nz = f.y * outward.x + f.x * outward.z;
    const double phi = atan2(-nz, nx) + pi_d;
    const double theta = acos(fmin(fmax(-outward.y, -1.0), 1.0));
    u = phi / (2.0 * pi_d);
    v = theta / pi_d;
}

// The hit point moved onto the sphere by one Newton step, for a checker (onto_sphere, sphere.cuh:137-168): f = |p|^2
// - 2 p.c + k with k = |c|^2 - r^2 from the host, taken while its rounding bound stays below the frame's limit
__device__ __forceinline__ v3 onto_sphere(v3 p, v3 outward, const sphere_d& ball, const frame_d& f)
{
    const v3 c = make_double3(ball.x, ball.y, ball.z);
    const double p_p = dot(p, p);
    const double p_c = dot(p, c);
    if (!(p_p + 2.0 * fabs(p_c) + fabs(f.z) < f.w))
    {
        return p;
    }
    const double value = p_p - 2.0 * p_c + f.z;
    return p - (value / (2.0 * ball.w)) * outward;
}

// The hit as the shading needs it (surface_at, camera.cuh:171-253) and the material there with its color
__device__ surface surface_at(const scene_view_f64& S, const path_state& ps, const hit_info& h, material_d& m)
{
    surface s;
    s.from = h.id;
    double u = 0.0, v = 0.0;
    sphere_d ball{};
    bool on_sphere = false;
    if (h.id >= S.medium_base)
    {
        // A particle of smoke: any normal will do, the CPU's (1, 0, 0) and the front; no surface to leave
        s.p = ps.o + h.t * ps.d;
        s.outward = make_double3(1.0, 0.0, 0.0);
        s.normal = s.outward;
        s.material = S.media[h.id - S.medium_base].material;
        s.from = -1;
        m = S.materials[s.material];
    }
    else
    {
        s.material = S.prim_material[h.id];
        m = S.materials[s.material];
        if (h.id < S.quad_base)
        {
            ball = sphere_at(S, h.id, ps.time);
            on_sphere = true;
            s.p = ps.o + h.t * ps.d;
            s.outward = (1.0 / ball.w) * (s.p - make_double3(ball.x, ball.y, ball.z));
        }
        else
        {
            // The quad's point as the CPU computes it, t * d rounded, then the sum (camera.cuh:175-195 at_unfused)
            const quad_v q = load_quad(S.quads[h.id - S.quad_base]);
            s.p = make_double3(__dadd_rn(ps.o.x, __dmul_rn(h.t, ps.d.x)), __dadd_rn(ps.o.y, __dmul_rn(h.t, ps.d.y)),
                               __dadd_rn(ps.o.z, __dmul_rn(h.t, ps.d.z)));
            s.outward = q.n;
            if (m.texture >= 0 && (m.texture_needs & texture_needs_uv) != 0)
            {
                const v3 rel = h.t * ps.d - (q.q - ps.o);
                u = dot(rel, q.a);
                v = dot(rel, q.b);
            }
        }
        s.normal = h.front ? s.outward : -s.outward;
    }
    s.color = make_double3(m.r, m.g, m.b);
    if (m.texture >= 0)
    {
        v3 point = s.p;
        if (on_sphere && (m.texture_needs & (texture_needs_uv | texture_needs_point)) != 0)
        {
            const frame_d f = S.sphere_frames[h.id];
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

// One segment of a books' path after its closest event (camera.cuh:364-437 trace_ray, diffuse_bounce 304-359,
// material.cuh:84-126 scatter): true when the sample is done, its value in `sample`
__device__ bool shade_books(const scene_view_f64& S, const camera_d& cam, const sampler& rng, path_state& ps,
                            const hit_info& h, v3& sample)
{
    const v3 black = make_double3(0.0, 0.0, 0.0);
    if (h.id < 0)
    {
        sample = ps.throughput * sky(cam, ps.d);
        return true;
    }
    material_d m;
    const surface s = surface_at(S, ps, h, m);
    const v3 albedo = s.color;
    v3 direction;
    if (m.kind == RT_DIFFUSE_LIGHT)
    {
        sample = h.front ? ps.throughput * albedo : black;
        return true;
    }
    const uniforms u = rng.draw(ps.depth, block_material);
    if (m.kind == RT_LAMBERTIAN || m.kind == RT_ISOTROPIC)
    {
        // A diffuse bounce: a matte surface, or a particle of smoke, which keeps its own density 1/(4 pi) except under
        // the lights strategy (isotropic::mixes_in_lights is false)
        const bool matte = m.kind == RT_LAMBERTIAN;
        int strategy = cam.sampling;
        if (!matte && strategy != RT_SAMPLING_LIGHTS)
        {
            strategy = RT_SAMPLING_MATERIAL;
        }
        if (strategy == RT_SAMPLING_MATERIAL)
        {
            direction = matte ? around(s.normal, random_cosine_direction(u.x, u.y)) : random_unit_vector(u.x, u.y);
            if (matte && !(dot(s.normal, direction) > 0.0))
            {
                sample = black;
                return true;
            }
            ps.throughput = ps.throughput * albedo;
        }
        else
        {
            bool toward_lights = strategy == RT_SAMPLING_LIGHTS;
            if (strategy == RT_SAMPLING_MIXTURE)
            {
                toward_lights = u.z < 0.5;
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
            const double p_scatter = matte ? cosine_density(s.normal, direction) : uniform_sphere_density;
            double p = uniform_sphere_density;
            if (strategy != RT_SAMPLING_UNIFORM)
            {
                const double p_lights = lights_pdf_value(S, s.p, direction, s.from);
                p = strategy == RT_SAMPLING_LIGHTS ? p_lights : 0.5 * p_lights + 0.5 * p_scatter;
            }
            if (!(p > 0.0) || !(p_scatter > 0.0))
            {
                sample = black;
                return true;
            }
            ps.throughput = (p_scatter / p) * (ps.throughput * albedo);
        }
    }
    else if (m.kind == RT_METAL)
    {
        direction = unit_vector<rounding::compiler>(reflect(ps.d, s.normal)) + m.fuzz * random_unit_vector(u.x, u.y);
        if (dot(direction, s.normal) <= 0.0)
        {
            sample = black;
            return true;
        }
        ps.throughput = ps.throughput * albedo;
    }
    else // dielectric
    {
        const double ri = h.front ? 1.0 / m.ior : m.ior;
        const v3 ud = unit_vector<rounding::y>(ps.d);
        const double cos_theta = fmin(dot<rounding::yz>(-ud, s.normal), 1.0);
        const double sin_theta = sqrt(1.0 - cos_theta * cos_theta);
        const bool cannot_refract = ri * sin_theta > 1.0;
        direction = cannot_refract || reflectance(cos_theta, ri) > u.z ? reflect<rounding::yz>(ud, s.normal)
                                                                       : refract(ud, s.normal, ri);
    }
    if (--ps.rays_left == 0)
    {
        sample = black;
        return true;
    }
    ps.o = s.p;
    ps.d = direction;
    ps.from = s.from;
    ps.inward = dot(direction, s.outward) < 0.0;
    return false;
}

// ---- the pool kernel in double ----------------------------------------------------------------------------------
// The float pool kernel's form (pool_kernel.cuh): a persistent warp keeps 64 paths in shared memory and walks, shades
// and starts them a warp's worth at a time; each finished sample's value goes to its place in a buffer that
// reduce_f64_kernel adds up in pass order, chunk by chunk. Against a persistent kernel with a path bound to each lane
// (162 registers, 12 warps a multiprocessor, walks and materials of a warp's lanes one after the other).
constexpr unsigned full_warp = 0xffffffffu;
constexpr int pool_paths = 64;
constexpr int pool_refill = 20;
constexpr long long sample_tied = 0x7ff8000000000001ll; // a NaN, which no finished sample's value is

struct pool_record
{
    double o[3][pool_paths], d[3][pool_paths], throughput[3][pool_paths];
    double time[pool_paths], hit_t[pool_paths];
    uint32_t pixel[pool_paths], pass[pool_paths], key[pool_paths], sample[pool_paths];
    uint32_t meta[pool_paths]; // depth << 1 | the ray starts inside the surface it leaves
    int32_t from[pool_paths];
    int32_t hit[pool_paths]; // id << 1 | front, or -1
    uint8_t walk[pool_paths], shade[pool_paths], free[pool_paths];
};

// A ray against the tree four wide in float: conservative, so that the walk meets every primitive the ray meets in
// double. A plane at n is met at T = (n - o) / d; fmaf(n, inv, -c) is off it by at most 2^-24 (2 |T| + 4 |o / d|), the
// direction's reciprocal, the origin and two products rounded; the near bound is set back and the far bound out by
// 2^-20 |o / d| and the boxes' margin, and what is proportional to T by a factor of 1 + 2^-20 on the entry's side.
struct float_ray
{
    float3 inv, near, far; // a near plane is met at fmaf(n, inv, -near), a far one at fmaf(n, inv, -far)
    uint32_t x, y, z;      // where the near bounds of an axis lie in a node (the far ones 16 bytes off)
};

__device__ __forceinline__ float_ray float_ray_of(v3 o, v3 d, double margin)
{
    const v3 inv = make_double3(safe_inverse(d.x), safe_inverse(d.y), safe_inverse(d.z));
    const auto axis = [&](double oa, double ia, float& f, float& near, float& far) {
        f = static_cast<float>(ia);
        const float os = static_cast<float>(oa) * f;
        const float w = fmaf(fabsf(os), 0x1p-20f, __double2float_ru(margin) * fabsf(f) * 1.001f);
        near = os + w;
        far = os - w;
    };
    float_ray r;
    axis(o.x, inv.x, r.inv.x, r.near.x, r.far.x);
    axis(o.y, inv.y, r.inv.y, r.near.y, r.far.y);
    axis(o.z, inv.z, r.inv.z, r.near.z, r.far.z);
    r.x = inv.x < 0.0 ? 16u : 0u;
    r.y = inv.y < 0.0 ? 48u : 32u;
    r.z = inv.z < 0.0 ? 80u : 64u;
    return r;
}

// STEPS: walks of the tree four wide, a lane's resumed from phase to phase; otherwise a whole search a phase
// (closest_hit: a flat scene, or a tree too deep to be four wide).
// Which of several primitives at one distance is the hit follows from the order of the walk, and the order is that of
// closest_hit, which walks the two-wide tree: a path whose four-wide walk meets another primitive at its hit's distance
// is dropped, its sample marked and the launch's flag raised, and a launch with AGAIN renders the marked samples by
// closest_hit. (GPU time before and after: weekend 400x225 x 32 1.30 and 1.31 ms, bouncing 1.58 and 1.57, final 300x300 x
// 32, where edges of neighbouring boxes meet, 5.10 and 5.70. The second search in the four-wide kernel itself, as rare
// as it is, spilled registers: 1.38, 1.64 and 5.72.)
template <bool STEPS, bool AGAIN = false>
__global__ void __launch_bounds__(render_block, 4) pool_f64_kernel(const __grid_constant__ launch_params_f64 P)
{
    if (AGAIN && *P.tied == 0ull)
    {
        return;
    }
    extern __shared__ __align__(16) unsigned char shared[];
    pool_record& R = reinterpret_cast<pool_record*>(shared)[threadIdx.x >> 5];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lanes_below = (1u << lane) - 1u;
    const camera_d& cam = P.cam;
    const scene_view_f64& S = P.scene;
    const auto put = [](double (*rows)[pool_paths], int p, v3 v) {
        rows[0][p] = v.x;
        rows[1][p] = v.y;
        rows[2][p] = v.z;
    };
    const auto get = [](const double (*rows)[pool_paths], int p) {
        return make_double3(rows[0][p], rows[1][p], rows[2][p]);
    };
    const auto push = [&](uint8_t* list, int count, bool which, int p) -> int {
        const unsigned lanes = __ballot_sync(full_warp, which);
        if (which)
        {
            list[count + __popc(lanes & lanes_below)] = static_cast<uint8_t>(p);
        }
        return count + __popc(lanes);
    };
    for (int p = static_cast<int>(lane); p < pool_paths; p += 32)
    {
        R.free[p] = static_cast<uint8_t>(p);
    }
    __syncwarp();
    int walk_count = 0, shade_count = 0, free_count = pool_paths;
    auto limit = static_cast<unsigned long long>(P.sample_count);
    unsigned long long own_next = 0; // AGAIN: a warp's own range of the samples
    if constexpr (AGAIN)
    {
        const unsigned long long warps = gridDim.x * (render_block / 32ull);
        const unsigned long long share = (limit + warps - 1) / warps;
        own_next = share * (blockIdx.x * (render_block / 32ull) + (threadIdx.x >> 5));
        limit = min(limit, own_next + share);
    }
    bool dry = own_next >= limit;
    uint32_t rays = 0;
    int slot = -1; // the path this lane walks for
    int link = traversal_done_link;
    int sp = 0;
    hit_info hit{-1, infinity_d, false};
    bool tied = false;
    int2 stack[STEPS ? wide_stack : 1];
    while (true)
    {
        enum class phase
        {
            walk,
            start,
            shade,
            end
        } next;
        if constexpr (STEPS)
        {
            bool answered = slot >= 0 && link == traversal_done_link;
            if (__any_sync(full_warp, answered && tied))
            {
                const bool drop = answered && tied;
                if (drop)
                {
                    P.samples[3 * static_cast<int64_t>(R.sample[slot])] = __longlong_as_double(sample_tied);
                    *P.tied = 1ull;
                }
                rays -= __reduce_add_sync(full_warp, drop ? (R.meta[slot] >> 1) + 1u : 0u); // counted again with its sample
                free_count = push(R.free, free_count, drop, slot);
                answered = answered && !drop;
                slot = drop ? -1 : slot;
            }
            if (answered)
            {
                R.hit_t[slot] = hit.t;
                R.hit[slot] = hit.id < 0 ? -1 : (hit.id << 1) | (hit.front ? 1 : 0);
            }
            shade_count = push(R.shade, shade_count, answered, slot);
            slot = answered ? -1 : slot;
            const unsigned idle = __ballot_sync(full_warp, slot < 0);
            const int taken = min(__popc(idle), walk_count);
            const int rank = __popc(idle & lanes_below);
            __syncwarp();
            if (slot < 0 && rank < taken)
            {
                slot = R.walk[walk_count - 1 - rank];
                hit = {-1, infinity_d, false};
                tied = false;
                sp = 0;
                link = 0;
            }
            walk_count -= taken;
            const int startable = dry ? 0 : free_count;
            const int walking = __popc(__ballot_sync(full_warp, slot >= 0));
            const bool few = walking < pool_refill && walking * 8 < (walking + shade_count + startable) * 5;
            next = walk_count == 0 && few ? (startable > shade_count ? phase::start : phase::shade)
                   : walking > 0          ? phase::walk
                                          : phase::end;
        }
        else
        {
            const int startable = dry ? 0 : free_count;
            if (walk_count >= 32 || (walk_count >= startable && walk_count >= shade_count))
            {
                next = walk_count > 0 ? phase::walk : phase::end;
            }
            else
            {
                next = startable > shade_count ? phase::start : phase::shade;
            }
        }
        if (next == phase::end)
        {
            break;
        }
        if (next == phase::walk && !STEPS)
        {
            const int taken = min(32, walk_count);
            const bool mine = static_cast<int>(lane) < taken;
            const int p = mine ? R.walk[walk_count - taken + static_cast<int>(lane)] : 0;
            walk_count -= taken;
            if (mine)
            {
                const hit_info h = closest_hit(S, get(R.o, p), get(R.d, p), R.time[p], R.from[p], (R.meta[p] & 1u) != 0u);
                R.hit_t[p] = h.t;
                R.hit[p] = h.id < 0 ? -1 : (h.id << 1) | (h.front ? 1 : 0);
            }
            shade_count = push(R.shade, shade_count, mine, p);
            __syncwarp();
            continue;
        }
        if (next == phase::walk)
        {
            const bool walks = slot >= 0;
            const int p = walks ? slot : 0;
            const float_ray r = float_ray_of(get(R.o, p), get(R.d, p), S.box_margin);
            float bound = __double2float_ru(hit.t); // the closest hit so far, rounded up
            const auto pop = [&]() -> int {
                while (sp > 0)
                {
                    const int2 e = stack[--sp];
                    if (__int_as_float(e.y) < bound)
                    {
                        return e.x;
                    }
                }
                return traversal_done_link;
            };
            const int total =
                __popc(__ballot_sync(full_warp, walks)) + walk_count + shade_count + (dry ? 0 : free_count);
            const int enough = min(pool_refill, (total * 5 + 7) / 8);
            while (true)
            {
                while (__any_sync(full_warp, walks && link >= 0))
                {
                    if (walks && link >= 0)
                    {
                        const char* const node = reinterpret_cast<const char*>(S.wide_nodes + link);
                        const auto row = [&](uint32_t at) { return __ldg(reinterpret_cast<const float4*>(node + at)); };
                        const float4 nx = row(r.x), fx = row(r.x ^ 16u);
                        const float4 ny = row(r.y), fy = row(r.y ^ 16u);
                        const float4 nz = row(r.z), fz = row(r.z ^ 16u);
                        const int4 nl = __ldg(reinterpret_cast<const int4*>(S.wide_nodes[link].link));
                        const auto entry = [&](float ax, float bx, float ay, float by, float az, float bz,
                                               int child) -> float {
                            const float enter =
                                0x1.ffffep-1f * fmaxf(fmaxf(fmaf(ax, r.inv.x, -r.near.x), fmaf(ay, r.inv.y, -r.near.y)),
                                                      fmaxf(fmaf(az, r.inv.z, -r.near.z), 0.00099f));
                            const float exit = fminf(fminf(fmaf(bx, r.inv.x, -r.far.x), fmaf(by, r.inv.y, -r.far.y)),
                                                     fminf(fmaf(bz, r.inv.z, -r.far.z), bound));
                            return enter <= exit * 0x1.00001p+0f && child != traversal_done_link
                                       ? enter
                                       : __int_as_float(0x7f800000);
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
                        const auto met = [](float k) { return k < __int_as_float(0x7f800000); };
                        if (met(k3))
                        {
                            stack[sp++] = make_int2(l3, __float_as_int(k3));
                        }
                        if (met(k2))
                        {
                            stack[sp++] = make_int2(l2, __float_as_int(k2));
                        }
                        if (met(k1))
                        {
                            stack[sp++] = make_int2(l1, __float_as_int(k1));
                        }
                        link = met(k0) ? l0 : pop();
                    }
                }
                // every walking lane holds a leaf, or is done
                if (walks && link != traversal_done_link)
                {
                    const v3 d = get(R.d, p);
                    // the leaf's own closest hit, up to a last bit beyond the closest so far: a sphere's interval is open
                    hit_info found{-1, hit.t * 0x1.0000000000001p+0, false};
                    test_leaf(S, link, get(R.o, p), d, R.time[p], 1.0 / length_squared<rounding::y>(d), R.from[p],
                              (R.meta[p] & 1u) != 0u, found);
                    if (found.t < hit.t)
                    {
                        hit = found;
                        tied = false;
                    }
                    else
                    {
                        tied = tied || (found.id >= 0 && found.t == hit.t);
                    }
                    bound = __double2float_ru(hit.t);
                    link = pop();
                }
                if (__popc(__ballot_sync(full_warp, walks && link != traversal_done_link)) < enough)
                {
                    break;
                }
            }
            __syncwarp();
            continue;
        }
        if (next == phase::start)
        {
            const int wanted = min(min(32, free_count), P.claim);
            unsigned long long base = 0;
            if constexpr (AGAIN)
            {
                base = own_next;
                own_next += wanted;
            }
            else
            {
                if (lane == 0u)
                {
                    base = atomicAdd(P.work_counter, static_cast<unsigned long long>(wanted));
                }
                base = __shfl_sync(full_warp, base, 0);
            }
            dry = base + static_cast<unsigned long long>(wanted) >= limit;
            const unsigned long long s = base + lane;
            bool started = static_cast<int>(lane) < wanted && s < limit &&
                           (!AGAIN || __double_as_longlong(P.samples[3 * s]) == sample_tied);
            int px = 0, py = 0;
            int64_t pass = 0;
            if (started)
            {
                // sample s: pass-major, then the pixels in 8 x 4 tiles; off the image for a tile over its edge
                const auto band = static_cast<unsigned long long>(P.band_pixels);
                const int q = P.first_pixel + static_cast<int>(s % band);
                pass = P.pass_begin + static_cast<int64_t>(s / band);
                const int tile = q >> 5;
                px = (tile % P.tiles_x) * 8 + (q & 7);
                py = (tile / P.tiles_x) * 4 + ((q & 31) >> 3);
                started = px < cam.width && py < cam.height;
            }
            const unsigned lanes = __ballot_sync(full_warp, started);
            const int p = started ? R.free[free_count - 1 - __popc(lanes & lanes_below)] : 0;
            __syncwarp();
            free_count -= __popc(lanes);
            if (started)
            {
                // Pass n is pass n % k^2 of round n / k^2, whose numbers come from seed + round * 2^32
                const int64_t round = pass / P.round_passes;
                const int in_round = static_cast<int>(pass - round * P.round_passes);
                const uint64_t key = P.seed + (static_cast<uint64_t>(round) << 32);
                sampler rng;
                rng.key = make_uint2(static_cast<uint32_t>(key), static_cast<uint32_t>(key >> 32));
                rng.pass = static_cast<uint32_t>(in_round);
                rng.pixel = static_cast<uint32_t>(py) * static_cast<uint32_t>(cam.width) + static_cast<uint32_t>(px);
                v3 o, d;
                camera_ray(cam, px, py, in_round % cam.sqrt_spp, in_round / cam.sqrt_spp, rng.draw(0, block_material), o,
                           d);
                put(R.o, p, o);
                put(R.d, p, d);
                put(R.throughput, p, make_double3(1.0, 1.0, 1.0));
                R.time[p] = S.has_motion ? rng.draw(0, block_time).x : 0.0;
                R.pixel[p] = rng.pixel;
                R.pass[p] = rng.pass;
                R.key[p] = rng.key.y;
                R.sample[p] = static_cast<uint32_t>(s);
                R.meta[p] = 0u;
                R.from[p] = -1;
            }
            walk_count = push(R.walk, walk_count, started, p);
            rays += static_cast<uint32_t>(__popc(lanes));
            __syncwarp();
            continue;
        }
        const int taken = min(32, shade_count);
        const bool mine = static_cast<int>(lane) < taken;
        const int p = mine ? R.shade[shade_count - taken + static_cast<int>(lane)] : 0;
        shade_count -= taken;
        bool goes_on = false;
        if (mine)
        {
            path_state ps;
            ps.o = get(R.o, p);
            ps.d = get(R.d, p);
            ps.throughput = get(R.throughput, p);
            ps.time = R.time[p];
            ps.depth = static_cast<int>(R.meta[p] >> 1);
            ps.inward = (R.meta[p] & 1u) != 0u;
            ps.rays_left = cam.max_depth - ps.depth;
            ps.from = R.from[p];
            sampler rng;
            rng.pixel = R.pixel[p];
            rng.pass = R.pass[p];
            rng.key = make_uint2(static_cast<uint32_t>(P.seed), R.key[p]);
            const int answer = R.hit[p];
            hit_info h{answer < 0 ? -1 : answer >> 1, R.hit_t[p], (answer & 1) != 0};
            ++ps.depth;
            if (S.medium_count > 0)
            {
                media_event(S, ps.o, ps.d, ps.time, rng, ps.depth, h);
            }
            v3 sample;
            goes_on = !shade_books(S, cam, rng, ps, h, sample);
            if (goes_on)
            {
                put(R.o, p, ps.o);
                put(R.d, p, ps.d);
                put(R.throughput, p, ps.throughput);
                R.meta[p] = (static_cast<uint32_t>(ps.depth) << 1) | (ps.inward ? 1u : 0u);
                R.from[p] = ps.from;
            }
            else
            {
                double* const out = P.samples + 3 * static_cast<int64_t>(R.sample[p]);
                out[0] = without_nan(sample.x);
                out[1] = without_nan(sample.y);
                out[2] = without_nan(sample.z);
            }
        }
        walk_count = push(R.walk, walk_count, goes_on, p);
        free_count = push(R.free, free_count, mine && !goes_on, p);
        rays += static_cast<uint32_t>(__popc(__ballot_sync(full_warp, goes_on)));
        __syncwarp();
    }
    if (lane == 0u && rays != 0u)
    {
        atomicAdd(P.counters, static_cast<unsigned long long>(rays));
    }
}

// The launch's samples into the image's sums: each chunk's in pass order into its partial, the partials in chunk order
// (the rows from first_y down that the band has pixels in)
__global__ void reduce_f64_kernel(const __grid_constant__ launch_params_f64 P, int first_y, double* sums)
{
    const int x = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    const int y = first_y + static_cast<int>(blockIdx.y);
    if (x >= P.cam.width || y >= P.cam.height)
    {
        return;
    }
    const int q = ((y >> 2) * P.tiles_x + (x >> 3)) * 32 + ((y & 3) << 3) + (x & 7) - P.first_pixel;
    if (q < 0 || q >= P.band_pixels)
    {
        return;
    }
    double* const sum = sums + 3 * (static_cast<int64_t>(y) * P.cam.width + x);
    double r = sum[0], g = sum[1], b = sum[2];
    for (int64_t pass = P.pass_begin; pass < P.pass_end;)
    {
        const int64_t chunk_end = (pass / P.chunk + 1) * P.chunk;
        const int64_t end = chunk_end < P.pass_end ? chunk_end : P.pass_end;
        double pr = 0.0, pg = 0.0, pb = 0.0;
        for (; pass < end; ++pass)
        {
            const double* const s = P.samples + 3 * ((pass - P.pass_begin) * P.band_pixels + q);
            pr += s[0];
            pg += s[1];
            pb += s[2];
        }
        r += pr;
        g += pg;
        b += pb;
    }
    sum[0] = r;
    sum[1] = g;
    sum[2] = b;
}

using pool_f64_function = void (*)(launch_params_f64);

bool walks_wide(const scene_view_f64& scene)
{
    return scene.flat == 0 && scene.wide_nodes != nullptr && scene.node_count > 0;
}

pool_f64_function pool_f64_of(const scene_view_f64& scene)
{
    return walks_wide(scene) ? pool_f64_kernel<true> : pool_f64_kernel<false>;
}

constexpr int pool_f64_shared = render_block / 32 * static_cast<int>(sizeof(pool_record));
} // namespace

cudaError_t launch_render_f64(const launch_params_f64& p, int grid, cudaStream_t stream, int32_t& kernels)
{
    launch_params_f64 q = p;
    const pool_launch l = pool_launch_of(p.sample_count, grid);
    q.claim = l.claim;
    if (const cudaError_t e = prepare_pool(p.work_counter, stream); e != cudaSuccess)
    {
        return e;
    }
    pool_f64_of(p.scene)<<<l.blocks, render_block, pool_f64_shared, stream>>>(q);
    kernels += 2;
    if (walks_wide(p.scene))
    {
        q.claim = 32;
        pool_f64_kernel<false, true><<<l.blocks, render_block, pool_f64_shared, stream>>>(q);
        ++kernels;
    }
    return cudaGetLastError();
}

cudaError_t launch_reduce_f64(const launch_params_f64& p, double* sums, cudaStream_t stream)
{
    const dim3 block(128, 1);
    const int64_t row = int64_t{p.tiles_x} * 32; // the padded pixels of a row of tiles, four rows of pixels
    const int first_y = static_cast<int>(p.first_pixel / row * 4);
    const int end_y =
        static_cast<int>(std::min<int64_t>(p.cam.height, (int64_t{p.first_pixel} + p.band_pixels + row - 1) / row * 4));
    const dim3 grid(static_cast<unsigned>((p.cam.width + 127) / 128), static_cast<unsigned>(end_y - first_y));
    reduce_f64_kernel<<<grid, block, 0, stream>>>(p, first_y, sums);
    return cudaGetLastError();
}

cudaError_t render_f64_attributes(const scene_view_f64& scene, kernel_attributes& out)
{
    return function_attributes(reinterpret_cast<const void*>(pool_f64_of(scene)), out, pool_f64_shared);
}
} // namespace rtb
