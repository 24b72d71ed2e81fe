// How the dot products of path.cuh are rounded in the kernels that include it. A source includes this first, names its
// table `rounds`, then includes path.cuh.
#pragma once

namespace rtb
{
enum class rounding
{
    compiler, // a.x * b.x + a.y * b.y + a.z * b.z, fused as the compiler chooses
    x,        // x fused onto y's product, z onto both
    y,        // y fused onto x's product, z onto both
    yz,       // y fused onto x's product, z's product rounded and added
};

// The kernels of kernels.cu: left to the compiler
struct rounds_compiler
{
    static constexpr bool bare = false;
    static constexpr rounding other = rounding::compiler;
    static constexpr rounding sky = rounding::compiler;
    static constexpr rounding flight = rounding::compiler;
    static constexpr rounding walk_flat = rounding::compiler;
    static constexpr rounding walk_features = rounding::compiler;
    static constexpr rounding dielectric_unit = rounding::compiler;
    static constexpr rounding dielectric_cosine = rounding::compiler;
    static constexpr rounding dielectric_reflect = rounding::compiler;
    static constexpr rounding view = rounding::compiler;
    static constexpr rounding lamp_distance = rounding::compiler;
    static constexpr rounding lamp_cosine = rounding::compiler;
    static constexpr rounding lamp_hit = rounding::compiler;
    static constexpr rounding ggx_eval_view = rounding::compiler;
    static constexpr rounding ggx_eval_half = rounding::compiler;
    static constexpr rounding ggx_light_length = rounding::compiler;
    static constexpr rounding ggx_gloss_length = rounding::compiler;
    static constexpr rounding ggx_gloss_light = rounding::compiler;
    static constexpr rounding ggx_sample_view = rounding::compiler;
    static constexpr rounding ggx_sample_half = rounding::compiler;
    static constexpr rounding energy = rounding::compiler;
    static constexpr rounding mirror_cosine = rounding::compiler;
    static constexpr rounding mirror_reflect = rounding::compiler;
};

// A session's wavefront, as its shade and trace kernels come out of the compiler: found by writing out one product at
// a time in those kernels and keeping the form that leaves every image (the built-in scenes under both integrators, scenes
// of each material alone, scenes drawn at random) the same bit for bit. The kernels that render a session's samples in
// another form take this table, so the form changes no image.
struct rounds_session
{
    static constexpr bool bare = false; // whether these kernels render the bare small scenes only
    static constexpr rounding other = rounding::x;
    static constexpr rounding sky = rounding::y;
    static constexpr rounding flight = rounding::y;
    static constexpr rounding walk_flat = rounding::x;
    static constexpr rounding walk_features = rounding::y;
    static constexpr rounding dielectric_unit = rounding::y;
    static constexpr rounding dielectric_cosine = rounding::yz;
    static constexpr rounding dielectric_reflect = rounding::yz;
    static constexpr rounding view = rounding::y;
    static constexpr rounding lamp_distance = rounding::y;
    static constexpr rounding lamp_cosine = rounding::y;
    static constexpr rounding lamp_hit = rounding::y;
    static constexpr rounding ggx_eval_view = rounding::y;
    static constexpr rounding ggx_eval_half = rounding::y;
    static constexpr rounding ggx_light_length = rounding::x;
    static constexpr rounding ggx_gloss_length = rounding::y;
    static constexpr rounding ggx_gloss_light = rounding::y;
    static constexpr rounding ggx_sample_view = rounding::y;
    static constexpr rounding ggx_sample_half = rounding::y;
    static constexpr rounding energy = rounding::y;
    static constexpr rounding mirror_cosine = rounding::yz;
    static constexpr rounding mirror_reflect = rounding::yz;
};

// The persistent kernel's flat search, which renders the bare small scenes: the same but for the ray's squared length
struct rounds_bare : rounds_session
{
    static constexpr bool bare = true;
    static constexpr rounding walk_flat = rounding::y;
};
} // namespace rtb
