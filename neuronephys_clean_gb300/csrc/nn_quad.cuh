// Four consecutive x cells of a grid row as two packed pairs (nn_hh.cuh), for
// the stencils that give a thread a quad of every plane it passes.
#pragma once

#include "nn_hh.cuh"

typedef nn_vf<2> V2;
struct Quad {
    V2 a, b;
};
__device__ __forceinline__ Quad quad_ld(const float* p)
{
    const float4 v = *reinterpret_cast<const float4*>(p);
    return {{{v.x, v.y}}, {{v.z, v.w}}};
}
__device__ __forceinline__ void quad_st(float* p, const Quad& q)
{
    *reinterpret_cast<float4*>(p) = make_float4(q.a.v[0], q.a.v[1], q.b.v[0], q.b.v[1]);
}
__device__ __forceinline__ Quad quad_ldcg(const float4* p)  // kept where it stands in the program
{
    Quad q;
    asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(q.a.v[0]), "=f"(q.a.v[1]), "=f"(q.b.v[0]), "=f"(q.b.v[1])
                 : "l"(p)
                 : "memory");
    return q;
}
__device__ __forceinline__ Quad quad_zero() { return {{{0, 0}}, {{0, 0}}}; }
__device__ __forceinline__ float& at(Quad& q, int e) { return e < 2 ? q.a.v[e] : q.b.v[e - 2]; }
__device__ __forceinline__ float at(const Quad& q, int e) { return e < 2 ? q.a.v[e] : q.b.v[e - 2]; }

