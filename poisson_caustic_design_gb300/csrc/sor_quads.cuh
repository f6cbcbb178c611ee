// sor_quads.cuh -- the FP32 red-black update on quads: four cells of one
// colour in a row, eight columns wide, held as a float4 (internal).
//
// Quad of colour c in row y at lane column q covers the cells
// x = 8 q + 2 t + s, t < 4, s = (y & 1) ^ c.  With the parity q = 1 - s: for
// q = 1 the cells sit at the even offsets and need the other colour's cell
// one to the left of the lane's eight columns, for q = 0 at the odd offsets
// and need the one to the right.
#pragma once

#include "common.cuh"

namespace pcd {
namespace quads {

__device__ __forceinline__ float4 lds4(unsigned a)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ float lds1(unsigned a)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts4(unsigned a, const float4 &v)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

// v + w ((l + r) + (u + d) - 4 v - r32) per cell, the cell's own value as every
// missing neighbour, in packed FP32 pairs (cells (x, y) and (z, w) of the quad
// share one instruction per step); nrh is -r32.  The steps and their rounding
// are those of the scalar form.
__device__ __forceinline__ float4 quad_ghost_q(int q, const float4 &v, const float4 &nrh, const float4 &u,
                                              const float4 &d, const float4 &m, float ex, float2 wA, float2 wB)
{
    const float h0 = q ? ex + m.x : m.x + m.y;
    const float h1 = q ? m.x + m.y : m.y + m.z;
    const float h2 = q ? m.y + m.z : m.z + m.w;
    const float h3 = q ? m.z + m.w : m.w + ex;
    const float2 vA = make_float2(v.x, v.y), vB = make_float2(v.z, v.w);
    const float2 m4 = make_float2(-4.f, -4.f);
    float2 tA = __fadd2_rn(make_float2(h0, h1), __fadd2_rn(make_float2(u.x, u.y), make_float2(d.x, d.y)));
    float2 tB = __fadd2_rn(make_float2(h2, h3), __fadd2_rn(make_float2(u.z, u.w), make_float2(d.z, d.w)));
    tA = __fadd2_rn(__ffma2_rn(m4, vA, tA), make_float2(nrh.x, nrh.y));
    tB = __fadd2_rn(__ffma2_rn(m4, vB, tB), make_float2(nrh.z, nrh.w));
    const float2 nA = __ffma2_rn(wA, tA, vA), nB = __ffma2_rn(wB, tB, vB);
    return make_float4(nA.x, nA.y, nB.x, nB.y);
}

// Sum of squares of r32 - L v over the quad (ghost neighbours; nrh is -r32).
__device__ __forceinline__ float quad_ghost_res2(int q, const float4 &v, const float4 &nrh, const float4 &u,
                                                const float4 &d, const float4 &m, float ex)
{
    const float l0 = q ? ex : m.x, r0v = q ? m.x : m.y;
    const float l1 = q ? m.x : m.y, r1v = q ? m.y : m.z;
    const float l2 = q ? m.y : m.z, r2v = q ? m.z : m.w;
    const float l3 = q ? m.z : m.w, r3v = q ? m.w : ex;
    const float a0 = nrh.x + fmaf(-4.f, v.x, (l0 + r0v) + (u.x + d.x));
    const float a1 = nrh.y + fmaf(-4.f, v.y, (l1 + r1v) + (u.y + d.y));
    const float a2 = nrh.z + fmaf(-4.f, v.z, (l2 + r2v) + (u.z + d.z));
    const float a3 = nrh.w + fmaf(-4.f, v.w, (l3 + r3v) + (u.w + d.w));
    return fmaf(a0, a0, fmaf(a1, a1, fmaf(a2, a2, a3 * a3)));
}

// A quad as two pairs: a its cells 0 and 2, b its cells 1 and 3.  Half of the
// horizontal sums are then a plain pair sum and the other half needs one
// packed register (the shifted pair), where consecutive pairs need three.
struct Quad {
    float2 a, b;
};

// The layout of a grid in HBM that the tiles read and write (the correction and
// minus its right-hand side): a row is KQ = ceil(W / 8) quads of its cells at
// even columns, then KQ quads of those at odd ones, a quad's floats in the order
// (a, b).  A lane's quad is one aligned 16-byte access, 16 lanes one run of 256
// bytes, and the quad lands in whole register pairs.  (From a row-major grid a
// lane read 32 bytes in two half-used accesses, and the registers of those
// loads, two cells of which make a pair, stayed tied to the sweep loop: 2700
// instructions a warp and tile pass against 1700.)
__host__ __device__ inline long quad_row_floats(int W) { return 8l * ((W + 7) / 8); }
// the float of cell (x, y) in its row: column x
__host__ __device__ inline int quad_column(int x, int KQ)
{
    const int t = (x >> 1) & 3;
    return ((x & 1) * KQ + (x >> 3)) * 4 + ((t & 1) << 1 | t >> 1);
}

__device__ __forceinline__ Quad quad_zero() { return {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
__device__ __forceinline__ Quad ldsq(unsigned p)
{
    Quad v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.a.x), "=f"(v.a.y), "=f"(v.b.x), "=f"(v.b.y)
                 : "r"(p));
    return v;
}
__device__ __forceinline__ void stsq(unsigned p, const Quad &v)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(p), "f"(v.a.x), "f"(v.a.y), "f"(v.b.x), "f"(v.b.y)
                 : "memory");
}

// Neighbour sums (l + r) + (u + d) of the quad's cells; m the other colour's
// quad of the same lane column, ex its cell beyond the lane column.
__device__ __forceinline__ Quad quad_sums(int q, const Quad &u, const Quad &d, const Quad &m, float ex)
{
    const float2 mid = __fadd2_rn(m.a, m.b);
    const float2 sh = q ? __fadd2_rn(make_float2(ex, m.b.x), m.a) : __fadd2_rn(m.b, make_float2(m.a.y, ex));
    return {__fadd2_rn(q ? sh : mid, __fadd2_rn(u.a, d.a)), __fadd2_rn(q ? mid : sh, __fadd2_rn(u.b, d.b))};
}

// nrh + (l + r) + (u + d) + c v per cell, nrh = -r32: the negated residual.
// c is -4, a missing neighbour taking the cell's own value, plus the number of
// neighbours that read 0 instead.
__device__ __forceinline__ Quad quad_defect(int q, const Quad &v, const Quad &nrh, const Quad &u, const Quad &d,
                                            const Quad &m, float ex, float2 ca, float2 cb)
{
    const Quad s = quad_sums(q, u, d, m, ex);
    return {__fadd2_rn(__ffma2_rn(ca, v.a, s.a), nrh.a), __fadd2_rn(__ffma2_rn(cb, v.b, s.b), nrh.b)};
}

// Largest |nv - v| over the quad (a NaN change does not raise it).
__device__ __forceinline__ float quad_max_change(const Quad &v, const Quad &nv)
{
    return fmaxf(fmaxf(fabsf(nv.a.x - v.a.x), fabsf(nv.a.y - v.a.y)),
                 fmaxf(fabsf(nv.b.x - v.b.x), fabsf(nv.b.y - v.b.y)));
}

}  // namespace quads
}  // namespace pcd
