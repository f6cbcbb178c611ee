// sor_tile.cuh -- a tile of FP32 red-black SOR in registers (internal): the
// sweeps that stay on the chip (sor_resident.cu) and the passes over grids in
// HBM (sor_tile.cu) run on it.
//
// A lane holds L consecutive rows of one lane column (eight cells: one quad of
// each colour, sor_quads.cuh).  CL lanes side by side make a tile row, so a
// warp holds 32 / CL groups of L rows, the CTA's groups one below the other.
// Horizontal neighbours come by shuffle from the next lane, vertical ones from
// the lane's own registers and, between groups, from the groups' edge rows in
// shared memory (double-buffered by colour: one block barrier a half sweep).
// -r32 sits in shared memory, one 16-byte load a quad and half sweep: in
// registers it doubled the instructions by register moves.
//
// A quad takes about 24 instructions: 12 packed FP32 operations, one packed
// register, shuffle, select, load, weights.  Held as consecutive cells, with
// three packed registers a half sum, it took 35.
#pragma once

#include "sor_quads.cuh"

namespace pcd {
namespace tile {

using namespace quads;

// UNI: every row has both vertical neighbours, so one set of weights serves
// them all (with a set a row, six rows and 128 registers, register moves
// doubled the instructions).
template <int L, int CL, bool RAG, bool UNI = false>
struct Tile {
    static constexpr int G = 32 / CL;              // row groups of a warp
    static constexpr int NS = RAG ? 2 : 1;         // weight sets of a row: one per parity where lanes differ
    static_assert(L % 2 == 0, "groups start on even grid rows");

    Quad e[2][L];
    // Per row: weight omega / cnt (0 outside the grid), as pairs.
    //   whole lane columns: wa both horizontal neighbours, wb the pair with
    //   the grid's first or last cell
    //   RAG: wa / wb of the quad's pairs by parity, and the coefficient of the
    //   cell's own value (-3 in a last column inside its lane, whose right
    //   neighbour reads 0)
    static constexpr int WR = UNI ? 1 : L;
    float2 wa[NS][WR], wb[NS][WR], ca[2], cb[2];
    bool own, zl, zr;
    bool brd, gin;           // warp with the grid's first or last row; group with a row of the grid
    int cl, gi, lr0, y0, H, nvalid;
    int wlo, whi;            // plane rows of the warp's groups
    unsigned edge_own, edge_up, edge_dn, edge_c;  // shared addresses; edge_c: bytes from colour 0 to 1
    // -r32 planes, one of the cells in even columns and one of those in odd ones:
    // shared address of the first row, bytes between the planes
    unsigned r_s, r_c;

    // w: omega / cnt
    __device__ __forceinline__ void setup_weights(bool act, int R, const float *w)
    {
        const bool line = H == 1;  // no vertical neighbour at all
#pragma unroll
        for (int j = 0; j < WR; j++) {
            const int y = y0 + j;
            const bool in = act && (UNI || (lr0 + j < R && y >= 0 && y < H)), mid = UNI || (y > 0 && y < H - 1);
            const float wi = !in ? 0.f : mid ? w[4] : line ? w[2] : w[3], we = !in ? 0.f : mid ? w[3] : line ? w[1] : w[2];
            if (RAG) {
#pragma unroll
                for (int q = 0; q < NS; q++) {
                    float v[4];
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        const int off = 2 * t + 1 - q, last = nvalid - 1;
                        const bool edge = (off == 0 && zl) || (off == 7 && zr) || (off == last && nvalid < 8);
                        v[t] = off > last ? 0.f : edge ? we : wi;
                    }
                    wa[q][j] = make_float2(v[0], v[2]);
                    wb[q][j] = make_float2(v[1], v[3]);
                }
            } else {
                wa[0][j] = make_float2(wi, wi);
                wb[0][j] = zl ? make_float2(we, wi) : zr ? make_float2(wi, we) : make_float2(wi, wi);
            }
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            auto c = [&](int t) { return RAG && nvalid < 8 && 2 * t + 1 - q == nvalid - 1 ? -3.f : -4.f; };
            ca[q] = make_float2(c(0), c(2));
            cb[q] = make_float2(c(1), c(3));
        }
    }
    __device__ __forceinline__ float2 weight_a(int q, int j) const
    {
        const int r = UNI ? 0 : j;
        return RAG ? wa[RAG ? q : 0][r] : q && zl ? wb[0][r] : wa[0][r];
    }
    __device__ __forceinline__ float2 weight_b(int q, int j) const
    {
        const int r = UNI ? 0 : j;
        return RAG ? wb[RAG ? q : 0][r] : !q && zr ? wb[0][r] : wa[0][r];
    }

    // Publishes the group's edge rows of colour CC.  The grid's first and last
    // row also go, as the other colour, into the rows just outside the grid:
    // a missing vertical neighbour takes the cell's own value.  (Those rows
    // weigh 0, and groups outside the grid publish nothing, so nobody else
    // writes them.)  Every warp runs the same update; a separate form for the
    // border rows would set the pace of the whole grid.
    template <int CC>
    __device__ __forceinline__ void put_edges()
    {
        constexpr int OC = 1 - CC;
        if (!UNI && brd) {
#pragma unroll
            for (int j = 0; j < L; j++) {
                if (y0 + j == 0) {
                    if (j > 0) e[OC][j > 0 ? j - 1 : 0] = e[CC][j];
                    else stsq(edge_up + (OC ? edge_c : 0u), e[CC][j]);
                }
                if (y0 + j == H - 1) {
                    if (j + 1 < L) e[OC][j + 1 < L ? j + 1 : j] = e[CC][j];
                    else stsq(edge_dn + (OC ? edge_c : 0u), e[CC][j]);
                }
            }
        }
        if (UNI || gin) {
            const unsigned a = edge_own + (CC ? edge_c : 0u);
            stsq(a, e[CC][0]);
            stsq(a + 16u * CL, e[CC][L - 1]);
        }
    }

    // the other colour's cell beyond the lane's eight columns, or beyond the
    // grid the cell's own value
    __device__ __forceinline__ float beyond(int q, const Quad &m, const Quad &v) const
    {
        const float x = q ? __shfl_up_sync(0xffffffffu, m.b.y, 1) : __shfl_down_sync(0xffffffffu, m.a.x, 1);
        return (q ? zl : zr) ? (q ? v.a.x : v.b.y) : x;
    }

    // the place of row j's quad of colour c in the planes at `from` (the group's
    // first row is even)
    __device__ __forceinline__ unsigned plane_at(unsigned from, int c, int j) const
    {
        return from + (((c ^ j) & 1) ? r_c : 0u) + 16u * (unsigned)(CL * j);
    }
    __device__ __forceinline__ unsigned rhs_at(int c, int j) const { return plane_at(r_s, c, j); }
    __device__ __forceinline__ Quad rhs(int c, int j) const
    {
        return ldsq(rhs_at(c, j));
    }

    // The negated residual of row j's quad of colour CC.
    template <int CC>
    __device__ __forceinline__ Quad defect(int j, const Quad &eu, const Quad &ed) const
    {
        constexpr int OC = 1 - CC;
        const int q = 1 - ((j ^ CC) & 1);  // the group's first row is even
        const Quad &v = e[CC][j], &m = e[OC][j];
        const float ex = beyond(q, m, v);
        return quad_defect(q, v, rhs(CC, j), j > 0 ? e[OC][j > 0 ? j - 1 : 0] : eu,
                           j + 1 < L ? e[OC][j + 1 < L ? j + 1 : j] : ed, m, ex, RAG ? ca[q] : make_float2(-4.f, -4.f),
                           RAG ? cb[q] : make_float2(-4.f, -4.f));
    }

    // Half sweep of colour CC.  TR: mx takes the largest |update| of the tile's
    // own cells (plane rows [olo, ohi)).
    template <int CC, bool TR>
    __device__ __forceinline__ void half(float &mx, int olo, int ohi)
    {
        constexpr int OC = 1 - CC;
        const Quad eu = ldsq(edge_up + (OC ? edge_c : 0u));
        const Quad ed = ldsq(edge_dn + (OC ? edge_c : 0u));
#pragma unroll
        for (int j = 0; j < L; j++) {
            const int q = 1 - ((j ^ CC) & 1);
            const Quad t = defect<CC>(j, eu, ed), v = e[CC][j];
            const Quad nv = {__ffma2_rn(weight_a(q, j), t.a, v.a), __ffma2_rn(weight_b(q, j), t.b, v.b)};
            if (TR && own && lr0 + j >= olo && lr0 + j < ohi) mx = fmaxf(mx, quad_max_change(v, nv));
            e[CC][j] = nv;
        }
        put_edges<CC>();
    }

    template <int CC>
    __device__ __forceinline__ float residual_of(int olo, int ohi) const
    {
        constexpr int OC = 1 - CC;
        float acc = 0.f;
        const Quad eu = ldsq(edge_up + (OC ? edge_c : 0u));
        const Quad ed = ldsq(edge_dn + (OC ? edge_c : 0u));
#pragma unroll
        for (int j = 0; j < L; j++) {
            const int o = (j ^ CC) & 1;  // offset of the quad's first cell
            Quad r = defect<CC>(j, eu, ed);
            if (RAG) {
                r.a.x = o < nvalid ? r.a.x : 0.f;
                r.b.x = o + 2 < nvalid ? r.b.x : 0.f;
                r.a.y = o + 4 < nvalid ? r.a.y : 0.f;
                r.b.y = o + 6 < nvalid ? r.b.y : 0.f;
            }
            const float s2 = fmaf(r.a.x, r.a.x, fmaf(r.b.x, r.b.x, fmaf(r.a.y, r.a.y, r.b.y * r.b.y)));
            acc += own && lr0 + j >= olo && lr0 + j < ohi ? s2 : 0.f;
        }
        return acc;
    }
    // Sum of (r32 - L e)^2 over the lane's own cells of plane rows [olo, ohi).
    __device__ __forceinline__ float residual(int olo, int ohi) const
    {
        return residual_of<0>(olo, ohi) + residual_of<1>(olo, ohi);
    }

    // The lane's quad of colour c of row j in a grid of the quads' layout
    // (sor_quads.cuh): floats behind the row's first; the group's first row is
    // even.
    static __device__ __forceinline__ int quad_at(int c, int j, int q, int KQ) { return (((c ^ j) & 1) * KQ + q) * 4; }
    // Copies row j's quads of such a grid to the lane's place (shared address
    // `to` of row 0; zeros unless in), asynchronously: copies_wait before use.
    __device__ __forceinline__ void copy_row(unsigned to, int j, const float *row, int q, int KQ, bool in) const
    {
#pragma unroll
        for (int c = 0; c < 2; c++)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(plane_at(to, c, j)),
                         "l"(in ? row + quad_at(c, j, q, KQ) : row), "r"(in ? 16 : 0)
                         : "memory");
    }
    static __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
    __device__ __forceinline__ void store_row(int j, float *row, int q, int KQ) const
    {
#pragma unroll
        for (int c = 0; c < 2; c++)
            *reinterpret_cast<float4 *>(row + quad_at(c, j, q, KQ)) =
                make_float4(e[c][j].a.x, e[c][j].a.y, e[c][j].b.x, e[c][j].b.y);
    }

    // The lane's place in a CTA with NG row groups, and the shared addresses:
    // smem holds edge_quads, then the -r32 planes.
    __device__ __forceinline__ void place(const void *smem, int NG)
    {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        cl = lane & (CL - 1);
        gi = w * G + lane / CL;
        lr0 = gi * L;
        wlo = w * G * L;
        whi = wlo + G * L;
        const unsigned base = (unsigned)__cvta_generic_to_shared(smem), grow = 16u * CL, at = 16u * cl;
        edge_c = 2u * ((unsigned)NG + 1u) * grow;
        edge_own = base + (unsigned)(2 * gi) * grow + at;
        edge_up = base + (unsigned)(gi > 0 ? 2 * gi - 1 : 2 * NG) * grow + at;
        edge_dn = base + (unsigned)(gi < NG - 1 ? 2 * gi + 2 : 2 * NG + 1) * grow + at;
        r_c = (unsigned)(NG * L) * grow;
        r_s = base + 2u * edge_c + (unsigned)lr0 * grow + at;
    }
};

// Quads of a CTA's shared memory: the groups' edge rows and, for each colour,
// one row above the first group and one below the last; a pair of planes.
__host__ __device__ inline size_t edge_quads(int CL, int NG) { return (size_t)4 * (NG + 1) * CL; }
__host__ __device__ inline size_t plane_quads(int L, int CL, int NG) { return (size_t)2 * NG * L * CL; }

}  // namespace tile
}  // namespace pcd
