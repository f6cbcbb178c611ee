// words.cuh -- values that carry the epoch they belong to (internal).
//
// Co-resident CTAs exchange values as 64-bit words of a 32-bit value and a
// 32-bit tag.  The reader polls the words themselves: a relaxed 64-bit access
// is single-copy atomic, so value and tag are never torn, and no fence, flag
// or second trip through L2 stands between a store and its use (fence, flag,
// poll and load take 4-5 us for a halo exchange, the words 1.2-2.3 us).  Four
// words make one 32-byte sector and one access; a vector access is four
// 64-bit ones.
#pragma once

#include "common.cuh"

namespace pcd {
namespace words {

__device__ __forceinline__ unsigned long long word(unsigned v, unsigned tag)
{
    return (unsigned long long)v | ((unsigned long long)tag << 32);
}

struct Words {
    unsigned long long x, y, z, w;
};

__device__ __forceinline__ void st4(Words *p, const Words &v)
{
    asm volatile("st.relaxed.gpu.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(v.x), "l"(v.y), "l"(v.z), "l"(v.w)
                 : "memory");
}

__device__ __forceinline__ Words ld4(const Words *p)
{
    Words v;
    asm volatile("ld.relaxed.gpu.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(v.x), "=l"(v.y), "=l"(v.z), "=l"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long ld1(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st1(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ bool fresh(unsigned long long v, unsigned tag) { return (unsigned)(v >> 32) == tag; }
__device__ __forceinline__ bool fresh(const Words &v, unsigned tag)
{
    return fresh(v.x, tag) && fresh(v.y, tag) && fresh(v.z, tag) && fresh(v.w, tag);
}

// Two doubles.
__device__ __forceinline__ Words pack(double a, double b, unsigned tag)
{
    return {word((unsigned)__double2loint(a), tag), word((unsigned)__double2hiint(a), tag),
            word((unsigned)__double2loint(b), tag), word((unsigned)__double2hiint(b), tag)};
}
__device__ __forceinline__ double first(const Words &v) { return __hiloint2double((int)(unsigned)v.y, (int)(unsigned)v.x); }
__device__ __forceinline__ double second(const Words &v) { return __hiloint2double((int)(unsigned)v.w, (int)(unsigned)v.z); }

// One more unsuccessful poll: false once the poll budget is spent (then
// PCD_TIMEOUT is recorded in *error) or another CTA recorded an error.
__device__ __forceinline__ bool again(int *error, long long limit, long long &it)
{
    if ((++it & 63) == 0) {
        if (*(volatile const int *)error) return false;
        if (it > limit) {
            atomicCAS(error, 0, PCD_TIMEOUT);
            return false;
        }
    }
    return true;
}

}  // namespace words
}  // namespace pcd
