// The device's uniforms and normals (csrc/rng.cuh) compiled for the host, the
// device intrinsics that they call restated. Reads words "hi1 lo1 hi2 lo2" from
// standard input and prints u1, u2 and the normal of each line.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include <cuda_runtime.h>
#ifndef __noinline__
#define __noinline__
#endif

static inline double __hiloint2double(int hi, int lo)
{
    const uint64_t b = ((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo;
    double d;
    std::memcpy(&d, &b, sizeof d);
    return d;
}
static inline long long __double_as_longlong(double d)
{
    long long b;
    std::memcpy(&b, &d, sizeof b);
    return b;
}
static inline double __longlong_as_double(long long b)
{
    double d;
    std::memcpy(&d, &b, sizeof d);
    return d;
}
static inline int __double2loint(double d) { return (int)(uint32_t)__double_as_longlong(d); }
static inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static inline float __fdividef(float a, float b) { return a / b; }
static inline float rsqrtf(float x) { return 1.0f / std::sqrt(x); }
using std::fabs;
using std::floor;
using std::fma;

#include "rng.cuh"

int main()
{
    unsigned h1, l1, h2, l2;
    while (std::scanf("%x %x %x %x", &h1, &l1, &h2, &l2) == 4) {
        const double u1 = wctb200::uniform53(h1, l1), u2 = wctb200::uniform53(h2, l2);
        std::printf("%.17g %.17g %.9g\n", u1, u2, (double)wctb200::box_muller(u1, u2));
    }
    return 0;
}
