// Host stand-in for the CUDA runtime header: a block's threads are host threads, its
// shared memory is heap memory, warps and blocks meet at std::barrier.  Enough of it to
// run the resident kernel (fdtd_resident.cuh) with the stand-ins of cluster.cuh and
// packed.cuh beside it.
#pragma once
#include <algorithm>
#include <barrier>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __shared__
#define __forceinline__ inline
#define __restrict__
#define __launch_bounds__(...)
#define __align__(n)

using std::max;
using std::min;

struct Index3 {
    int x, y, z;
};
struct uchar4 {
    unsigned char x, y, z, w;
};
struct uint4 {
    unsigned x, y, z, w;
};
struct float2 {
    float x, y;
};
struct float4 {
    float x, y, z, w;
};
struct double2 {
    double x, y;
};
inline float2 make_float2(float a, float b) { return {a, b}; }
inline float4 make_float4(float a, float b, float c, float d) { return {a, b, c, d}; }
inline double2 make_double2(double a, double b) { return {a, b}; }

inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }

struct HostWarp {
    std::barrier<> meet{32};
    alignas(16) unsigned char slot[32][16];
};
struct HostBlock {
    std::unique_ptr<std::barrier<>> meet;
    std::vector<HostWarp> warps;
    std::vector<unsigned char> memory;
    unsigned char* smem = nullptr;
};
inline thread_local Index3 threadIdx, blockIdx;
inline Index3 blockDim, gridDim;
inline thread_local HostBlock* this_block;
inline thread_local HostWarp* this_warp;

inline unsigned long long __cvta_generic_to_shared(const void*) { return 0; }
template <class T>
void __stcg(T* p, T v) {
    *p = v;
}
inline void __syncthreads() { this_block->meet->arrive_and_wait(); }
inline void __syncwarp() { this_warp->meet.arrive_and_wait(); }
template <class T>
T lane_value(T v, int from) {
    std::memcpy(this_warp->slot[threadIdx.x & 31], &v, sizeof(T));
    __syncwarp();
    T r;
    std::memcpy(&r, this_warp->slot[from], sizeof(T));
    __syncwarp();
    return r;
}
template <class T>
T __shfl_sync(unsigned, T v, int s) {
    return lane_value(v, s & 31);
}
template <class T>
T __shfl_down_sync(unsigned, T v, int d) {
    const int l = threadIdx.x & 31;
    return lane_value(v, l + d < 32 ? l + d : l);
}
template <class T>
T __shfl_up_sync(unsigned, T v, int d) {
    const int l = threadIdx.x & 31;
    return lane_value(v, l >= d ? l - d : l);
}
inline unsigned __reduce_or_sync(unsigned, unsigned v) {
    std::memcpy(this_warp->slot[threadIdx.x & 31], &v, sizeof(v));
    __syncwarp();
    unsigned r = 0;
    for (int i = 0; i < 32; ++i) {
        unsigned q;
        std::memcpy(&q, this_warp->slot[i], sizeof(q));
        r |= q;
    }
    __syncwarp();
    return r;
}
inline bool __any_sync(unsigned m, bool p) { return __reduce_or_sync(m, p) != 0; }
inline bool __all_sync(unsigned m, bool p) { return !__any_sync(m, !p); }
inline int atomicAdd(int* p, int v) { return __sync_fetch_and_add(p, v); }
inline unsigned atomicOr(unsigned* p, unsigned v) { return __sync_fetch_and_or(p, v); }
long long clock64();
