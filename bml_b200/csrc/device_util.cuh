// Device helpers shared by the kernel translation units.
#pragma once

#include "internal.h"

namespace b200 {

constexpr unsigned FULL = 0xffffffffu;

// Correctly rounded multiply / add that the compiler may not contract into an
// FMA.  The reference is built -std=c99 without -mfma, so every product and
// sum it forms is a separately rounded IEEE operation; these reproduce that.
template <typename T> __device__ __forceinline__ T mul_rn(T a, T b);
template <> __device__ __forceinline__ double mul_rn<double>(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ float mul_rn<float>(float a, float b) { return __fmul_rn(a, b); }
template <typename T> __device__ __forceinline__ T add_rn(T a, T b);
template <> __device__ __forceinline__ double add_rn<double>(double a, double b) { return __dadd_rn(a, b); }
template <> __device__ __forceinline__ float add_rn<float>(float a, float b) { return __fadd_rn(a, b); }

// x + s*y where s is a double scalar and x, y are of the matrix precision,
// evaluated the way C evaluates `x + alpha * y` with a double alpha: in double,
// then rounded once to the matrix precision.
template <typename T> __device__ __forceinline__ T axpy_d(T x, double s, T y)
{
    return (T) __dadd_rn((double) x, __dmul_rn(s, (double) y));
}

__device__ __forceinline__ unsigned lanemask_lt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Barrier over the W warps of one team; team t uses named barrier t+1.
template <int W> __device__ __forceinline__ void team_sync(int team)
{
    if (W == 1)
        __syncwarp();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(W * 32) : "memory");
}

__device__ __forceinline__ unsigned hash_slot(int k, unsigned mask)
{
    return ((unsigned) k * 2654435761u) & mask;
}

// Open-addressing insert of key k with payload v into (keys, pay) of size
// mask+1; returns the slot, or -1 when the table is full.  Concurrent inserts
// of distinct keys are safe.
__device__ __forceinline__ int hash_put(int *keys, int *pay, unsigned mask, int k, int v)
{
    unsigned h = hash_slot(k, mask);
    volatile int *vk = keys;
#pragma unroll 1
    for (unsigned p = 0; p <= mask; ++p)
    {
        const int cur = vk[h];
        if (cur == B200_EMPTY_KEY)
        {
            const int old = atomicCAS(&keys[h], B200_EMPTY_KEY, k);
            if (old == B200_EMPTY_KEY || old == k)
            {
                pay[h] = v;
                return (int) h;
            }
        }
        else if (cur == k)
        {
            pay[h] = v;
            return (int) h;
        }
        h = (h + 1) & mask;
    }
    return -1;
}

// Lookup of key k; returns its payload or -1.
__device__ __forceinline__ int hash_get(const int *keys, const int *pay, unsigned mask, int k)
{
    unsigned h = hash_slot(k, mask);
#pragma unroll 1
    for (unsigned p = 0; p <= mask; ++p)
    {
        const int cur = keys[h];
        if (cur == k)
            return pay[h];
        if (cur == B200_EMPTY_KEY)
            return -1;
        h = (h + 1) & mask;
    }
    return -1;
}

// Place of column k in the hash, or -1.
__device__ __forceinline__ int hash_find(const int *keys, unsigned mask, int k)
{
    unsigned h = hash_slot(k, mask);
#pragma unroll 1
    for (unsigned p = 0; p <= mask; ++p)
    {
        const int cur = keys[h];
        if (cur == k)
            return (int) h;
        if (cur == B200_EMPTY_KEY)
            return -1;
        h = (h + 1) & mask;
    }
    return -1;
}

// hash_put that tells whether the column was there already.
__device__ __forceinline__ bool hash_add(int *keys, int *pay, unsigned mask, int k, int v)
{
    unsigned h = hash_slot(k, mask);
    volatile int *vk = keys;
#pragma unroll 1
    for (unsigned p = 0; p <= mask; ++p)
    {
        int old = vk[h];
        if (old == B200_EMPTY_KEY)
            old = atomicCAS(&keys[h], B200_EMPTY_KEY, k);
        if (old == B200_EMPTY_KEY || old == k)
        {
            pay[h] = v;
            return old == k;
        }
        h = (h + 1) & mask;
    }
    return false;
}

// Whether a product of two matrices is the tile form's (ellpack_tiles.cu), by its
// counts (cost 0: whatever they are): what the
// sparse form takes longer for, in us, a row, an entry of A (each visits a row
// of B) and a product, against a tile product and what the tile form's twelve
// launches take whatever the sizes.  Fitted to 143 products of bands, lattices,
// diagonals and scattered matrices of 500 to 64000 rows, on which it takes
// neither form where the other is more than 3 % faster (tile form / sparse form,
// us: bands of 3 and 3 of 4096 rows 114 / 83, of 8000 144 / 135, of 20000 243 /
// 303, of 31 and 31 122 / 109, 160 / 192 and 270 / 427, of 301 and 301 of 500
// rows 209 / 114, of 1700 231 / 351, of 4096 261 / 799; a diagonal times a 16^3
// lattice 130 / 105, times a 28^3 one 416 / 562; lattices of radii 3 and 3.5, 14^3
// 222 / 196, 22^3 628 / 784, of 2 and 4.5, 18^3 345 / 333, 23^3 711 / 734; 4096
// scattered rows of 20 1059 / 142).
__host__ __device__ __forceinline__ bool general_pays(double rows, double stored, double products, double tiles2,
                                                      double cost)
{
    return cost == 0.0 || 10e-3 * rows + 1.4e-4 * stored + 1e-6 * products - 30e-6 * tiles2 > 90.0;
}

// Whether the row lengths of A and B speak for tiles, with 40 products per tile
// product (lattices have 20 to 60, bands hundreds).  One CTA of 1024 threads;
// the answer is thread 0's.
__device__ __forceinline__ bool rows_for_tiles(const int *An, int lda, const int *Bn, int ldb, int n)
{
    __shared__ double part[2][32];
    double a = 0.0, b = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += 1024)
    {
        a += min(max(An[i], 0), lda);
        b += min(max(Bn[i], 0), ldb);
    }
    for (int o = 16; o; o >>= 1)
    {
        a += __shfl_xor_sync(FULL, a, o);
        b += __shfl_xor_sync(FULL, b, o);
    }
    if ((threadIdx.x & 31) == 0)
    {
        part[0][threadIdx.x >> 5] = a;
        part[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    for (int w = 1; threadIdx.x == 0 && w < 32; ++w)
    {
        a += part[0][w];
        b += part[1][w];
    }
    const double products = a * b / n;
    return general_pays(n, a, products, products / 40.0, 1.0);
}

} // namespace b200

// Sum of one or two per-row arrays in FP64 with a fixed order (each thread a
// contiguous stripe, then a tree), written to out[0..1].  Launch <<<1, 1024>>>.
__global__ void b200_sum_rows_kernel(const double *a, const double *b, int n, double *out);
// Max and min of per-row arrays (hi, lo) into out[0] = max(init_max, hi[i]),
// out[1] = min(init_min, lo[i]).  Launch <<<1, 1024>>>.
__global__ void b200_maxmin_rows_kernel(const double *hi, const double *lo, int n,
                                        double init_max, double init_min, double *out);
