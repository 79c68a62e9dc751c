// FP64 ELLBLOCK product for a uniform partition of 32 x 32 blocks, on the FP64
// tensor instructions (mma.sync m8n8k4): the unordered form of
// ellblock/bml_multiply_ellblock_typed.c:246-442 (X^2) and :455-621 (A*B).
// The same blocks in the same (first-touch) order and the same keep rule as
// eb_mul32_kernel; a product's sums run as fused multiply-adds, like its
// fused form.
//
// Why.  eb_mul32_kernel adds every block product into an accumulator in
// device memory (16 KB of traffic per product, 12 TFLOP/s).  Here a block of C
// is formed by one warp in registers over all its pairs, and stored once.  A
// warp takes 16 columns of the block at a time, so that the registers hold the
// sum and, apart from it, the product of the current pair: a sum of pair
// products, as in eb_mul32_kernel, rounds less than one chain over all pairs
// (against 80-bit sums, block lattices of 3^3 to 5^3: 1.8e-16 of the result's
// norm, as eb_mul32_kernel; on the 11^3 lattice a chain is four times as far
// from an FP64 product as this).
//
// Steps.  A table T[kb][j] gives the slot of block (j, kb) of B (X^2 of a
// symmetric X: of block (kb, j), which is its transpose, so both operands are
// read along their rows).  The symbolic kernel lists the block columns of
// every row of C in first-touch order.  In the numeric kernel a warp takes a
// block (ib, kb), finds its pairs through T and the row ib, and multiplies
// them, the fragments of the next 8 columns loaded while the current 8 are
// multiplied (16-byte loads; lane q of a quad holds columns 2q and 2q + 1, the
// same permutation of the summed index on both sides).  The block is stored
// at its first-touch position: nothing is staged when every block is kept, and
// a last kernel closes the gaps of dropped blocks row by row.  Positions past
// C's MB go to a spill area.
//
// Symmetric X^2 (A == B, equal patterns and equal mirrored blocks, checked on
// the device): only blocks kb >= ib are formed, each stored also at its
// mirrored place, so C is exactly symmetric.
//
// Measured (X^2 of the radius-2 block lattice, FP64): 11^3 blocks 6.2 -> 1.93
// ms, 6^3 blocks 1.65 -> 0.37 ms.  At 11^3 the stores of the result alone take
// 0.35 ms; the products of one triangle 0.93 ms at 37 TFLOP/s, the rest is the
// latency of the first loads of a block (4.2 pairs on average).
#include "device_util.cuh"
#include "ellblock.h"

#include <algorithm>
#include <cstring>

using namespace b200;

namespace {

constexpr int PT = 256;            // threads of the per-row kernels
constexpr int FW = 4;              // warps of a numeric CTA
constexpr int FMIN = 3;            // numeric CTAs per SM (160 registers a thread; 4 spill: 2.02 against 1.97 ms)
constexpr int CHUNK = 16;          // blocks of a row a numeric CTA takes at a time
constexpr int PAIRS = 512;         // pairs a warp lists at a time
constexpr int F64_MAX_NB = 8192;   // tables of NB^2 16-bit entries
constexpr unsigned short NONE = 0xffffu;
constexpr size_t F64_SMALL = 45056; // place in the context's small buffers

struct F64Flags
{
    unsigned long long spill; // blocks past C's MB before thresholding
    int asym;
    int max_touched;
    int next;
    int overflow, max_kept;
    int done;                 // CTAs of the closing kernel that have finished
    double trA, trC;
};

struct F64Args
{
    const double *Ap; const int *Ai; const int *An; int MA;
    const double *Bp; const int *Bi; const int *Bn; int MBb;
    double *Cp; int *Ci; int *Cn; int MC;
    int NB;
    int square;                   // A == B
    double thr;
    unsigned short *rowT;         // [ib][jb]: slot of block (ib, jb) of A (square only)
    unsigned short *colT;         // [kb][j]: slot of block (j, kb) of B
    unsigned short *list;         // [ib][q]: block column at first-touch position q
    unsigned short *where;        // [ib][kb]: its position
    int *count;                   // touched block columns of a row
    unsigned long long *spill_at; // first spill block of a row
    unsigned char *keep;          // [ib][q]
    double *spill;
    double *dA, *dC;              // per-row traces
    F64Flags *flags, *host;       // host: pinned, written by the closing kernel's last CTA, then
    int told;                     // this to the word behind it
};

// Rows of up to SHORT_NB blocks into a C with room for all of them: nothing can
// spill, so the product is queued without the host learning the lists' lengths
// first, a numeric kernel for either outcome of the symmetry check among it.
// (8 block rows of 4 blocks: 80 us with that wait, four memsets and a copy at
// the end, 57 in the accumulating form, 55 so; 27 rows of up to 7 85, 92 and 62.)
constexpr int SHORT_NB = 128;
constexpr int TOLD = 32;

__global__ void __launch_bounds__(PT) f64_table_kernel(F64Args g)
{
    for (int j = blockIdx.x; j < g.NB; j += gridDim.x)
    {
        const int n = g.Bn[j];
        for (int p = threadIdx.x; p < n; p += PT)
        {
            const int kb = g.Bi[(size_t) j * g.MBb + p];
            g.colT[(size_t) kb * g.NB + j] = (unsigned short) p;
            if (g.square)
                g.rowT[(size_t) j * g.NB + kb] = (unsigned short) p;
        }
    }
}

// X against its transpose: blocks (ib, jb), jb >= ib, one warp each, the
// mirrored block through shared memory (its column reads in place: 100 us
// against 68 at 11^3 blocks).
__global__ void __launch_bounds__(128) f64_sym_kernel(F64Args g)
{
    __shared__ double t[4][32][33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int ib = blockIdx.x; ib < g.NB; ib += gridDim.x)
    {
        if (__any_sync(FULL, *(volatile int *) &g.flags->asym)) // other warps set it meanwhile
            return;
        const int n = g.An[ib];
        int bad = 0;
        for (int p = warp; p < n; p += 4)
        {
            const int jb = g.Ai[(size_t) ib * g.MA + p];
            const int s = g.rowT[(size_t) jb * g.NB + ib];
            if (s == NONE)
            {
                bad = 1;
                continue;
            }
            if (jb < ib)
                continue;
            const double *x = g.Ap + ((size_t) ib * g.MA + p) * 1024 + lane;
            const double *y = g.Ap + ((size_t) jb * g.MA + s) * 1024 + lane;
#pragma unroll 16
            for (int r = 0; r < 32; ++r)
                t[warp][r][lane] = y[r * 32];
            __syncwarp();
#pragma unroll 16
            for (int r = 0; r < 32; ++r)
                bad |= x[r * 32] != t[warp][lane][r];
            __syncwarp();
        }
        if (__any_sync(FULL, bad) && lane == 0)
            atomicExch(&g.flags->asym, 1);
    }
}

// First-touch lists.  Shared memory: mark[NB], position + 1 of a block column.
__global__ void __launch_bounds__(PT) f64_symbolic_kernel(F64Args g)
{
    extern __shared__ unsigned short mark[];
    __shared__ int wcnt[PT / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int ib = blockIdx.x; ib < g.NB; ib += gridDim.x)
    {
        for (int k = tid; k < g.NB; k += PT)
            mark[k] = 0;
        __syncthreads();
        const int na = g.An[ib];
        int lb = 0; // uniform
        double tr = 0.0;
        for (int jp = 0; jp < na; ++jp)
        {
            const int jb = g.Ai[(size_t) ib * g.MA + jp];
            if (jb == ib && warp == 0)
                tr += g.Ap[((size_t) ib * g.MA + jp) * 1024 + lane * 33];
            const int nk = g.Bn[jb];
            for (int c0 = 0; c0 < nk; c0 += PT)
            {
                const int p = c0 + tid;
                int kb = 0;
                bool fresh = false;
                if (p < nk)
                {
                    kb = g.Bi[(size_t) jb * g.MBb + p];
                    fresh = mark[kb] == 0;
                }
                const unsigned bal = __ballot_sync(FULL, fresh);
                if (lane == 0)
                    wcnt[warp] = __popc(bal);
                __syncthreads();
                int pos = lb, tot = 0;
                for (int w = 0; w < PT / 32; ++w)
                {
                    pos += w < warp ? wcnt[w] : 0;
                    tot += wcnt[w];
                }
                if (fresh)
                {
                    pos += __popc(bal & lanemask_lt());
                    mark[kb] = (unsigned short) (pos + 1);
                    g.list[(size_t) ib * g.NB + pos] = (unsigned short) kb;
                    g.where[(size_t) ib * g.NB + kb] = (unsigned short) pos;
                }
                lb += tot;
                __syncthreads();
            }
        }
        for (int o = 16; o; o >>= 1)
            tr += __shfl_xor_sync(FULL, tr, o);
        if (tid == 0)
        {
            g.count[ib] = lb;
            g.dA[ib] = tr;
            g.dC[ib] = 0.0;
            if (lb > g.MC)
                g.spill_at[ib] = atomicAdd(&g.flags->spill, (unsigned long long) (lb - g.MC));
            atomicMax(&g.flags->max_touched, lb);
        }
        __syncthreads();
    }
}

__device__ __forceinline__ double *place_of(const F64Args &g, int ib, int q)
{
    return q < g.MC ? g.Cp + ((size_t) ib * g.MC + q) * 1024
                    : g.spill + (size_t) (g.spill_at[ib] + (unsigned long long) (q - g.MC)) * 1024;
}

// SYM: X^2 of a symmetric X, both operands read along their rows.
// only: return unless the symmetry check came out for this form.
template <bool SYM> __global__ void __launch_bounds__(FW * 32, FMIN) f64_numeric_kernel(F64Args g, int chunks, int only)
{
    if (only && SYM == (g.flags->asym != 0))
        return;
    __shared__ unsigned queue[FW][PAIRS];
    __shared__ int item, nextq;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r8 = lane >> 2, q4 = lane & 3;
    unsigned *qu = queue[warp];
    const int items = g.NB * chunks;
    for (;;)
    {
        __syncthreads();
        if (threadIdx.x == 0)
        {
            item = atomicAdd(&g.flags->next, 1);
            nextq = 0;
        }
        __syncthreads();
        const int it = item;
        if (it >= items)
            break;
        const int ib = it / chunks;
        const int q0 = (it - ib * chunks) * CHUNK, q1 = min(q0 + CHUNK, g.count[ib]);
        const int na = g.An[ib];
        const int *arow = g.Ai + (size_t) ib * g.MA;
        const double *Ablk = g.Ap + (size_t) ib * g.MA * 1024 + r8 * 32 + 2 * q4;
        for (;;)
        {
            int q = 0;
            if (lane == 0)
                q = q0 + atomicAdd(&nextq, 1);
            q = __shfl_sync(FULL, q, 0);
            if (q >= q1)
                break;
            const int kb = g.list[(size_t) ib * g.NB + q];
            if (SYM && kb < ib)
                continue;
            const unsigned short *T = (SYM ? g.rowT : g.colT) + (size_t) kb * g.NB;
            const bool diag = kb == ib;
            double *dst = place_of(g, ib, q);
            const int qm = SYM && !diag ? g.where[(size_t) kb * g.NB + ib] : 0;
            double *mir = SYM ? (diag ? dst : place_of(g, kb, qm)) : nullptr;
            double mx = 0.0, tr = 0.0;
            int npairs = 0;
            // two halves of 16 columns: room for the sum and for the product of one pair
            for (int half = 0; half < 2; ++half)
            {
                double acc[4][2][2], part[4][2][2];
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < 2; ++b)
                        acc[a][b][0] = acc[a][b][1] = part[a][b][0] = part[a][b][1] = 0.0;
                // the second half finds the list as the first left it, if it held all pairs
                const bool listed = half && na <= PAIRS;
                int n = listed ? npairs : 0;
                for (int p0 = listed ? na : 0;; p0 += 32)
                {
                    // pairs of the next 32 left blocks: slot in row ib, slot of the right block
                    const int p = p0 + lane;
                    unsigned s = NONE;
                    int j = 0;
                    if (p < na)
                    {
                        j = arow[p];
                        s = T[j];
                    }
                    const unsigned bal = __ballot_sync(FULL, s != NONE);
                    const int tot = __popc(bal);
                    if (n > 0 && (p0 >= na || n + tot > PAIRS))
                    {
                        __syncwarp();
                        const int steps = 4 * n;
                        npairs = n;
                        double2 A0[4], A1[4], B0[2], B1[2];
                        auto load = [&](int step, double2(&A)[4], double2(&Bf)[2]) {
                            const unsigned e = qu[step >> 2];
                            const int k8 = 8 * (step & 3);
                            const double *pa = Ablk + (size_t) (e & 0xffffu) * 1024 + k8;
#pragma unroll
                            for (int m = 0; m < 4; ++m)
                                A[m] = __ldg(reinterpret_cast<const double2 *>(pa + m * 256));
                            if (SYM)
                            {
                                const double *pb = g.Bp + ((size_t) kb * g.MBb + (e >> 16)) * 1024 +
                                                   (16 * half + r8) * 32 + 2 * q4 + k8;
#pragma unroll
                                for (int m = 0; m < 2; ++m)
                                    Bf[m] = __ldg(reinterpret_cast<const double2 *>(pb + m * 256));
                            }
                            else
                            {
                                const int jb = arow[e & 0xffffu];
                                const double *pb = g.Bp + ((size_t) jb * g.MBb + (e >> 16)) * 1024 +
                                                   (k8 + 2 * q4) * 32 + 16 * half + r8;
#pragma unroll
                                for (int m = 0; m < 2; ++m)
                                    Bf[m] = make_double2(__ldg(pb + 8 * m), __ldg(pb + 32 + 8 * m));
                            }
                        };
                        auto mul = [&](const double2(&A)[4], const double2(&Bf)[2]) {
#pragma unroll
                            for (int h = 0; h < 2; ++h)
#pragma unroll
                                for (int a = 0; a < 4; ++a)
#pragma unroll
                                    for (int b = 0; b < 2; ++b)
                                        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, "
                                                     "{%3}, {%0,%1};"
                                                     : "+d"(part[a][b][0]), "+d"(part[a][b][1])
                                                     : "d"(h ? A[a].y : A[a].x), "d"(h ? Bf[b].y : Bf[b].x));
                        };
                        load(0, A0, B0);
                        for (int t = 0; t < steps; t += 2) // four steps per pair
                        {
                            load(t + 1, A1, B1);
                            mul(A0, B0);
                            if (t + 2 < steps)
                                load(t + 2, A0, B0);
                            mul(A1, B1);
                            if (t & 2)
                            {
                                // the pair is complete: its product joins the sum
#pragma unroll
                                for (int a = 0; a < 4; ++a)
#pragma unroll
                                    for (int b = 0; b < 2; ++b)
#pragma unroll
                                        for (int h = 0; h < 2; ++h)
                                        {
                                            acc[a][b][h] += part[a][b][h];
                                            part[a][b][h] = 0.0;
                                        }
                            }
                        }
                        n = 0;
                        __syncwarp();
                    }
                    if (p0 >= na)
                        break;
                    if (s != NONE)
                        qu[n + __popc(bal & lanemask_lt())] = (unsigned) p | s << 16;
                    n += tot;
                }

                // the half block to its first-touch place (and its mirror's)
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < 2; ++b)
                    {
                        const int r = 8 * a + r8, c = 16 * half + 8 * b + 2 * q4;
                        mx = fmax(mx, fmax(fabs(acc[a][b][0]), fabs(acc[a][b][1])));
                        if (c == r)
                            tr += acc[a][b][0];
                        if (c + 1 == r)
                            tr += acc[a][b][1];
                        if (!SYM || !diag)
                            *reinterpret_cast<double2 *>(dst + r * 32 + c) = make_double2(acc[a][b][0], acc[a][b][1]);
                        else
                        {
                            // the diagonal block: its upper triangle, stored twice
                            if (c >= r)
                                dst[r * 32 + c] = acc[a][b][0];
                            if (c + 1 >= r)
                                dst[r * 32 + c + 1] = acc[a][b][1];
                        }
                        if (SYM)
                        {
                            if (!diag || c > r)
                                mir[c * 32 + r] = acc[a][b][0];
                            if (!diag || c + 1 > r)
                                mir[(c + 1) * 32 + r] = acc[a][b][1];
                        }
                    }
            }
            for (int o = 16; o; o >>= 1)
                mx = fmax(mx, __shfl_xor_sync(FULL, mx, o));
            const unsigned char kept = diag || mx > g.thr;
            if (lane == 0)
            {
                g.keep[(size_t) ib * g.NB + q] = kept;
                if (SYM && !diag)
                    g.keep[(size_t) kb * g.NB + qm] = kept;
            }
            if (diag)
            {
                for (int o = 16; o; o >>= 1)
                    tr += __shfl_xor_sync(FULL, tr, o);
                if (lane == 0)
                    g.dC[ib] = tr;
            }
        }
    }
}

// Kept blocks of a row to the front, in order; the row's list.  Every
// destination lies at or before its source, and the sources of later blocks
// behind it, so W blocks are moved at a time: all read, then all written.
__global__ void __launch_bounds__(PT) f64_close_kernel(F64Args g)
{
    constexpr int W = PT / 32;
    __shared__ unsigned short src[1024];
    __shared__ int wcnt[W];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int ib = blockIdx.x; ib < g.NB; ib += gridDim.x)
    {
        const int n = g.count[ib];
        int kept = 0; // uniform
        for (int c0 = 0; c0 < n; c0 += PT)
        {
            const int q = c0 + tid;
            const bool k = q < n && g.keep[(size_t) ib * g.NB + q];
            const unsigned bal = __ballot_sync(FULL, k);
            if (lane == 0)
                wcnt[warp] = __popc(bal);
            __syncthreads();
            int pos = 0, tot = 0;
            for (int w = 0; w < W; ++w)
            {
                pos += w < warp ? wcnt[w] : 0;
                tot += wcnt[w];
            }
            if (k)
            {
                pos += __popc(bal & lanemask_lt());
                src[pos] = (unsigned short) q;
                if (kept + pos < g.MC)
                    g.Ci[(size_t) ib * g.MC + kept + pos] = g.list[(size_t) ib * g.NB + q];
            }
            __syncthreads();
            for (int b = 0; b < tot; b += W)
            {
                const int d = kept + b + warp;
                const bool move = b + warp < tot && d < g.MC && src[b + warp] != d;
                if (!__syncthreads_or(move))
                    continue;
                const double2 *s = nullptr;
                if (move)
                    s = reinterpret_cast<const double2 *>(place_of(g, ib, src[b + warp])) + lane;
                double2 *t = reinterpret_cast<double2 *>(g.Cp + ((size_t) ib * g.MC + d) * 1024) + lane;
                for (int h = 0; h < 2; ++h)
                {
                    double2 v[8];
                    if (move)
                    {
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            v[u] = s[(8 * h + u) * 32];
                    }
                    __syncthreads();
                    if (move)
                    {
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            t[(8 * h + u) * 32] = v[u];
                    }
                }
            }
            kept += tot;
            __syncthreads();
        }
        if (tid == 0)
        {
            g.Cn[ib] = min(kept, g.MC);
            atomicMax(&g.flags->max_kept, kept);
            if (kept > g.MC)
                atomicExch(&g.flags->overflow, 1);
        }
    }
    // the traces, summed over rows in a fixed order by the CTA that finishes last, and the flags for the host
    __shared__ double part[2][W];
    __shared__ int fin;
    __syncthreads();
    if (tid == 0)
    {
        __threadfence(); // this CTA's rows come before its count
        fin = atomicAdd(&g.flags->done, 1) == (int) gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!fin)
        return;
    double a = 0.0, d = 0.0;
    for (int ib = tid; ib < g.NB; ib += PT)
    {
        a += __ldcg(g.dA + ib);
        d += __ldcg(g.dC + ib);
    }
    for (int o = 16; o; o >>= 1)
    {
        a += __shfl_xor_sync(FULL, a, o);
        d += __shfl_xor_sync(FULL, d, o);
    }
    if (lane == 0)
    {
        part[0][warp] = a;
        part[1][warp] = d;
    }
    __syncthreads();
    if (tid != 0)
        return;
    for (int w = 1; w < W; ++w)
    {
        a += part[0][w];
        d += part[1][w];
    }
    volatile F64Flags *h = g.host;
    const volatile F64Flags *f = g.flags;
    h->asym = f->asym;
    h->overflow = f->overflow;
    h->max_kept = f->max_kept;
    h->trA = a;
    h->trC = d;
    __threadfence_system();
    reinterpret_cast<volatile int *>(g.host)[TOLD] = g.told;
}

} // namespace

bool eb_multiply_f64(bml_matrix_ellblock_t *A, bml_matrix_ellblock_t *B, bml_matrix_ellblock_t *C, double threshold,
                     double *trace, size_t budget, bool *taken)
{
    *taken = false;
    const int NB = A->NB;
    if (NB > F64_MAX_NB || A->MB >= NONE || B->MB >= NONE)
        return true;
    B200Context *c = b200_ctx();
    if (!c)
        return false;
    F64Args g{};
    g.Ap = static_cast<const double *>(A->d_pool); g.Ai = A->d_indexb; g.An = A->d_nnzb; g.MA = A->MB;
    g.Bp = static_cast<const double *>(B->d_pool); g.Bi = B->d_indexb; g.Bn = B->d_nnzb; g.MBb = B->MB;
    g.Cp = static_cast<double *>(C->d_pool); g.Ci = C->d_indexb; g.Cn = C->d_nnzb; g.MC = C->MB;
    g.NB = NB;
    g.square = A == B ? 1 : 0;
    g.thr = threshold;
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t nn = (size_t) NB * NB;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at = al(at + bytes);
        return o;
    };
    const size_t o_row = take(g.square ? nn * 2 : 0), o_col = take(nn * 2), o_list = take(nn * 2);
    const size_t o_where = take(nn * 2), o_keep = take(nn);
    const size_t o_count = take((size_t) NB * sizeof(int)), o_sat = take((size_t) NB * 8);
    const size_t o_diag = take((size_t) 2 * NB * sizeof(double));
    const size_t fixed = at;
    unsigned char *small = static_cast<unsigned char *>(c->d_small) + F64_SMALL;
    unsigned char *pin = static_cast<unsigned char *>(c->pinned) + F64_SMALL;
    F64Flags *hf = reinterpret_cast<F64Flags *>(pin);
    g.flags = reinterpret_cast<F64Flags *>(small);
    g.host = hf;
    const bool brief = NB <= SHORT_NB && C->MB >= NB;
    const int rows = std::min(NB, c->sm_count * 8);
    const size_t smemS = (size_t) NB * sizeof(unsigned short);
    size_t spill = 0;
    for (int attempt = 0; attempt < 2; ++attempt)
    {
        unsigned char *scr = static_cast<unsigned char *>(b200_scratch_try(fixed + spill * 8192));
        if (!scr)
            return true; // the accumulating form asks for what it needs
        g.rowT = reinterpret_cast<unsigned short *>(scr + o_row);
        g.colT = reinterpret_cast<unsigned short *>(scr + o_col);
        g.list = reinterpret_cast<unsigned short *>(scr + o_list);
        g.where = reinterpret_cast<unsigned short *>(scr + o_where);
        g.keep = scr + o_keep;
        g.count = reinterpret_cast<int *>(scr + o_count);
        g.spill_at = reinterpret_cast<unsigned long long *>(scr + o_sat);
        g.dA = reinterpret_cast<double *>(scr + o_diag);
        g.dC = g.dA + NB;
        g.spill = reinterpret_cast<double *>(scr + fixed);
        // (both tables: they lie side by side)
        if (!CUDA_OK(cudaMemsetAsync(small, 0, sizeof(F64Flags), c->stream)) ||
            !CUDA_OK(cudaMemsetAsync(scr + o_row, 0xff, o_list - o_row, c->stream)))
            return false;
        f64_table_kernel<<<rows, PT, 0, c->stream>>>(g);
        if (!LAUNCH_OK("f64_table_kernel"))
            return false;
        if (g.square)
        {
            f64_sym_kernel<<<rows, 128, 0, c->stream>>>(g);
            if (!LAUNCH_OK("f64_sym_kernel"))
                return false;
        }
        f64_symbolic_kernel<<<rows, PT, smemS, c->stream>>>(g);
        if (!LAUNCH_OK("f64_symbolic_kernel"))
            return false;
        if (brief)
            break;
        if (!CUDA_OK(cudaMemcpyAsync(pin, small, sizeof(F64Flags), cudaMemcpyDeviceToHost, c->stream)) || !b200_sync())
            return false;
        if (hf->spill * 8192 > budget)
            return true;
        if (hf->spill <= spill)
            break;
        // room for the blocks past MB: the lists are made again in the larger arena
        spill = (size_t) hf->spill;
    }
    const int chunks = ((brief ? NB : std::max(hf->max_touched, 1)) + CHUNK - 1) / CHUNK;
    const int grid = (int) std::min<long long>((long long) NB * chunks, (long long) c->sm_count * FMIN);
    if (g.square && (brief || !hf->asym))
    {
        f64_numeric_kernel<true><<<grid, FW * 32, 0, c->stream>>>(g, chunks, brief);
        if (!LAUNCH_OK("f64_numeric_kernel"))
            return false;
    }
    if (!g.square || brief || hf->asym)
    {
        f64_numeric_kernel<false><<<grid, FW * 32, 0, c->stream>>>(g, chunks, g.square && brief);
        if (!LAUNCH_OK("f64_numeric_kernel"))
            return false;
    }
    g.told = b200_next_told();
    f64_close_kernel<<<rows, PT, 0, c->stream>>>(g);
    if (!LAUNCH_OK("f64_close_kernel") || !b200_told(reinterpret_cast<const int *>(hf) + TOLD, g.told))
        return false;
    *taken = true;
    if (trace)
    {
        trace[0] = hf->trA;
        trace[1] = hf->trC;
    }
    if (hf->overflow)
    {
        b200_set_error(BML_B200_ERR_ROW_OVERFLOW,
                       "Number of non-zeroes blocks per row > MB, Increase MB (need %d, MB = %d)", hf->max_kept, C->MB);
        return false;
    }
    return true;
}
