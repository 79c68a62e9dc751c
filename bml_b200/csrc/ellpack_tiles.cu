// Tile form of the unordered X^2 of a symmetric ELLPACK matrix: the same
// result set as the unordered kernel's symmetric form (ellpack_x2_fast.cu;
// ellpack/bml_multiply_ellpack_typed.c:252-333), with the products formed by
// FP64 tensor instructions (mma.sync m8n8k4) on 8 x 8 tiles.
//
// Why.  The shared-memory accumulator of the unordered kernel is bound by the
// shared atomics: 0.39 T products/s on the 40^3 lattice's wide iterate, 2 % of
// the FP64 pipe.  The matrices of this path are local in row order (bands, and
// runs along x on a lattice), so rows i..i+7 touch nearly the same columns and
// X packs into 8 x 8 tiles that are a fifth to a half full.  Multiplying the
// padded tiles costs 5 to 20 times the products of the sparse form, at 37
// TFLOP/s (18.5 T products/s) and with the sums in registers.
//
// X is symmetric, so X^2 = X X^T and C(I,K) = sum_J X(I,J) X(K,J)^T: both
// operands are tiles of block rows, stored once, in the order in which a
// warp's lanes hold them (element (r, c) of a tile at 2 (4 r + c % 4) + c / 4,
// the A fragments of the two k-steps next to each other, so a tile is 16 bytes
// per lane; as the second operand of X X^T the same order is the B fragment).
//
// Work unit: a group is 32 rows (4 tile rows).  A group lists the tile columns
// J that any of its 4 tile rows touches, with a 4-bit mask and room for four
// tiles, and a bitmap over J ranked by word.  One warp forms the 32 x 32 block
// C(G,H), H >= G: it intersects the bitmaps of G and H, and for every common J
// multiplies the pairs of tiles present (up to 16, two m8n8k4 each) into 16
// accumulator tiles (64 registers a lane).  The tiles travel through a ring in
// shared memory, each lane copying (cp.async) what it will read, two columns
// ahead: from registers loaded one column ahead the kernel waited for L2 (12
// warps per SM, 29.0 ms on the 40^3 iterate; the ring frees registers for 16
// warps, 24.3 ms).  Groups of 16 rows would load more tiles per product, of 64
// would not fit the registers.
//
// The kept entries of a block (|c| > threshold, or the diagonal) are packed:
// 32 row masks and the kept values, in a pool, with the block's place in a
// table [G][H - G].  Nothing is ordered between warps.  A second kernel
// writes the rows of C: for a group it walks the blocks (H, G), H <= G,
// transposed, and then (G, H), so every row comes out in ascending column
// order, exactly symmetric, and without a sort.
//
// The masked product (the adjoint's C = A B at a given pattern) runs on the
// same kernel, the second operand packed as rows of its transpose, the blocks
// those that hold an entry of the pattern.
//
// Which form.  The counts of both forms' products decide (TILE_COST,
// general_pays).  A counting kernel makes them, and a sample of entries looks
// for mirrors, so that an X that is not symmetric is mostly known before it is
// packed; a small X is counted while it is packed, and the symmetry check tells
// the host at its start what was counted, so that a form that does not apply
// costs the fill kernel and not the rest (X^2 without symmetry, us, sparse form
// alone | with a packing and a wait before it | so: 500 rows of 21 59 | 75 |
// 61, 2000 rows of 21 87 | 108 | 88; symmetric but scattered, which the sparse
// form has to check once more: 500 rows of 40 86 | 130 | 108, 4096 rows of 40 259
// | 353 | 285).
//
// The general product (A B, and X^2 of an X that is not symmetric) packs the
// second operand the same way, forms the blocks (G, H) with H on both sides of
// G, and writes rows from them alone.  The columns that a row touches, which
// A B's width check and the diagonal's keep rule ask for, come from the OR of
// the bitmaps of B's rows.
//
// Measured against the sparse form on one B200: X^2 of the 40^3 lattice's wide
// iterate (rows of 825) 65.0 -> 21.1 ms, first X^2 of that lattice (rows of
// 113) 6.3 -> 2.5 ms, FP32 on 26999 rows 2.07 -> 0.82 ms, a chain of 4096 rows
// of 340 745 -> 132 us, of 512 rows of 33 71 -> 55 us; the masked products of
// the adjoint of 3 iterations on the 16^3 lattice 24.4 -> 3.7 ms.
// At 40^3 the MMAs that have both tiles take 9.0 ms of the product kernel's 18,
// those in a pair with only one about 2; the rest is the handling of a common
// column (4.4 products on average there, 7.8 at 30^3).
#include "device_util.cuh"

#include <algorithm>
#include <climits>
#include <cstring>
#include <type_traits>

using namespace b200;

namespace {

constexpr int GR = 32;             // rows of a group
constexpr int PT = 256;            // threads of the per-row and checking kernels
// A group's rows are read by a warp each and written by 32 warps: with 8 warps
// a group, the 128 groups of a 4096-row chain took 64 us to pack and 36 us to
// write (22 and 18 us so); 2000 groups gain a few per cent.
constexpr int FT = 1024, RT = 1024;
constexpr int TW = 4;              // warps of a product CTA
constexpr int TMIN = 4;            // CTAs per SM: 128 registers a thread
constexpr int SG = 48, SC = 32;    // a patch of blocks (G, H - G)
constexpr int TS = 3;              // common tile columns whose tiles a warp has in flight or in use
constexpr int QCAP = 128;          // common tile columns a warp lists at a time (at least 32)
constexpr int WARP_SMEM = TS * 4096 + QCAP * 8;
constexpr size_t TL_SMALL = 40960; // place in the context's small buffers

// The tile form runs when its tile products, at TILE_COST sparse products
// each, are fewer than the sparse form's (X^2 of random band patterns, tile
// form against sparse form in us, by sparse products per tile product: 0.33
// 3880 to 7360 / 3840, 0.64 2050 / 2110, 1.45 (2000 rows) 167 to 185 / 134,
// 1.88 847 / 1770, 1.94 370 / 807, 5.3 140 / 475; lattices have 8 to 70).
constexpr double TILE_COST = 1.5;
constexpr long long LAZY_BYTES = 128 << 20; // most tile places of a matrix laid out without counting them

// 0 never, 1 where the rules below take it for the faster form, 2 wherever it applies.
int g_tiles = 1;

struct TileFlags
{
    unsigned long long products; // the sparse form's products: sum over rows of width^2 (X symmetric), or over entries
    unsigned long long stored;   // entries of X
    unsigned long long tiles2;   // tile products: sum over tile rows of tiles^2, or over tiles
    unsigned long long pool;     // words of the packed result taken
    int entries;                 // (group, J) entries handed out
    int counted;                 // those the counting kernels found
    int reach, reachB;           // largest |column - row|; of the second operand
    int bad;                     // a row length or column out of range
    int odd;                     // an entry not finite, or a row whose tiles are zero: not for this form
    int asym;
    int alone;                   // tiles above the groups' diagonal blocks that have a mirror, less those below
    int next;                    // work item counter
    int full;                    // the pool ran out
    int overflow, max_width;
    int skipped;                 // a group was not packed
    int counters, done;          // CTAs of the counting and of the row kernel that have finished
    int blocks;                  // blocks of the masked product
    double trA, trC;
};

struct TileArgs
{
    const void *Xv; const int *Xi; const int *Xn; int ld; int N; int ncols;
    int NG, nw;                  // groups; words of a group's bitmap
    unsigned *bits;              // [NG][nw] union bitmap over tile columns
    unsigned short *rank;        // [NG][nw] entries before the word
    int *eoff;                   // first entry of the group
    int2 *range;                 // words {first, last} of the group's bitmap that are used
    int *last;                   // last group H whose block with G can be non-zero
    unsigned *ent;               // entry << 4 | mask of the tile rows present; its tiles at 4 entry + row
    unsigned short *entJ;        // tile column of an entry
    double *tiles;               // 64 doubles per tile, four places per entry
    int *tileN, *tileC;          // product of two matrices: tiles of a tile row of B, of a tile column of A
    const int *nB;               // row lengths of B
    double cost;                 // sparse products that a tile product is taken for (0: whatever they are)
    int4 *early;                 // pinned: {told, products, tile products, stored entries * 2 + asym} before the check
    int sample;                  // who counts looks for the mirrors of a few entries, and packs no group that packs badly
    int *tab; int span;          // [NG][span] place of block (G, G + s) in the pool, or -1
    unsigned long long *pool; unsigned long long cap;
    void *Cv; int *Ci; int *Cn; int ldc; int Mc;
    double thr;
    double *dA, *dC;             // per-group sums of the diagonals of X and X^2
    TileFlags *flags, *host;     // host: pinned, written by the last CTA of the counting and of the row kernel,
    int told;                    // which then set the word behind it to this
    // second operand, as rows of its transpose (the sparse X^2: the same lists)
    const unsigned *bitsB; const unsigned short *rankB; const int *eoffB; const int2 *rangeB;
    // masked product
    unsigned *gb;                // [NG][4][nw] bitmaps of the transpose of X, made by its rows
    const int *Pi; const int *Pn; int ldp; int hw; // pattern; words of a bitmap over groups
    unsigned *pbits; int *prank; // [NG][hw] groups H with an entry of the pattern, and blocks before the word
    int2 *pblk;                  // blocks (G, H) of the pattern
    double *out;                 // 1024 doubles per block
    int masked, count_only;
    // general product
    int general, back;           // blocks (G, G - back + s), s < span
    unsigned *rowbits; int rw;   // [N][rw] bitmaps of B's rows
    int *touched;                // rows of C whose diagonal is touched
    int reach, check_pre;
};

constexpr int TOLD = 32; // the word behind the host's copy of the flags
constexpr size_t EARLY = 1024; // and where the early counts lie

// The flags as they are in L2, into the host's copy, and then the word that
// the host waits for (0: it waits for the kernel); one warp.
__device__ __forceinline__ void tell_host(const TileArgs &g, int lane)
{
    static_assert(sizeof(TileFlags) <= TOLD * sizeof(int), "a word per lane");
    volatile int *host = reinterpret_cast<volatile int *>(g.host);
    if (lane < (int) (sizeof(TileFlags) / sizeof(int)))
        host[lane] = reinterpret_cast<const volatile int *>(g.flags)[lane];
    __threadfence_system();
    __syncwarp();
    if (lane == 0 && g.told)
        host[TOLD] = g.told;
}

// By the counts the sparse form does better, or a sample told that X is not
// symmetric.
__host__ __device__ __forceinline__ bool left_to_sparse(const TileFlags &f, double cost)
{
    return f.bad || f.asym || (double) f.tiles2 * cost > (double) f.products;
}

// The form does not apply: the kernels after the fill do nothing.  (`alone` says
// so only when the symmetry check is through; the others are set for good.)
__device__ __forceinline__ bool unpacked(const TileArgs &g)
{
    const TileFlags *f = g.flags;
    return f->bad || f->odd || f->skipped || (!g.general && left_to_sparse(*f, g.cost));
}
__device__ __forceinline__ bool declined(const TileArgs &g)
{
    return unpacked(g) || (!g.general && g.flags->alone);
}

// The four tile rows' bitmaps of group G from the stored columns, in shared
// memory, and which rows are strictly ascending (bit of *order; zero before);
// false (uniform) when a row or column is out of range.
template <bool CROSS>
__device__ __forceinline__ bool group_bitmaps(const TileArgs &g, int G, unsigned *bm, int *reach, unsigned *order,
                                              unsigned long long *products)
{
    for (int w = threadIdx.x; w < 4 * g.nw; w += FT)
        bm[w] = 0u;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int bad = 0, far = 0;
    unsigned long long prod = 0;
    for (int r = warp; r < GR; r += FT / 32)
    {
        const int i = G * GR + r;
        if (i >= g.N)
            continue;
        const int n = g.Xn[i];
        if (n < 0 || n > g.ld)
        {
            bad = 1;
            continue;
        }
        unsigned *row = bm + (r >> 3) * g.nw;
        bool desc = false;
        for (int p0 = lane; p0 < n; p0 += 128)
        {
            int kk[4], next[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
            {
                const int *at = g.Xi + (size_t) i * g.ld + p0 + 32 * u;
                kk[u] = p0 + 32 * u < n ? __ldg(at) : i;
                next[u] = p0 + 32 * u + 1 < n ? __ldg(at + 1) : INT_MAX;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
            {
                const int k = kk[u];
                if (p0 + 32 * u >= n)
                    continue;
                desc |= next[u] <= k;
                if (k < 0 || k >= g.ncols)
                {
                    bad = 1;
                    continue;
                }
                far = max(far, abs(k - i));
                if (CROSS)
                    prod += max(0, __ldg(g.nB + k));
                const unsigned bit = 1u << ((k >> 3) & 31);
                if (!(*(volatile unsigned *) &row[k >> 8] & bit))
                    atomicOr(&row[k >> 8], bit);
            }
        }
        if (order && !__any_sync(FULL, desc) && lane == 0)
            atomicOr(order, 1u << r);
    }
    *reach = far;
    if (CROSS)
        *products = prod;
    return __syncthreads_or(bad) == 0;
}

// Tiles of each tile row and entries of group G (tot[0..4], zero before), and
// its share of both forms' products and of the reach; sums[0..2] (zero
// before): products, tile products, stored entries.  CROSS: of a product of two
// matrices (products: this thread's; the tiles go to their columns).
template <bool CROSS>
__device__ __forceinline__ void group_counts(const TileArgs &g, int G, const unsigned *bm, int far,
                                             unsigned long long products, int *tot, unsigned long long *sums)
{
    int c[5] = {0, 0, 0, 0, 0};
    for (int w = threadIdx.x; w < g.nw; w += FT)
    {
        unsigned any = 0u;
#pragma unroll
        for (int a = 0; a < 4; ++a)
        {
            const unsigned b = bm[a * g.nw + w];
            c[a] += __popc(b);
            any |= b;
        }
        c[4] += __popc(any);
        if (CROSS)
            for (unsigned m = any; m; m &= m - 1)
            {
                const int q = __ffs(m) - 1;
                int n = 0;
#pragma unroll
                for (int a = 0; a < 4; ++a)
                    n += bm[a * g.nw + w] >> q & 1u;
                atomicAdd(&g.tileC[w * 32 + q], n);
            }
    }
    const int n1 = threadIdx.x < GR && G * GR + threadIdx.x < g.N ? g.Xn[G * GR + threadIdx.x] : 0;
    int n = n1;
    unsigned long long n2 = CROSS ? products : (unsigned long long) n1 * n1;
    for (int o = 16; o; o >>= 1)
    {
#pragma unroll
        for (int a = 0; a < 5; ++a)
            c[a] += __shfl_xor_sync(FULL, c[a], o);
        n += __shfl_xor_sync(FULL, n, o);
        n2 += __shfl_xor_sync(FULL, n2, o);
        far = max(far, __shfl_xor_sync(FULL, far, o));
    }
    if ((threadIdx.x & 31) == 0)
    {
#pragma unroll
        for (int a = 0; a < 5; ++a)
            if (c[a])
                atomicAdd(&tot[a], c[a]);
        if (n2)
            atomicAdd(&sums[0], n2);
        if (n)
            atomicAdd(&sums[2], (unsigned long long) n);
        if (far > *(volatile int *) &g.flags->reach)
            atomicMax(&g.flags->reach, far);
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        unsigned long long t2 = 0;
        for (int a = 0; a < 4 && !CROSS; ++a)
            t2 += (unsigned long long) tot[a] * tot[a];
        sums[1] = t2;
        atomicAdd(&g.flags->products, sums[0]);
        atomicAdd(&g.flags->stored, sums[2]);
        if (!CROSS)
            atomicAdd(&g.flags->tiles2, t2);
        atomicAdd(&g.flags->counted, tot[4]);
    }
}

// A look for the mirror of a row's last entry, in two parts, so that the loads
// of the first are under way while the caller counts; missing() tells of a row
// without it.  (Of ascending rows the mirror is the first in its own: any entry
// of rows of 700 took 8 us longer to find.)  One warp.
template <typename T, int U> struct MirrorSample
{
    int i, k, kk[U];
    T x, v[U];

    __device__ __forceinline__ void choose(const TileArgs &g, int row)
    {
        i = row;
        k = -1;
        const int n = i < g.N ? g.Xn[i] : 0;
        if (n < 1 || n > g.ld)
            return;
        const size_t at = (size_t) i * g.ld + n - 1;
        k = __ldg(g.Xi + at);
        x = __ldg(static_cast<const T *>(g.Xv) + at);
    }
    __device__ __forceinline__ void load(const TileArgs &g, int p0, int lane)
    {
#pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const int p = p0 + 32 * u + lane;
            const size_t at = (size_t) k * g.ld + p;
            kk[u] = k >= 0 && k < g.N && p < g.ld ? __ldg(g.Xi + at) : -1;
            v[u] = k >= 0 && k < g.N && p < g.ld ? __ldg(static_cast<const T *>(g.Xv) + at) : T(0);
        }
    }
    __device__ __forceinline__ bool missing(const TileArgs &g, int lane)
    {
        if (k < 0 || k >= g.N)
            return false;
        const int m = min(g.Xn[k], g.ld);
        bool twin = false;
        for (int p0 = 0;;)
        {
#pragma unroll
            for (int u = 0; u < U; ++u)
                twin |= p0 + 32 * u + lane < m && kk[u] == i && v[u] == x;
            p0 += 32 * U;
            if (__any_sync(FULL, twin) || p0 >= m)
                break;
            load(g, p0, lane);
        }
        return !__any_sync(FULL, twin);
    }
};

// The last CTA of a launch to come here (uniform), with what all have counted.
__device__ __forceinline__ bool last_cta(const TileArgs &g, int *fin)
{
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence(); // this CTA's counts come before its own
        *fin = atomicAdd(&g.flags->counters, 1) == (int) gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    return *fin;
}

// Counts: tiles, entries and the products of both forms.
// Two CTAs per SM, and so 32 registers a thread: one took 45 us instead of 27
// for 26999 rows.
template <typename T> __global__ void __launch_bounds__(FT, 2) tile_count_kernel(TileArgs g)
{
    extern __shared__ unsigned bm[];
    __shared__ int tot[5];
    __shared__ unsigned long long sums[3];
    __shared__ int fin;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int G = blockIdx.x; G < g.NG; G += gridDim.x)
    {
        if (threadIdx.x < 5)
            tot[threadIdx.x] = 0;
        if (threadIdx.x < 3)
            sums[threadIdx.x] = 0;
        // one row in eight of one group in 32 (in eight: 15 us of the 120 for 64000 rows of 925)
        MirrorSample<T, 1> look;
        const bool looks = g.sample && !(G & 31) && !(warp & 7);
        if (looks)
            look.choose(g, G * GR + warp);
        int far = 0;
        if (!group_bitmaps<false>(g, G, bm, &far, nullptr, nullptr))
        {
            if (threadIdx.x == 0)
                atomicExch(&g.flags->bad, 1);
            break;
        }
        if (looks)
            look.load(g, 0, lane);
        group_counts<false>(g, G, bm, far, 0, tot, sums);
        if (looks && look.missing(g, lane) && lane == 0)
            atomicExch(&g.flags->asym, 1);
        __syncthreads();
    }
    if (g.told && last_cta(g, &fin) && warp == 0)
        tell_host(g, lane);
}

// Before the counts of a product of two matrices: whether the row lengths speak
// for tiles at all.  The counts are left out if not, and the host, told by one
// store of 8 bytes, begins the sparse form.  One CTA.
__global__ void __launch_bounds__(1024) tile_lengths_kernel(TileArgs a, TileArgs b, int told)
{
    const int go = rows_for_tiles(a.Xn, a.ld, b.Xn, b.ld, a.N);
    if (threadIdx.x)
        return;
    a.flags->skipped = !go;
    asm volatile("st.volatile.global.v2.s32 [%0], {%1, %2};" ::"l"(a.early), "r"(told), "r"(go) : "memory");
}

// The same for a product of two matrices: a's counts, the products of its
// entries with b's rows, and, once all groups of both have been through, the
// tile products: tiles of a's tile column J times tiles of b's tile row J.
__global__ void __launch_bounds__(FT, 2) tile_cross_kernel(TileArgs a, TileArgs b)
{
    extern __shared__ unsigned bm[];
    __shared__ int tot[5];
    __shared__ unsigned long long sums[3];
    __shared__ int fin;
    const int lane = threadIdx.x & 31;
    if (a.flags->skipped)
        return;
    bool ok = true;
    for (int q = blockIdx.x; ok && q < 2 * a.NG; q += gridDim.x)
    {
        if (threadIdx.x < 5)
            tot[threadIdx.x] = 0;
        if (threadIdx.x < 3)
            sums[threadIdx.x] = 0;
        int far = 0;
        unsigned long long products = 0;
        if (q < a.NG)
        {
            ok = group_bitmaps<true>(a, q, bm, &far, nullptr, &products);
            if (ok)
                group_counts<true>(a, q, bm, far, products, tot, sums);
        }
        else
        {
            ok = group_bitmaps<false>(b, q - a.NG, bm, &far, nullptr, nullptr);
            // a warp per tile row
            if (ok && threadIdx.x < 128)
            {
                int n = 0;
                for (int w = lane; w < b.nw; w += 32)
                    n += __popc(bm[(threadIdx.x >> 5) * b.nw + w]);
                for (int o = 16; o; o >>= 1)
                    n += __shfl_xor_sync(FULL, n, o);
                if (lane == 0)
                    a.tileN[4 * (q - a.NG) + (threadIdx.x >> 5)] = n;
            }
        }
        __syncthreads();
    }
    if (!ok && threadIdx.x == 0)
        atomicExch(&a.flags->bad, 1);
    if (!last_cta(a, &fin))
        return;
    unsigned long long t2 = 0;
    for (int J = threadIdx.x; J < 4 * a.NG; J += FT)
        t2 += (unsigned long long) __ldcg(a.tileC + J) * __ldcg(a.tileN + J);
    for (int o = 16; o; o >>= 1)
        t2 += __shfl_xor_sync(FULL, t2, o);
    if (lane == 0)
        atomicAdd(&a.flags->tiles2, t2);
    __threadfence();
    __syncthreads();
    if (threadIdx.x < 32)
        tell_host(a, lane);
}

__device__ __forceinline__ int tile_at(int r, int c) { return 2 * (4 * r + (c & 3)) + (c >> 2); }

// Lists, zero-filled tiles and the scatter of group G's entries.  Rows in
// ascending order have distinct columns and are stored; other rows are added
// (duplicate columns add up, as they do in the sparse form).
// LAZY: there was no counting pass, and no more groups than SMs.
// CTAS per SM: two for narrow rows, one, with the registers for its loads, for
// wide ones (FP64, of the whole call: 20000 rows of 101 193 us with two and 201
// with one, 8000 of 257 397 and 398; the kernel on 64000 of 925 652 and 600).
template <typename T, bool LAZY, int CTAS> __global__ void __launch_bounds__(FT, CTAS) tile_fill_kernel(TileArgs g)
{
    extern __shared__ unsigned bm[]; // [4][nw] bitmaps | [nw] entries before the word
    int *before = reinterpret_cast<int *>(bm + 4 * g.nw);
    __shared__ int wsum[FT / 32];
    __shared__ int run, place;
    __shared__ unsigned order; // rows in strictly ascending order
    __shared__ int2 used;
    __shared__ double diag[GR];
    __shared__ int tot[5];
    __shared__ unsigned long long sums[3];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int G = blockIdx.x; G < g.NG; G += gridDim.x)
    {
        if (tid == 0)
        {
            run = 0;
            order = 0u;
            used = make_int2(INT_MAX, -1);
        }
        if (tid < 5)
            tot[tid] = 0;
        if (tid < 3)
            sums[tid] = 0;
        MirrorSample<T, 4> look;
        const bool looks = LAZY && g.sample && !(warp & 7);
        if (looks)
            look.choose(g, G * GR + warp);
        int far = 0;
        if (g.gb)
        {
            for (int w = tid; w < 4 * g.nw; w += FT)
                bm[w] = g.gb[(size_t) G * 4 * g.nw + w];
            __syncthreads();
        }
        else if (!group_bitmaps<false>(g, G, bm, &far, &order, nullptr))
        {
            if (tid == 0)
                atomicExch(&g.flags->bad, 1);
            return;
        }
        if (LAZY)
        {
            if (looks)
                look.load(g, 0, lane);
            group_counts<false>(g, G, bm, far, 0, tot, sums);
            const bool alone = looks && look.missing(g, lane);
            if (alone && lane == 0)
                atomicExch(&g.flags->asym, 1);
            // a group that packs badly is not packed until the counts of all say that the others make up for it
            const bool badly = g.sample && (double) sums[1] * g.cost > 2.0 * (double) sums[0];
            if (badly && tid == 0)
                g.flags->skipped = 1;
            if (__syncthreads_or(alone || badly))
                continue;
        }
        for (int s = tid; s < g.span; s += FT)
            g.tab[(size_t) G * g.span + s] = -1;
        if (tid == 0 && !g.masked)
            g.dC[G] = 0.0;
        // entries before every word (block prefix, FT words at a time)
        for (int w0 = 0; w0 < g.nw; w0 += FT)
        {
            const int w = w0 + tid;
            const unsigned any =
                w < g.nw ? bm[w] | bm[g.nw + w] | bm[2 * g.nw + w] | bm[3 * g.nw + w] : 0u;
            const int n = __popc(any);
            int sum = n;
            for (int o = 1; o < 32; o <<= 1)
            {
                const int u = __shfl_up_sync(FULL, sum, o);
                if (lane >= o)
                    sum += u;
            }
            if (lane == 31)
                wsum[warp] = sum;
            __syncthreads();
            int base = run;
            for (int v = 0; v < warp; ++v)
                base += wsum[v];
            if (w < g.nw)
            {
                g.bits[(size_t) G * g.nw + w] = any;
                g.rank[(size_t) G * g.nw + w] = (unsigned short) (base + sum - n);
                before[w] = base + sum - n;
                if (any)
                {
                    atomicMin(&used.x, w);
                    atomicMax(&used.y, w);
                }
            }
            __syncthreads();
            if (tid == FT - 1)
                run = base + sum;
            __syncthreads();
        }
        if (tid == 0)
        {
            place = atomicAdd(&g.flags->entries, run);
            g.eoff[G] = place;
            g.range[G] = used.y < 0 ? make_int2(0, -1) : used; // an empty group intersects nothing
        }
        __syncthreads();
        const int e0 = place, ne = run;
        for (int w = tid; w < g.nw; w += FT)
        {
            unsigned b[4];
#pragma unroll
            for (int a = 0; a < 4; ++a)
                b[a] = bm[a * g.nw + w];
            unsigned any = b[0] | b[1] | b[2] | b[3];
            for (int e = e0 + before[w]; any; ++e)
            {
                const int q = __ffs(any) - 1;
                any &= any - 1;
                unsigned m = 0u;
#pragma unroll
                for (int a = 0; a < 4; ++a)
                    m |= ((b[a] >> q) & 1u) << a;
                g.ent[e] = (unsigned) e << 4 | m;
                g.entJ[e] = (unsigned short) (w * 32 + q);
            }
        }
        __syncthreads();
        double2 *z = reinterpret_cast<double2 *>(g.tiles + (size_t) e0 * 256);
        for (int p = tid; p < ne * 128; p += FT)
            if (g.ent[e0 + (p >> 7)] >> ((p >> 5) & 3) & 1u)
                z[p] = make_double2(0.0, 0.0);
        __syncthreads();
        if (g.gb) // the transpose's entries are placed by tile_scatter_kernel
            continue;
        int odd = 0;
        for (int r = warp; r < GR; r += FT / 32)
        {
            const int i = G * GR + r;
            if (i >= g.N)
            {
                if (lane == 0)
                    diag[r] = 0.0;
                continue;
            }
            const int n = g.Xn[i];
            const T *xv = static_cast<const T *>(g.Xv) + (size_t) i * g.ld;
            const int *xi = g.Xi + (size_t) i * g.ld;
            const bool sorted = order >> r & 1u;
            const int a = r >> 3;
            double d = 0.0;
            for (int p0 = lane; p0 < n; p0 += 128)
            {
                int kk[4];
                T vv[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                {
                    const int p = p0 + 32 * u;
                    kk[u] = p < n ? __ldg(xi + p) : 0;
                    vv[u] = p < n ? __ldg(xv + p) : T(0);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                {
                    if (p0 + 32 * u >= n)
                        continue;
                    const int k = kk[u];
                    const double v = (double) vv[u];
                    odd |= !(fabs(v) <= 1.7976931348623157e308);
                    if (k == i)
                        d += v;
                    const int w = k >> 8;
                    const unsigned below = (1u << ((k >> 3) & 31)) - 1u;
                    const unsigned any = bm[w] | bm[g.nw + w] | bm[2 * g.nw + w] | bm[3 * g.nw + w];
                    const int t = 4 * (e0 + before[w] + __popc(any & below)) + a;
                    double *at = g.tiles + (size_t) t * 64 + tile_at(r & 7, k & 7);
                    if (sorted)
                        *at = v;
                    else
                        atomicAdd(at, v);
                }
            }
            for (int o = 16; o; o >>= 1)
                d += __shfl_xor_sync(FULL, d, o);
            if (lane == 0)
                diag[r] = d;
        }
        if (__syncthreads_or(odd) && tid == 0)
            atomicExch(&g.flags->odd, 1);
        if (warp == 0 && !g.masked)
        {
            double d = diag[lane];
            for (int o = 16; o; o >>= 1)
                d += __shfl_xor_sync(FULL, d, o);
            if (lane == 0)
                g.dA[G] = d;
        }
        __syncthreads();
    }
}

// Every tile (I, J), J >= I, against tile (J, I): equal bits, or no tile and
// zeros.  A tile below its group's diagonal block has a mirror when the tiles
// there are as many as those above that have one: checking that each has its
// mirror took the lists of the other group once more.  Also the last group H
// that has a column in common with G.
__global__ void __launch_bounds__(PT) tile_sym_kernel(TileArgs g)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ int lastH, alone;
    if (g.early && blockIdx.x == 0 && threadIdx.x == 0)
        // one store of 16 bytes: the host sees all of it or nothing
        asm volatile("st.volatile.global.v4.s32 [%0], {%1, %2, %3, %4};" ::"l"(g.early), "r"(g.told),
                     "r"(__float_as_int((float) g.flags->products)), "r"(__float_as_int((float) g.flags->tiles2)),
                     "r"((int) g.flags->stored * 2 + (g.flags->asym || g.flags->bad))
                     : "memory");
    if (__syncthreads_or(unpacked(g))) // other CTAs may find an entry without its mirror meanwhile
        return;
    for (int G = blockIdx.x; G < g.NG; G += gridDim.x)
    {
        if (threadIdx.x == 0)
        {
            lastH = G;
            alone = 0;
        }
        __syncthreads();
        const int2 rg = g.range[G];
        int ne = 0;
        if (rg.y >= 0)
            ne = g.rank[(size_t) G * g.nw + rg.y] + __popc(g.bits[(size_t) G * g.nw + rg.y]);
        int last = G, asym = 0, mirrors = 0;
        for (int e = warp; e < ne; e += PT / 32)
        {
            const unsigned en = g.ent[g.eoff[G] + e];
            const int J = g.entJ[g.eoff[G] + e];
            const int H = J >> 2;
            const int2 rh = H < g.NG ? g.range[H] : make_int2(0, -1);
            // the four tile rows of G lie in one word of H's bitmap, its tiles there are consecutive entries
            const int s0 = (4 * G) & 31;
            const bool in = H < g.NG && J >= 4 * G;
            const unsigned b = in ? g.bits[(size_t) H * g.nw + (4 * G >> 5)] : 0u;
            int f = in ? g.eoff[H] + g.rank[(size_t) H * g.nw + (4 * G >> 5)] + __popc(b & ((1u << s0) - 1u)) : 0;
            if (rh.y >= 0)
            {
                // the last tile column of group H
                const unsigned bl = g.bits[(size_t) H * g.nw + rh.y];
                last = max(last, (rh.y * 32 + 31 - __clz(bl)) >> 2);
            }
            if (J < 4 * G)
            {
                mirrors -= __popc(en & 15u);
                continue;
            }
            const double2 *tp = reinterpret_cast<const double2 *>(g.tiles) + (size_t) (en >> 4) * 128 + lane;
            double2 x[4];
            double m0[4], m1[4];
#pragma unroll
            for (int a = 0; a < 4; ++a)
            {
                x[a] = make_double2(0.0, 0.0);
                m0[a] = m1[a] = 0.0;
                const unsigned fn = b >> (s0 + a) & 1u ? g.ent[f++] : 0u;
                const bool both = fn >> (J & 3) & 1u;
                if (en >> a & 1u)
                {
                    x[a] = tp[32 * a];
                    if (both)
                    {
                        mirrors += J >= 4 * G + 4;
                        const double *q = g.tiles + (size_t) (4 * (fn >> 4) + (J & 3)) * 64;
                        const int r = lane >> 2, c = lane & 3;
                        m0[a] = q[tile_at(c, r)];
                        m1[a] = q[tile_at(c + 4, r)];
                    }
                }
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
                asym |= x[a].x != m0[a] || x[a].y != m1[a];
        }
        for (int o = 16; o; o >>= 1)
            last = max(last, __shfl_xor_sync(FULL, last, o));
        if (lane == 0)
        {
            atomicMax(&lastH, last);
            atomicAdd(&alone, mirrors);
        }
        asym = __syncthreads_or(asym);
        if (threadIdx.x == 0)
        {
            if (alone)
                atomicAdd(&g.flags->alone, alone);
            g.last[G] = min(lastH, g.NG - 1);
            if (asym)
                atomicExch(&g.flags->asym, 1);
        }
        __syncthreads();
    }
}

template <typename T> __device__ __forceinline__ bool over(T x, double thr);
template <> __device__ __forceinline__ bool over<double>(double x, double thr) { return fabs(x) > thr; }
template <> __device__ __forceinline__ bool over<float>(float x, double thr) { return fabsf(x) > (float) thr; }

#define TILE_BITS(E)                                                                                                    \
    "{\n\t.reg .pred p0, p1, p2, p3;\n\t.reg .b32 t;\n\t"                                                             \
    "and.b32 t, " E ", 1;\n\tsetp.ne.b32 p0, t, 0;\n\tand.b32 t, " E ", 2;\n\tsetp.ne.b32 p1, t, 0;\n\t"               \
    "and.b32 t, " E ", 4;\n\tsetp.ne.b32 p2, t, 0;\n\tand.b32 t, " E ", 8;\n\tsetp.ne.b32 p3, t, 0;\n\t"

// The tiles present of one entry into a stage, 16 bytes per lane each.  An
// entry has room for four tiles, so a tile's place is the entry's plus a
// constant.
__device__ __forceinline__ void copy_tiles(unsigned dst, const double2 *tiles, unsigned en)
{
    asm volatile(TILE_BITS("%2")
                 "@p0 cp.async.cg.shared.global [%0], [%1], 16;\n\t"
                 "@p1 cp.async.cg.shared.global [%0 + 512], [%1 + 512], 16;\n\t"
                 "@p2 cp.async.cg.shared.global [%0 + 1024], [%1 + 1024], 16;\n\t"
                 "@p3 cp.async.cg.shared.global [%0 + 1536], [%1 + 1536], 16;\n\t}" ::"r"(dst),
                 "l"(tiles + (size_t) (en >> 4) * 128), "r"(en)
                 : "memory");
}

// The same tiles from the stage (each lane reads what it copied).
__device__ __forceinline__ void load_tiles(unsigned src, unsigned en, double2 (&f)[4])
{
    asm volatile(TILE_BITS("%9")
                 "@p0 ld.shared.v2.f64 {%0, %1}, [%8];\n\t"
                 "@p1 ld.shared.v2.f64 {%2, %3}, [%8 + 512];\n\t"
                 "@p2 ld.shared.v2.f64 {%4, %5}, [%8 + 1024];\n\t"
                 "@p3 ld.shared.v2.f64 {%6, %7}, [%8 + 1536];\n\t}"
                 : "+d"(f[0].x), "+d"(f[0].y), "+d"(f[1].x), "+d"(f[1].y), "+d"(f[2].x), "+d"(f[2].y), "+d"(f[3].x),
                   "+d"(f[3].y)
                 : "r"(src), "r"(en)
                 : "memory");
}

#define TILE_MMA(P, C0, C1, AX, BX) \
    "@" P " mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {" C0 ", " C1 "}, {" AX "}, {" BX "}, {" C0 ", " C1 "};\n\t"

// A tile of the first operand against two adjacent ones of the second, where
// present; the first k-step of both before the second of either, so that no
// MMA waits for the one before it.
__device__ __forceinline__ void mul_pair(unsigned bit0, unsigned bit1, const double2 &A, const double2 &B0,
                                         const double2 &B1, double (&c0)[2], double (&c1)[2])
{
    asm volatile("{\n\t.reg .pred p0, p1;\n\tsetp.ne.b32 p0, %10, 0;\n\tsetp.ne.b32 p1, %11, 0;\n\t"
                 TILE_MMA("p0", "%0", "%1", "%4", "%6") TILE_MMA("p1", "%2", "%3", "%4", "%8")
                 TILE_MMA("p0", "%0", "%1", "%5", "%7") TILE_MMA("p1", "%2", "%3", "%5", "%9") "}"
                 : "+d"(c0[0]), "+d"(c0[1]), "+d"(c1[0]), "+d"(c1[1])
                 : "d"(A.x), "d"(A.y), "d"(B0.x), "d"(B0.y), "d"(B1.x), "d"(B1.y), "r"(bit0), "r"(bit1));
}

// An MMA whose predicate is off still takes its cycles of the tensor pipe (75 %
// busy with half of its instructions off, when only the rows of the first
// operand were branched over), so pairs without a tile are branched over too:
// the masks are mostly runs.  X^2 of the 40^3 iterate: 24.3 ms with a branch
// per row, 21.9 per pair, 24.8 per tile, 22.2 with a jump on the second mask,
// 36.0 with a jump on both (225 straight pieces miss the instruction cache).
__device__ __forceinline__ void mul_tiles(unsigned ea, unsigned eb, const double2 (&A)[4], const double2 (&B)[4],
                                          double (&acc)[4][4][2])
{
#pragma unroll
    for (int a = 0; a < 4; ++a)
        if (ea >> a & 1u)
        {
            if (eb & 3u)
                mul_pair(eb & 1u, eb & 2u, A[a], B[0], B[1], acc[a][0], acc[a][1]);
            if (eb & 12u)
                mul_pair(eb & 4u, eb & 8u, A[a], B[2], B[3], acc[a][2], acc[a][3]);
        }
}

// Blocks C(G, H), one warp each: H >= G of a symmetric square, those that hold
// an entry of the pattern, or H on both sides of G.
constexpr int TILE_SQUARE = 0, TILE_MASKED = 1, TILE_GENERAL = 2;

template <typename T, int MODE> __global__ void __launch_bounds__(TW * 32, TMIN) tile_x2_kernel(TileArgs g)
{
    constexpr bool MASKED = MODE == TILE_MASKED, GENERAL = MODE == TILE_GENERAL;
    extern __shared__ __align__(16) unsigned char tsm[]; // per warp: stages[TS][8 tiles] | queue[QCAP]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (__any_sync(FULL, MASKED ? g.flags->odd : declined(g))) // other warps may set odd meanwhile
        return;
    uint2 *qu = reinterpret_cast<uint2 *>(tsm + warp * WARP_SMEM + TS * 4096);
    const unsigned stage0 = (unsigned) __cvta_generic_to_shared(tsm + warp * WARP_SMEM) + lane * 16;
    const double2 *tiles = reinterpret_cast<const double2 *>(g.tiles) + lane;
    // blocks in patches of SG x SC of (G, H - G), claimed by warps: the blocks in flight read a compact set of
    // groups from L2
    const int pc = (g.span + SC - 1) / SC;
    const int items = MASKED ? g.flags->blocks : (g.NG + SG - 1) / SG * pc * (SG * SC);
    for (;;)
    {
        int it = 0;
        if (lane == 0)
            it = atomicAdd(&g.flags->next, 1);
        it = __shfl_sync(FULL, it, 0);
        if (it >= items)
            break;
        int G, H, s = 0;
        if (MASKED)
        {
            const int2 e = g.pblk[it];
            G = e.x;
            H = e.y;
        }
        else
        {
            const int patch = it / (SG * SC), in = it % (SG * SC);
            G = patch / pc * SG + in % SG;
            s = patch % pc * SC + in / SG;
            H = GENERAL ? G - g.back + s : G + s;
            if (G >= g.NG || s >= g.span || (GENERAL ? H < 0 || H >= g.NG : H > g.last[G]))
                continue;
        }
        const int2 ra = g.range[G], rb = g.rangeB[H];
        const int wlo = max(ra.x, rb.x), whi = min(ra.y, rb.y);
        const int ea0 = g.eoff[G], eb0 = g.eoffB[H];
        double acc[4][4][2];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b)
                acc[a][b][0] = acc[a][b][1] = 0.0;
        bool any = false;
        double2 A[4], Bf[4];
#pragma unroll
        for (int a = 0; a < 4; ++a)
            A[a] = Bf[a] = make_double2(0.0, 0.0);
        int n = 0, w0 = wlo;
        unsigned a = 0u, b = 0u, c = 0u, xa = 0u, xb = 0u;
        for (;;)
        {
            // common tile columns into the queue, as many as fit; a lane holds one word of the bitmaps
            while (!__any_sync(FULL, c != 0u) && w0 <= whi)
            {
                const int w = w0 + lane;
                c = 0u;
                if (w <= whi)
                {
                    a = __ldg(g.bits + (size_t) G * g.nw + w);
                    b = __ldg(g.bitsB + (size_t) H * g.nw + w);
                    xa = g.rank[(size_t) G * g.nw + w];
                    xb = g.rankB[(size_t) H * g.nw + w];
                    c = a & b;
                }
                w0 += 32;
            }
            const bool end = !__any_sync(FULL, c != 0u);
            if (!end)
            {
                any = true;
                const int cnt = __popc(c);
                int pre = cnt;
                for (int o = 1; o < 32; o <<= 1)
                {
                    const int u = __shfl_up_sync(FULL, pre, o);
                    if (lane >= o)
                        pre += u;
                }
                const bool fits = n + pre <= QCAP; // a prefix of the lanes
                const int nfit = __popc(__ballot_sync(FULL, fits));
                if (fits)
                {
                    int at = n + pre - cnt;
                    while (c)
                    {
                        const unsigned below = (c & (0u - c)) - 1u;
                        qu[at++].x = (xa + __popc(a & below)) | (xb + __popc(b & below)) << 16;
                        c &= c - 1;
                    }
                }
                if (nfit)
                    n += __shfl_sync(FULL, pre, nfit - 1);
                __syncwarp();
                if (!__any_sync(FULL, c != 0u) && w0 <= whi && n + 32 <= QCAP)
                    continue; // room for more
            }
            // the entries' tiles through the ring, TS - 1 columns ahead
            __syncwarp();
            for (int t = lane; t < n; t += 32)
            {
                const unsigned q = qu[t].x;
                qu[t] = make_uint2(__ldg(g.ent + ea0 + (q & 0xffffu)), __ldg(g.ent + eb0 + (q >> 16)));
            }
            __syncwarp();
            auto issue = [&](int t) {
                if (t < n)
                {
                    const uint2 e = qu[t];
                    const unsigned st = stage0 + (t % TS) * 4096;
                    copy_tiles(st, tiles, e.x);
                    copy_tiles(st + 2048, tiles, e.y);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
#pragma unroll
            for (int t = 0; t < TS - 1; ++t)
                issue(t);
            for (int t = 0; t < n; ++t)
            {
                asm volatile("cp.async.wait_group %0;" ::"n"(TS - 2) : "memory");
                const uint2 e = qu[t];
                const unsigned st = stage0 + (t % TS) * 4096;
                load_tiles(st, e.x, A);
                load_tiles(st + 2048, e.y, Bf);
                issue(t + TS - 1); // into the stage of column t - 1, whose loads have been used
                mul_tiles(e.x, e.y, A, Bf, acc);
            }
            n = 0;
            __syncwarp();
            if (end)
                break;
        }
        if (MASKED)
        {
            double *o = g.out + (size_t) it * 1024 + (lane >> 2) * 32 + 2 * (lane & 3);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    *reinterpret_cast<double2 *>(o + a * 256 + 8 * b) = make_double2(acc[a][b][0], acc[a][b][1]);
            continue;
        }
        if (!any)
            continue;

        // keep, pack, and place in the pool
        const bool dg = G == H;
        const int q4 = lane >> 2;
        unsigned mask[4];
        int pre[4], total = 0;
        double dsum = 0.0;
        bool zero = false;
#pragma unroll
        for (int a = 0; a < 4; ++a)
        {
            const int r = 8 * a + q4, i = G * GR + r;
            const bool live = dg && i < g.N && (GENERAL ? g.touched[i] : g.Xn[i]) > 0; // the diagonal is touched
            unsigned m = 0u;
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    const int c = 8 * b + 2 * (lane & 3) + h;
                    const T x = (T) acc[a][b][h];
                    bool keep = over<T>(x, g.thr);
                    if (dg)
                    {
                        keep = c == r ? live : keep && (GENERAL || c > r);
                        if (c == r && live)
                        {
                            dsum += (double) x;
                            zero |= acc[a][b][h] == 0.0;
                        }
                    }
                    m |= (keep ? 1u : 0u) << c;
                }
            m |= __shfl_xor_sync(FULL, m, 1);
            m |= __shfl_xor_sync(FULL, m, 2);
            mask[a] = m;
            const int cnt = __popc(m);
            int p = cnt;
#pragma unroll
            for (int o = 4; o < 32; o <<= 1)
            {
                const int u = __shfl_up_sync(FULL, p, o);
                if (lane >= o)
                    p += u;
            }
            pre[a] = total + p - cnt;
            total += __shfl_sync(FULL, p, 31);
        }
        if (dg)
        {
            for (int o = 16; o; o >>= 1)
                dsum += __shfl_xor_sync(FULL, dsum, o);
            if (lane == 0)
                g.dC[G] = dsum;
            // a row of stored zeros, or of entries that cancel: the tiles of a symmetric square do not tell whether
            // a product touches its diagonal
            if (!GENERAL && zero)
                atomicExch(&g.flags->odd, 1);
        }
        if (total == 0)
            continue;
        const unsigned long long need = 16 + ((unsigned long long) total * sizeof(T) + 7) / 8;
        unsigned long long at = 0;
        if (lane == 0)
            at = atomicAdd(&g.flags->pool, need);
        at = __shfl_sync(FULL, at, 0);
        if (at + need > g.cap)
        {
            if (lane == 0)
                atomicExch(&g.flags->full, 1);
            continue;
        }
        unsigned *head = reinterpret_cast<unsigned *>(g.pool + at);
        T *vals = reinterpret_cast<T *>(g.pool + at + 16);
#pragma unroll
        for (int a = 0; a < 4; ++a)
        {
            if ((lane & 3) == 0)
                head[8 * a + q4] = mask[a];
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    const int c = 8 * b + 2 * (lane & 3) + h;
                    if (mask[a] >> c & 1u)
                        vals[pre[a] + __popc(mask[a] & ((1u << c) - 1u))] = (T) acc[a][b][h];
                }
        }
        if (lane == 0)
            g.tab[(size_t) G * g.span + s] = (int) at;
    }
}

// Transpose of a 32 x 32 bit matrix, row `lane` in each lane.
__device__ __forceinline__ unsigned transpose_bits(unsigned x, int lane)
{
    unsigned m = 0x0000ffffu;
#pragma unroll
    for (int j = 16; j; j >>= 1)
    {
        const unsigned y = __shfl_xor_sync(FULL, x, j);
        x = (lane & j) ? ((x & ~m) | ((y & ~m) >> j)) : ((x & m) | ((y & m) << j));
        m ^= m << (j >> 1);
    }
    return x;
}

// Rows of C: one CTA per group.  Shared memory: the group's blocks in column
// order ({place, column group * 2 + transposed}), at most 2 span of them.
template <typename T> __global__ void __launch_bounds__(RT, sizeof(T) == 8 ? 1 : 2) tile_rows_kernel(TileArgs g)
{
    extern __shared__ int2 blk[];
    constexpr int W = RT / 32, RB = sizeof(T) == 8 ? 8 : 4;
    __shared__ int cnt[W][32];
    __shared__ int wtot[W];
    __shared__ int nblk;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (declined(g) || g.flags->full)
    {
        if (blockIdx.x == 0 && warp == 0)
            tell_host(g, lane);
        return;
    }
    for (int G = blockIdx.x; G < g.NG; G += gridDim.x)
    {
        // candidates in column order: (G - span + 1 + c, G) transposed for c < span, then (G, G + c - span)
        if (tid == 0)
            nblk = 0;
        __syncthreads();
        for (int c0 = 0; c0 < (g.general ? g.span : 2 * g.span); c0 += RT)
        {
            const int c = c0 + tid;
            int at = -1, key = 0;
            if (g.general)
            {
                const int H = G - g.back + c;
                if (c < g.span && H >= 0 && H < g.NG)
                    at = g.tab[(size_t) G * g.span + c];
                key = H * 2;
            }
            else if (c < g.span)
            {
                const int H = G - g.span + 1 + c;
                if (H >= 0)
                    at = g.tab[(size_t) H * g.span + (G - H)];
                key = H * 2 + 1;
            }
            else if (c < 2 * g.span)
            {
                const int H = G + c - g.span;
                if (H < g.NG)
                    at = g.tab[(size_t) G * g.span + (c - g.span)];
                key = H * 2;
            }
            const unsigned bal = __ballot_sync(FULL, at >= 0);
            if (lane == 0)
                wtot[warp] = __popc(bal);
            __syncthreads();
            int pos = nblk, all = 0;
            for (int v = 0; v < W; ++v)
            {
                pos += v < warp ? wtot[v] : 0;
                all += wtot[v];
            }
            if (at >= 0)
                blk[pos + __popc(bal & lanemask_lt())] = make_int2(at, key);
            __syncthreads();
            if (tid == 0)
                nblk += all;
            __syncthreads();
        }
        const int nb = nblk;
        const int per = (nb + W - 1) / W;
        const int b0 = min(nb, warp * per), b1 = min(nb, b0 + per);
        // the masks of output rows (lane = row), transposed blocks strictly below the diagonal
        auto masks = [&](int2 e, unsigned &own, unsigned &out) {
            own = __ldg(reinterpret_cast<const unsigned *>(g.pool + e.x) + lane);
            if (e.y & 1)
                out = transpose_bits((e.y >> 1) == G ? own & ~(1u << lane) : own, lane);
            else
                out = own;
        };
        int c = 0;
        for (int b = b0; b < b1; ++b)
        {
            unsigned own, out;
            masks(blk[b], own, out);
            c += __popc(out);
        }
        cnt[warp][lane] = c;
        __syncthreads();
        int off = 0, total = 0;
        for (int v = 0; v < W; ++v)
        {
            off += v < warp ? cnt[v][lane] : 0;
            total += cnt[v][lane];
        }
        const int i0 = G * GR;
        for (int b = b0; b < b1; ++b)
        {
            const int2 e = blk[b];
            unsigned own, out;
            masks(e, own, out);
            const T *vals = reinterpret_cast<const T *>(g.pool + e.x + 16);
            int p = __popc(own);
            for (int o = 1; o < 32; o <<= 1)
            {
                const int u = __shfl_up_sync(FULL, p, o);
                if (lane >= o)
                    p += u;
            }
            p -= __popc(own); // values before row `lane` of the block
            const bool tr = e.y & 1;
            const int k = (e.y >> 1) * GR + lane;
            // the loads of RB rows before their stores: a store between two loads orders them, and the walk was a
            // chain of 32 loads (27 us of a call on 512 rows, 17 us so; 75 us of the 2.31 ms of A*B on a 28^3
            // lattice).  FP32 with RB = 8 and one CTA per SM: 852 us against 819 for X^2 on 26999 rows; FP64 with
            // RB = 4 and two: 57 against 56 us on 512 rows.
            for (int r0 = 0; r0 < 32; r0 += RB)
            {
                T x[RB];
                int q[RB];
#pragma unroll
                for (int s = 0; s < RB; ++s)
                {
                    const int r = r0 + s;
                    const unsigned mr = __shfl_sync(FULL, out, r);
                    const int o = __shfl_sync(FULL, off, r), pr = __shfl_sync(FULL, p, r);
                    q[s] = mr >> lane & 1u ? o + __popc(mr & lanemask_lt()) : INT_MAX;
                    if (mr >> lane & 1u)
                        x[s] = tr ? vals[p + __popc(own & ((1u << r) - 1u))] : vals[pr + __popc(mr & lanemask_lt())];
                }
#pragma unroll
                for (int s = 0; s < RB; ++s)
                    if (q[s] < g.Mc)
                    {
                        static_cast<T *>(g.Cv)[(size_t) (i0 + r0 + s) * g.ldc + q[s]] = x[s];
                        g.Ci[(size_t) (i0 + r0 + s) * g.ldc + q[s]] = k;
                    }
            }
            off += __popc(out);
        }
        if (warp == 0)
        {
            const int i = i0 + lane;
            if (i < g.N)
                g.Cn[i] = min(total, g.Mc);
            int w = total;
            for (int o = 16; o; o >>= 1)
                w = max(w, __shfl_xor_sync(FULL, w, o));
            if (lane == 0)
            {
                if (w > *(volatile int *) &g.flags->max_width)
                    atomicMax(&g.flags->max_width, w);
                if (w > g.Mc)
                    atomicExch(&g.flags->overflow, 1);
            }
        }
        __syncthreads();
    }
    // the traces, summed over groups in a fixed order by the CTA that finishes last
    __shared__ double part[2][W];
    __shared__ int fin;
    if (tid == 0)
    {
        __threadfence(); // this CTA's width and overflow come before its count
        fin = atomicAdd(&g.flags->done, 1) == (int) gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!fin)
        return;
    double a = 0.0, d = 0.0;
    for (int G = tid; G < g.NG; G += RT)
    {
        a += g.dA[G];
        d += g.dC[G];
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
    if (tid == 0)
    {
        for (int v = 1; v < W; ++v)
        {
            a += part[0][v];
            d += part[1][v];
        }
        g.flags->trA = a;
        g.flags->trC = d;
        __threadfence();
    }
    if (warp == 0)
    {
        __syncwarp();
        tell_host(g, lane);
    }
}

// -------------------------------------------------------------------------
// Masked product C = A B at P's pattern: the second operand's tiles are those
// of its transpose, so a block is again a product of two group rows, and only
// the blocks that hold an entry of P are formed, whole, and read from.
// -------------------------------------------------------------------------

// Bitmaps of the transpose's groups from B's rows; one warp per row.
__global__ void __launch_bounds__(PT) tile_tbits_kernel(TileArgs g)
{
    const int lane = threadIdx.x & 31, warps = (gridDim.x * PT) >> 5;
    for (int j = (blockIdx.x * PT + threadIdx.x) >> 5; j < g.N; j += warps)
    {
        const int n = g.Xn[j];
        if (n < 0 || n > g.ld)
        {
            if (lane == 0)
                atomicExch(&g.flags->bad, 1);
            continue;
        }
        if (lane == 0 && n && !g.general)
            atomicAdd(&g.flags->products, (unsigned long long) n * n);
        const unsigned bit = 1u << ((j >> 3) & 31);
        int far = 0;
        for (int p = lane; p < n; p += 32)
        {
            const int k = g.Xi[(size_t) j * g.ld + p];
            if (k < 0 || k >= g.ncols)
            {
                atomicExch(&g.flags->bad, 1);
                continue;
            }
            far = max(far, abs(k - j));
            unsigned *w = g.gb + (size_t) (k >> 3) * g.nw + (j >> 8);
            if (!(*(volatile unsigned *) w & bit))
                atomicOr(w, bit);
        }
        for (int o = 16; o; o >>= 1)
            far = max(far, __shfl_xor_sync(FULL, far, o));
        if (lane == 0 && far > *(volatile int *) &g.flags->reachB)
            atomicMax(&g.flags->reachB, far);
    }
}

// Entries of the transpose's groups, and its share of the tile products.
__global__ void __launch_bounds__(PT) tile_tcount_kernel(TileArgs g)
{
    __shared__ int tot[5];
    __shared__ int fin;
    for (int G = blockIdx.x; G < g.NG; G += gridDim.x)
    {
        if (threadIdx.x < 5)
            tot[threadIdx.x] = 0;
        __syncthreads();
        int c[5] = {0, 0, 0, 0, 0};
        for (int w = threadIdx.x; w < g.nw; w += PT)
        {
            unsigned any = 0u;
#pragma unroll
            for (int a = 0; a < 4; ++a)
            {
                const unsigned b = g.gb[((size_t) G * 4 + a) * g.nw + w];
                c[a] += __popc(b);
                any |= b;
            }
            c[4] += __popc(any);
        }
#pragma unroll
        for (int a = 0; a < 5; ++a)
            if (c[a])
                atomicAdd(&tot[a], c[a]);
        __syncthreads();
        if (threadIdx.x == 0)
        {
            unsigned long long t2 = 0;
            for (int a = 0; a < 4; ++a)
                t2 += (unsigned long long) tot[a] * tot[a];
            if (!g.general)
                atomicAdd(&g.flags->tiles2, t2);
            atomicAdd(&g.flags->counted, tot[4]);
        }
        __syncthreads();
    }
    if (g.told && last_cta(g, &fin) && threadIdx.x < 32)
        tell_host(g, threadIdx.x);
}

// B's entries into the transpose's tiles; one warp per row of B.
template <typename T> __global__ void __launch_bounds__(PT) tile_scatter_kernel(TileArgs g)
{
    const int lane = threadIdx.x & 31, warps = (gridDim.x * PT) >> 5;
    for (int j = (blockIdx.x * PT + threadIdx.x) >> 5; j < g.N; j += warps)
    {
        const int n = g.Xn[j];
        const T *xv = static_cast<const T *>(g.Xv) + (size_t) j * g.ld;
        const int *xi = g.Xi + (size_t) j * g.ld;
        bool desc = false;
        for (int p = lane; p + 1 < n; p += 32)
            desc |= xi[p + 1] <= xi[p];
        const bool sorted = !__any_sync(FULL, desc);
        const int w = j >> 8;
        const unsigned below = (1u << ((j >> 3) & 31)) - 1u;
        bool odd = false;
        for (int p = lane; p < n; p += 32)
        {
            const int k = xi[p], G = k >> 5;
            const double v = (double) xv[p];
            odd |= !(fabs(v) <= 1.7976931348623157e308);
            const size_t at = (size_t) G * g.nw + w;
            const size_t t = 4 * (size_t) (g.eoff[G] + g.rank[at] + __popc(g.bits[at] & below)) + ((k >> 3) & 3);
            double *to = g.tiles + t * 64 + tile_at(k & 7, j & 7);
            if (sorted)
                *to = v;
            else
                atomicAdd(to, v);
        }
        if (__any_sync(FULL, odd) && lane == 0)
            atomicExch(&g.flags->odd, 1);
    }
}

// Groups H with an entry of P in the rows of G: counted (count_only), or
// listed with their ranks.  Shared memory: bitmap[hw].
__global__ void __launch_bounds__(FT) tile_pattern_kernel(TileArgs g)
{
    extern __shared__ unsigned pb[];
    __shared__ int sum, base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int G = blockIdx.x; G < g.NG; G += gridDim.x)
    {
        for (int w = tid; w < g.hw; w += FT)
            pb[w] = 0u;
        if (tid == 0)
            sum = 0;
        __syncthreads();
        for (int r = warp; r < GR; r += FT / 32)
        {
            const int i = G * GR + r;
            const int n = i < g.N ? g.Pn[i] : 0;
            if (n < 0 || n > g.ldp || n > g.Mc)
            {
                if (lane == 0)
                    atomicExch(&g.flags->bad, 1);
                continue;
            }
            for (int p = lane; p < n; p += 32)
            {
                const int k = g.Pi[(size_t) i * g.ldp + p];
                if (k < 0 || k >= g.ncols)
                    atomicExch(&g.flags->bad, 1);
                else if (!(*(volatile unsigned *) &pb[k >> 10] >> ((k >> 5) & 31) & 1u))
                    atomicOr(&pb[k >> 10], 1u << ((k >> 5) & 31));
            }
        }
        __syncthreads();
        int c = 0;
        for (int w = tid; w < g.hw; w += FT)
            c += __popc(pb[w]);
        if (c)
            atomicAdd(&sum, c);
        __syncthreads();
        if (tid == 0)
            base = atomicAdd(&g.flags->blocks, sum);
        __syncthreads();
        if (!g.count_only && warp == 0)
        {
            int at = base;
            for (int w0 = 0; w0 < g.hw; w0 += 32)
            {
                const int w = w0 + lane;
                unsigned b = w < g.hw ? pb[w] : 0u;
                const int n = __popc(b);
                int pre = n;
                for (int o = 1; o < 32; o <<= 1)
                {
                    const int u = __shfl_up_sync(FULL, pre, o);
                    if (lane >= o)
                        pre += u;
                }
                if (w < g.hw)
                {
                    g.pbits[(size_t) G * g.hw + w] = b;
                    g.prank[(size_t) G * g.hw + w] = at + pre - n;
                }
                for (int e = at + pre - n; b; b &= b - 1, ++e)
                    g.pblk[e] = make_int2(G, w * 32 + __ffs(b) - 1);
                at += __shfl_sync(FULL, pre, 31);
            }
        }
        __syncthreads();
    }
}

// Row i of C: P's columns with their sums; one warp per row.
template <typename T> __global__ void __launch_bounds__(PT) tile_gather_kernel(TileArgs g)
{
    const int lane = threadIdx.x & 31, warps = (gridDim.x * PT) >> 5;
    if (g.flags->odd)
        return;
    for (int i = (blockIdx.x * PT + threadIdx.x) >> 5; i < g.N; i += warps)
    {
        const int n = g.Pn[i], G = i >> 5;
        for (int p = lane; p < n; p += 32)
        {
            const int k = g.Pi[(size_t) i * g.ldp + p];
            const size_t w = (size_t) G * g.hw + (k >> 10);
            const int e = g.prank[w] + __popc(g.pbits[w] & ((1u << ((k >> 5) & 31)) - 1u));
            static_cast<T *>(g.Cv)[(size_t) i * g.ldc + p] = (T) g.out[(size_t) e * 1024 + (i & 31) * 32 + (k & 31)];
            g.Ci[(size_t) i * g.ldc + p] = k;
        }
        if (lane == 0)
            g.Cn[i] = n;
    }
}

// What the symmetry check has told of the counts at its start, if it does
// within the wait.
bool early_told(const TileArgs &g, TileOutcome *out)
{
    const volatile int4 *e = g.early;
    if (!b200_spin(&e->x, g.told))
        return false;
    const int p = e->y, t = e->z, w = e->w;
    float products, tiles2;
    memcpy(&products, &p, 4);
    memcpy(&tiles2, &t, 4);
    out->asym = w & 1;
    out->counted = true;
    out->counts = {(unsigned long long) products, (unsigned long long) (w >> 1), (unsigned long long) tiles2, 0, 0};
    return true;
}

// The fill kernel after a counting pass.
constexpr int FILL_WIDE = 300; // entries a row
template <typename T> void tile_fill(const TileArgs &g, int grid, size_t smem, cudaStream_t stream, double stored)
{
    if (sizeof(T) == 8 && stored >= (double) FILL_WIDE * g.N)
        tile_fill_kernel<T, false, 1><<<grid, FT, smem, stream>>>(g);
    else
        tile_fill_kernel<T, false, 2><<<grid, FT, smem, stream>>>(g);
}

template <typename T> bool tile_masked_typed(TileArgs a, TileArgs b, bool *taken)
{
    B200Context *c = b200_ctx();
    if (!c)
        return false;
    unsigned char *small = static_cast<unsigned char *>(c->d_small) + TL_SMALL;
    TileFlags *hf = reinterpret_cast<TileFlags *>(static_cast<unsigned char *>(c->pinned) + TL_SMALL);
    a.flags = b.flags = reinterpret_cast<TileFlags *>(small);
    const int NG = a.NG, nw = a.nw;
    const int per = std::min(NG, c->sm_count * 8);
    const size_t smemC = (size_t) 4 * nw * sizeof(unsigned), smemF = (size_t) 5 * nw * sizeof(unsigned);
    const size_t smemP = (size_t) a.hw * sizeof(unsigned);
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at = al(at + bytes);
        return o;
    };
    const size_t o_gb = take((size_t) NG * 4 * nw * sizeof(unsigned));
    const size_t o_bits = take((size_t) 2 * NG * nw * sizeof(unsigned));
    const size_t o_rank = take((size_t) 2 * NG * nw * sizeof(unsigned short));
    const size_t o_eoff = take((size_t) 2 * NG * sizeof(int)), o_range = take((size_t) 2 * NG * sizeof(int2));
    const size_t o_pb = take((size_t) NG * a.hw * sizeof(unsigned)), o_pr = take((size_t) NG * a.hw * sizeof(int));
    const size_t fixed = at;
    unsigned char *scr = nullptr;
    double stored = 0.0;
    // the counts, then the layout; a larger arena loses the transpose's bitmaps, which are then made again
    for (int attempt = 0; attempt < 2; ++attempt)
    {
        const bool grown = attempt && (size_t) at > c->scratch_bytes;
        if (attempt && !grown)
            break;
        scr = static_cast<unsigned char *>(b200_scratch_try(attempt ? at : fixed));
        if (!scr)
            return true; // the sparse form takes less
        b.gb = reinterpret_cast<unsigned *>(scr + o_gb);
        if (!CUDA_OK(cudaMemsetAsync(b.gb, 0, (size_t) NG * 4 * nw * sizeof(unsigned), c->stream)) ||
            !CUDA_OK(cudaMemsetAsync(small, 0, sizeof(TileFlags), c->stream)))
            return false;
        tile_tbits_kernel<<<std::min(b200_ceil_div(b.N, PT / 32), c->sm_count * 8), PT, 0, c->stream>>>(b);
        if (!LAUNCH_OK("tile_tbits_kernel"))
            return false;
        if (attempt)
            break;
        tile_tcount_kernel<<<per, PT, 0, c->stream>>>(b);
        if (!LAUNCH_OK("tile_tcount_kernel"))
            return false;
        tile_count_kernel<T><<<per, FT, smemC, c->stream>>>(a);
        if (!LAUNCH_OK("tile_count_kernel"))
            return false;
        a.count_only = 1;
        tile_pattern_kernel<<<per, FT, smemP, c->stream>>>(a);
        if (!LAUNCH_OK("tile_pattern_kernel") ||
            !CUDA_OK(cudaMemcpyAsync(hf, small, sizeof(TileFlags), cudaMemcpyDeviceToHost, c->stream)) || !b200_sync())
            return false;
        if (hf->counted >= (1 << 28) || left_to_sparse(*hf, a.cost))
            return true;
        stored = (double) hf->stored;
        take(0);
        const size_t o_ent = take((size_t) hf->counted * sizeof(unsigned));
        const size_t o_entJ = take((size_t) hf->counted * sizeof(unsigned short));
        const size_t o_tiles = take((size_t) hf->counted * 2048);
        const size_t o_blk = take((size_t) hf->blocks * sizeof(int2));
        const size_t o_out = take((size_t) hf->blocks * 8192);
        if (at > ((size_t) 64 << 30))
            return true;
        a.ent = reinterpret_cast<unsigned *>(o_ent); // offsets until the arena is settled
        a.entJ = reinterpret_cast<unsigned short *>(o_entJ);
        a.tiles = reinterpret_cast<double *>(o_tiles);
        a.pblk = reinterpret_cast<int2 *>(o_blk);
        a.out = reinterpret_cast<double *>(o_out);
    }
    auto place = [&](auto *&p) { p = reinterpret_cast<std::decay_t<decltype(p)>>(scr + reinterpret_cast<size_t>(p)); };
    place(a.ent);
    place(a.entJ);
    place(a.tiles);
    place(a.pblk);
    place(a.out);
    b.ent = a.ent;
    b.entJ = a.entJ;
    b.tiles = a.tiles;
    a.bits = reinterpret_cast<unsigned *>(scr + o_bits);
    a.rank = reinterpret_cast<unsigned short *>(scr + o_rank);
    a.eoff = reinterpret_cast<int *>(scr + o_eoff);
    a.range = reinterpret_cast<int2 *>(scr + o_range);
    a.bitsB = b.bits = a.bits + (size_t) NG * nw;
    a.rankB = b.rank = a.rank + (size_t) NG * nw;
    a.eoffB = b.eoff = a.eoff + NG;
    a.rangeB = b.range = a.range + NG;
    a.pbits = reinterpret_cast<unsigned *>(scr + o_pb);
    a.prank = reinterpret_cast<int *>(scr + o_pr);
    a.count_only = 0;
    if (!CUDA_OK(cudaMemsetAsync(small, 0, sizeof(TileFlags), c->stream)))
        return false;
    tile_fill<T>(a, per, smemF, c->stream, stored);
    if (!LAUNCH_OK("tile_fill_kernel"))
        return false;
    tile_fill<T>(b, per, smemF, c->stream, 0.0);
    if (!LAUNCH_OK("tile_fill_kernel"))
        return false;
    tile_scatter_kernel<T><<<std::min(b200_ceil_div(b.N, PT / 32), c->sm_count * 8), PT, 0, c->stream>>>(b);
    if (!LAUNCH_OK("tile_scatter_kernel"))
        return false;
    tile_pattern_kernel<<<per, FT, smemP, c->stream>>>(a);
    if (!LAUNCH_OK("tile_pattern_kernel"))
        return false;
    const size_t smemQ = (size_t) TW * WARP_SMEM;
    if (!CUDA_OK(cudaFuncSetAttribute(tile_x2_kernel<T, TILE_MASKED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int) smemQ)))
        return false;
    tile_x2_kernel<T, TILE_MASKED><<<c->sm_count * TMIN, TW * 32, smemQ, c->stream>>>(a);
    if (!LAUNCH_OK("tile_x2_kernel"))
        return false;
    tile_gather_kernel<T><<<std::min(b200_ceil_div(a.N, PT / 32), c->sm_count * 8), PT, 0, c->stream>>>(a);
    if (!LAUNCH_OK("tile_gather_kernel") ||
        !CUDA_OK(cudaMemcpyAsync(hf, small, sizeof(TileFlags), cudaMemcpyDeviceToHost, c->stream)) || !b200_sync())
        return false;
    *taken = !hf->odd && !hf->bad;
    return true;
}

// -------------------------------------------------------------------------
// General product: which columns a row touches.
// -------------------------------------------------------------------------

// Bitmaps over columns of B's rows (zero before); one warp per row.
__global__ void __launch_bounds__(PT) tile_rowbits_kernel(TileArgs g)
{
    const int lane = threadIdx.x & 31, warps = (gridDim.x * PT) >> 5;
    for (int j = (blockIdx.x * PT + threadIdx.x) >> 5; j < g.N; j += warps)
    {
        const int n = g.Xn[j];
        for (int p = lane; p < n; p += 32)
        {
            const int k = g.Xi[(size_t) j * g.ld + p];
            atomicOr(&g.rowbits[(size_t) j * g.rw + (k >> 5)], 1u << (k & 31));
        }
    }
}

// Row i of C touches the OR of the bitmaps of the rows of B that A's row i
// names: its width against M (check_pre), and whether it holds the diagonal.
// One warp per row, 128 words (16 bytes a lane) of the row's window (g.reach
// columns on each side) at a time.
__global__ void __launch_bounds__(PT) tile_touch_kernel(TileArgs g)
{
    const int lane = threadIdx.x & 31, warps = (gridDim.x * PT) >> 5;
    for (int i = (blockIdx.x * PT + threadIdx.x) >> 5; i < g.N; i += warps)
    {
        const int n = g.Xn[i];
        const int lo = max(0, i - g.reach) >> 7, hi = min(g.N - 1, i + g.reach) >> 7; // in words of 128 columns
        int width = 0;
        bool diag = false;
        for (int w0 = lo; w0 <= hi; w0 += 32)
        {
            const int w = w0 + lane;
            uint4 any = make_uint4(0u, 0u, 0u, 0u);
            for (int p0 = 0; p0 < n; p0 += 32)
            {
                const int mine = p0 + lane < n ? g.Xi[(size_t) i * g.ld + p0 + lane] : 0;
                const int m = min(32, n - p0);
#pragma unroll 8
                for (int t = 0; t < m; ++t)
                {
                    const int j = __shfl_sync(FULL, mine, t);
                    if (w <= hi)
                    {
                        const uint4 b = __ldg(reinterpret_cast<const uint4 *>(g.rowbits + (size_t) j * g.rw) + w);
                        any.x |= b.x;
                        any.y |= b.y;
                        any.z |= b.z;
                        any.w |= b.w;
                    }
                }
            }
            width += __popc(any.x) + __popc(any.y) + __popc(any.z) + __popc(any.w);
            const int q = (i >> 5) & 3;
            diag |= w == i >> 7 && ((q == 0 ? any.x : q == 1 ? any.y : q == 2 ? any.z : any.w) >> (i & 31) & 1u);
        }
        for (int o = 16; o; o >>= 1)
            width += __shfl_xor_sync(FULL, width, o);
        diag = __any_sync(FULL, diag);
        if (lane == 0)
        {
            g.touched[i] = diag;
            if (g.check_pre && width > g.Mc)
                atomicExch(&g.flags->overflow, 1);
        }
    }
}

// Rows below which the row lengths are asked in the sparse form's flight, from
// there to 9000 ahead of the counts.  Most products of fewer rows stay on the
// sparse form, which then pays 3 us; most of more rows take tiles, which would
// pay 10 to 17 us for the flight stopped and pay 3 so (18^3 lattices of radii 3
// and 2.5 316 and 306; of 2 and 2.5, which stay, 220 and 227, 240 with the counts
// alone, 217 with nothing asked).
constexpr int FEW_ROWS = 4096;

// Whether the counts can say so at all, by the room of the rows.
bool general_may_pay(const bml_matrix_ellpack_t *A, const bml_matrix_ellpack_t *B, double cost)
{
    const double stored = (double) A->N * A->ld;
    return general_pays(A->N, stored, stored * B->ld, 0.0, cost);
}

template <typename T>
bool tile_general_typed(TileArgs a, TileArgs b, const TileCounts *known, double *trace, int *required_M, bool *taken,
                        cudaEvent_t *timer)
{
    B200Context *c = b200_ctx();
    if (!c)
        return false;
    unsigned char *small = static_cast<unsigned char *>(c->d_small) + TL_SMALL;
    TileFlags *hf = reinterpret_cast<TileFlags *>(static_cast<unsigned char *>(c->pinned) + TL_SMALL);
    a.flags = b.flags = reinterpret_cast<TileFlags *>(small);
    a.host = b.host = hf;
    const int NG = a.NG, nw = a.nw;
    const int per = std::min(NG, c->sm_count * 8);
    const int rows = std::min(b200_ceil_div(a.N, PT / 32), c->sm_count * 8);
    const size_t smemC = (size_t) 4 * nw * sizeof(unsigned), smemF = (size_t) 5 * nw * sizeof(unsigned);
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at = al(at + bytes);
        return o;
    };
    const size_t n_gb = (size_t) NG * 4 * nw * sizeof(unsigned), n_rb = (size_t) b.N * b.rw * sizeof(unsigned);
    const size_t o_gb = take(n_gb), o_rb = take(n_rb);
    const size_t o_bits = take((size_t) 2 * NG * nw * sizeof(unsigned));
    const size_t o_rank = take((size_t) 2 * NG * nw * sizeof(unsigned short));
    const size_t o_eoff = take((size_t) 2 * NG * sizeof(int)), o_range = take((size_t) 2 * NG * sizeof(int2));
    const size_t o_touched = take((size_t) a.N * sizeof(int)), o_diag = take((size_t) 2 * NG * sizeof(double));
    const size_t o_tileN = take((size_t) 8 * NG * sizeof(int));
    const size_t fixed = at;
    size_t o_ent = 0, o_entJ = 0, o_tiles = 0, o_tab = 0, o_pool = 0;
    unsigned char *scr = static_cast<unsigned char *>(b200_scratch_try(fixed));
    if (!scr)
        return true; // the sparse form takes less
    // the products of both forms, unless X^2's symmetric attempt has counted them
    TileCounts n{};
    if (known)
        n = *known;
    else
    {
        a.told = b200_next_told();
        if (!CUDA_OK(cudaMemsetAsync(small, 0, sizeof(TileFlags), c->stream)))
            return false;
        if (a.Xi == b.Xi)
            tile_count_kernel<T><<<per, FT, smemC, c->stream>>>(a);
        else
        {
            TileArgs rows_b = b;
            a.nB = b.Xn;
            a.tileN = reinterpret_cast<int *>(scr + o_tileN);
            a.tileC = a.tileN + 4 * NG;
            if (!CUDA_OK(cudaMemsetAsync(a.tileC, 0, (size_t) 4 * NG * sizeof(int), c->stream)))
                return false;
            const int told = b200_next_told();
            // (of fewer rows they were asked before the call came here)
            const bool lengths = a.N >= FEW_ROWS && !general_pays(a.N, 0.0, 0.0, 0.0, a.cost);
            if (lengths)
            {
                a.early = reinterpret_cast<int4 *>(reinterpret_cast<unsigned char *>(hf) + EARLY);
                tile_lengths_kernel<<<1, 1024, 0, c->stream>>>(a, b, told);
                if (!LAUNCH_OK("tile_lengths_kernel"))
                    return false;
            }
            tile_cross_kernel<<<std::min(2 * NG, c->sm_count * 8), FT, smemC, c->stream>>>(a, rows_b);
            if (lengths)
            {
                const volatile int4 *e = a.early;
                if (!LAUNCH_OK("tile_cross_kernel") || !b200_told(&e->x, told))
                    return false;
                if (!e->y)
                    return true;
                a.early = nullptr;
            }
        }
        if (!LAUNCH_OK("tile counts") || !b200_told(reinterpret_cast<const int *>(hf) + TOLD, a.told))
            return false;
        a.told = 0;
        if (hf->bad)
            return true;
        n = {hf->products, hf->stored, hf->tiles2, hf->counted, hf->reach};
    }
    if (n.entries <= 0 || !general_pays(a.N, (double) n.stored, (double) n.products, (double) n.tiles2, a.cost))
        return true;
    int reach = 0;
    // the second operand's entries, then the layout; a larger arena loses B's bitmaps, which are then made again
    for (int attempt = 0; attempt < 2; ++attempt)
    {
        if (attempt && at <= c->scratch_bytes)
        {
            if (!CUDA_OK(cudaMemsetAsync(b.rowbits, 0, n_rb, c->stream)))
                return false;
            break;
        }
        scr = static_cast<unsigned char *>(b200_scratch_try(attempt ? at : fixed));
        if (!scr)
            return true; // the sparse form takes less
        b.gb = reinterpret_cast<unsigned *>(scr + o_gb);
        b.rowbits = reinterpret_cast<unsigned *>(scr + o_rb);
        if (!CUDA_OK(cudaMemsetAsync(small, 0, sizeof(TileFlags), c->stream)) ||
            !CUDA_OK(cudaMemsetAsync(b.gb, 0, n_gb, c->stream)) ||
            (attempt && !CUDA_OK(cudaMemsetAsync(b.rowbits, 0, n_rb, c->stream))))
            return false;
        tile_tbits_kernel<<<rows, PT, 0, c->stream>>>(b);
        if (!LAUNCH_OK("tile_tbits_kernel"))
            return false;
        if (attempt)
            break;
        b.told = b200_next_told();
        tile_tcount_kernel<<<per, PT, 0, c->stream>>>(b);
        if (!LAUNCH_OK("tile_tcount_kernel") || !b200_told(reinterpret_cast<const int *>(hf) + TOLD, b.told))
            return false;
        b.told = 0;
        const long long entries = (long long) n.entries + hf->counted;
        if (hf->bad || hf->counted <= 0 || entries >= (1 << 28))
            return true;
        reach = std::min(a.N, n.reach + hf->reachB);
        a.back = std::min(NG - 1, reach / GR + 1);
        a.span = 2 * a.back + 1;
        const size_t words = (size_t) a.N * a.Mc * sizeof(T) / 8 + 1 + (size_t) 17 * NG * a.span;
        if ((size_t) a.span * sizeof(int2) > c->smem_optin - 8192 || words >= ((size_t) 1 << 31) ||
            (long long) ((NG + SG - 1) / SG * SG) * ((a.span + SC - 1) / SC * SC) >= 1 << 30)
            return true;
        o_ent = take((size_t) entries * sizeof(unsigned));
        o_entJ = take((size_t) entries * sizeof(unsigned short));
        o_tiles = take((size_t) entries * 2048);
        o_tab = take((size_t) NG * a.span * sizeof(int));
        o_pool = take(words * 8);
        a.cap = words;
        if (at > ((size_t) 64 << 30))
            return true;
    }
    a.ent = b.ent = reinterpret_cast<unsigned *>(scr + o_ent);
    a.entJ = b.entJ = reinterpret_cast<unsigned short *>(scr + o_entJ);
    a.tiles = b.tiles = reinterpret_cast<double *>(scr + o_tiles);
    a.bits = reinterpret_cast<unsigned *>(scr + o_bits);
    a.rank = reinterpret_cast<unsigned short *>(scr + o_rank);
    a.eoff = reinterpret_cast<int *>(scr + o_eoff);
    a.range = reinterpret_cast<int2 *>(scr + o_range);
    a.bitsB = b.bits = a.bits + (size_t) NG * nw;
    a.rankB = b.rank = a.rank + (size_t) NG * nw;
    a.eoffB = b.eoff = a.eoff + NG;
    a.rangeB = b.range = a.range + NG;
    a.touched = reinterpret_cast<int *>(scr + o_touched);
    a.dA = reinterpret_cast<double *>(scr + o_diag);
    a.dC = a.dA + NG;
    a.tab = reinterpret_cast<int *>(scr + o_tab);
    a.pool = reinterpret_cast<unsigned long long *>(scr + o_pool);
    a.rowbits = b.rowbits;
    a.reach = reach;
    if (!CUDA_OK(cudaMemsetAsync(small, 0, sizeof(TileFlags), c->stream)))
        return false;
    tile_rowbits_kernel<<<rows, PT, 0, c->stream>>>(b);
    if (!LAUNCH_OK("tile_rowbits_kernel"))
        return false;
    tile_touch_kernel<<<rows, PT, 0, c->stream>>>(a);
    if (!LAUNCH_OK("tile_touch_kernel"))
        return false;
    tile_fill<T>(a, per, smemF, c->stream, (double) n.stored);
    if (!LAUNCH_OK("tile_fill_kernel"))
        return false;
    tile_fill<T>(b, per, smemF, c->stream, 0.0);
    if (!LAUNCH_OK("tile_fill_kernel"))
        return false;
    tile_scatter_kernel<T><<<rows, PT, 0, c->stream>>>(b);
    if (!LAUNCH_OK("tile_scatter_kernel"))
        return false;
    const size_t smemQ = (size_t) TW * WARP_SMEM;
    const size_t smemR = (size_t) a.span * sizeof(int2);
    if (!CUDA_OK(cudaFuncSetAttribute(tile_x2_kernel<T, TILE_GENERAL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int) smemQ)) ||
        (smemR > 32768 && !CUDA_OK(cudaFuncSetAttribute(
                              tile_rows_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smemR))) ||
        (timer && !CUDA_OK(cudaEventRecord(timer[0], c->stream))))
        return false;
    tile_x2_kernel<T, TILE_GENERAL><<<c->sm_count * TMIN, TW * 32, smemQ, c->stream>>>(a);
    if (!LAUNCH_OK("tile_x2_kernel"))
        return false;
    if (timer && !CUDA_OK(cudaEventRecord(timer[1], c->stream)))
        return false;
    a.told = b200_next_told();
    tile_rows_kernel<T><<<NG, RT, smemR, c->stream>>>(a);
    if (!LAUNCH_OK("tile_rows_kernel") || !b200_told(reinterpret_cast<const int *>(hf) + TOLD, a.told))
        return false;
    if (hf->bad || hf->odd || hf->full)
        return true;
    *taken = true;
    if (required_M)
        *required_M = hf->max_width;
    if (trace)
    {
        trace[0] = hf->trA;
        trace[1] = hf->trC;
    }
    if (hf->overflow)
    {
        b200_set_error(BML_B200_ERR_ROW_OVERFLOW, "Number of non-zeroes per row > M, Increase M (need %d, M = %d)",
                       hf->max_width, a.Mc);
        return false;
    }
    return true;
}

template <typename T>
bool tile_x2_typed(TileArgs g, double *trace, int *required_M, TileOutcome *out, cudaEvent_t *timer,
                   bool pack_all = false)
{
    B200Context *c = b200_ctx();
    if (!c)
        return false;
    unsigned char *small = static_cast<unsigned char *>(c->d_small) + TL_SMALL;
    TileFlags *hf = reinterpret_cast<TileFlags *>(static_cast<unsigned char *>(c->pinned) + TL_SMALL);
    g.flags = reinterpret_cast<TileFlags *>(small);
    g.host = hf;
    const int per = (int) std::min<long long>(g.NG, (long long) c->sm_count * 8);
    const size_t smemC = (size_t) 4 * g.nw * sizeof(unsigned);
    const size_t smemF = (size_t) 5 * g.nw * sizeof(unsigned); // at most 40 KB
    if (!CUDA_OK(cudaMemsetAsync(small, 0, sizeof(TileFlags), c->stream)))
        return false;
    // Small matrices are laid out for the most tiles they can have, which saves the counting pass and its round trip;
    // the fill kernel then counts, and the later kernels find the form declined.  (LAZY_BYTES admits 4096 rows: X^2 of
    // rows of 33 and of 341 takes 71 and 138 us there, 76 and 151 at 4097, with the counting pass.)
    const long long nbk = b200_ceil_div(g.N, 8);
    long long entries = std::min((long long) g.NG * nbk, (long long) g.N * g.ld);
    int span = g.NG;
    const bool lazy = entries * 2048 <= LAZY_BYTES;
    auto note = [&]() {
        out->asym = hf->asym || hf->alone;
        out->counted = out->complete = !hf->bad;
        out->counts = {hf->products, hf->stored, hf->tiles2, hf->counted, hf->reach};
    };
    g.sample = pack_all ? 0 : 1;
    if (!lazy)
    {
        g.told = b200_next_told();
        tile_count_kernel<T><<<per, FT, smemC, c->stream>>>(g);
        if (!LAUNCH_OK("tile_count_kernel") || !b200_told(reinterpret_cast<const int *>(hf) + TOLD, g.told))
            return false;
        g.told = 0;
        note();
        if (hf->counted <= 0 || hf->counted >= (1 << 28) || left_to_sparse(*hf, g.cost))
            return true;
        entries = hf->counted;
        span = std::min(g.NG, 2 * (hf->reach / GR + 1) + 1);
    }
    const size_t smemR = (size_t) 2 * span * sizeof(int2);
    if (smemR > c->smem_optin - 8192)
        return true;
    // pool: the kept entries of the upper triangle when no row is wider than M, and a header per block
    const size_t vals = ((size_t) g.N * ((size_t) g.Mc + 1) / 2 + 1) * sizeof(T) / 8 + 1;
    const size_t words = vals + (size_t) 17 * g.NG * span;
    if (words >= ((size_t) 1 << 31))
        return true;
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at = al(at + bytes);
        return o;
    };
    const size_t o_bits = take((size_t) g.NG * g.nw * sizeof(unsigned));
    const size_t o_rank = take((size_t) g.NG * g.nw * sizeof(unsigned short));
    const size_t o_eoff = take((size_t) g.NG * sizeof(int));
    const size_t o_range = take((size_t) g.NG * sizeof(int2));
    const size_t o_last = take((size_t) g.NG * sizeof(int));
    const size_t o_ent = take((size_t) entries * sizeof(unsigned));
    const size_t o_entJ = take((size_t) entries * sizeof(unsigned short));
    const size_t o_diag = take((size_t) 2 * g.NG * sizeof(double));
    const size_t o_tab = take((size_t) g.NG * span * sizeof(int));
    const size_t o_tiles = take((size_t) entries * 256 * sizeof(double));
    const size_t o_pool = take(words * 8);
    if (at > ((size_t) 64 << 30))
        return true;
    unsigned char *scr = static_cast<unsigned char *>(b200_scratch_try(at));
    if (!scr)
        return true; // the sparse form takes less
    g.bits = reinterpret_cast<unsigned *>(scr + o_bits);
    g.rank = reinterpret_cast<unsigned short *>(scr + o_rank);
    g.eoff = reinterpret_cast<int *>(scr + o_eoff);
    g.range = reinterpret_cast<int2 *>(scr + o_range);
    g.last = reinterpret_cast<int *>(scr + o_last);
    g.ent = reinterpret_cast<unsigned *>(scr + o_ent);
    g.entJ = reinterpret_cast<unsigned short *>(scr + o_entJ);
    g.dA = reinterpret_cast<double *>(scr + o_diag);
    g.dC = g.dA + g.NG;
    g.tab = reinterpret_cast<int *>(scr + o_tab);
    g.span = span;
    g.tiles = reinterpret_cast<double *>(scr + o_tiles);
    g.pool = reinterpret_cast<unsigned long long *>(scr + o_pool);
    g.cap = words;
    g.bitsB = g.bits;
    g.rankB = g.rank;
    g.eoffB = g.eoff;
    g.rangeB = g.range;
    const long long items =
        (long long) ((g.NG + SG - 1) / SG * SG) * ((span + SC - 1) / SC * SC); // counted in an int by the kernel
    if (items >= 1 << 30)
        return true;
    const size_t smemQ = (size_t) TW * WARP_SMEM;
    if (!CUDA_OK(cudaFuncSetAttribute(tile_x2_kernel<T, TILE_SQUARE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int) smemQ)) ||
        (smemR > 32768 && !CUDA_OK(cudaFuncSetAttribute(tile_rows_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        (int) smemR))))
        return false;
    if (!lazy)
        tile_fill<T>(g, per, smemF, c->stream, (double) out->counts.stored);
    else
    {
        g.told = b200_next_told();
        g.early = reinterpret_cast<int4 *>(reinterpret_cast<unsigned char *>(hf) + EARLY);
        tile_fill_kernel<T, true, 1><<<per, FT, smemF, c->stream>>>(g);
    }
    if (!LAUNCH_OK("tile_fill_kernel"))
        return false;
    tile_sym_kernel<<<per, PT, 0, c->stream>>>(g);
    if (!LAUNCH_OK("tile_sym_kernel"))
        return false;
    // what follows is queued while the check runs, or left out; if the word does not come, the flags will tell
    if (lazy && early_told(g, out) && (out->asym || (double) out->counts.tiles2 * g.cost > (double) out->counts.products))
        return true;
    if (timer && !CUDA_OK(cudaEventRecord(timer[0], c->stream)))
        return false;
    const int grid = (int) std::min<long long>((items + TW - 1) / TW, (long long) c->sm_count * TMIN);
    tile_x2_kernel<T, TILE_SQUARE><<<grid, TW * 32, smemQ, c->stream>>>(g);
    if (!LAUNCH_OK("tile_x2_kernel"))
        return false;
    if (timer && !CUDA_OK(cudaEventRecord(timer[1], c->stream)))
        return false;
    g.told = b200_next_told();
    tile_rows_kernel<T><<<g.NG, RT, smemR, c->stream>>>(g);
    if (!LAUNCH_OK("tile_rows_kernel") || !b200_told(reinterpret_cast<const int *>(hf) + TOLD, g.told))
        return false;
    note();
    if (hf->skipped && !hf->odd && !out->asym && !left_to_sparse(*hf, g.cost))
        return tile_x2_typed<T>(g, trace, required_M, out, timer, true);
    if (hf->bad || hf->odd || hf->skipped || out->asym || hf->full || left_to_sparse(*hf, g.cost))
        return true;
    out->taken = true;
    if (required_M)
        *required_M = hf->max_width;
    if (trace)
    {
        trace[0] = hf->trA;
        trace[1] = hf->trC;
    }
    if (hf->overflow)
    {
        b200_set_error(BML_B200_ERR_ROW_OVERFLOW, "Number of non-zeroes per row > M, Increase M (need %d, M = %d)",
                       hf->max_width, g.Mc);
        return false;
    }
    return true;
}

} // namespace

bool ell_x2_tiles(bml_matrix_ellpack_t *X, bml_matrix_ellpack_t *C, double threshold, double *trace, int *required_M,
                  TileOutcome *out, cudaEvent_t *timer)
{
    *out = TileOutcome{};
    // a place in a group's list is kept in 16 bits
    const int nbk = b200_ceil_div(X->N, 8);
    if (!g_tiles || !(threshold >= 0.0) || X->N != C->N || X->N < 1 || nbk > 65535)
        return true;
    TileArgs g{};
    g.cost = g_tiles == 1 ? TILE_COST : 0.0;
    g.Xv = X->d_value;
    g.Xi = X->d_index;
    g.Xn = X->d_nnz;
    g.ld = X->ld;
    g.N = X->N;
    g.ncols = X->N;
    g.NG = b200_ceil_div(X->N, GR);
    g.nw = b200_ceil_div(nbk, 32);
    g.Cv = C->d_value;
    g.Ci = C->d_index;
    g.Cn = C->d_nnz;
    g.ldc = C->ld;
    g.Mc = C->M;
    g.thr = threshold;
    return X->matrix_precision == double_real ? tile_x2_typed<double>(g, trace, required_M, out, timer)
                                              : tile_x2_typed<float>(g, trace, required_M, out, timer);
}

bool ell_masked_tiles(bml_matrix_ellpack_t *A, bml_matrix_ellpack_t *B, bml_matrix_ellpack_t *P,
                      bml_matrix_ellpack_t *C, bool *taken)
{
    *taken = false;
    const int nbk = b200_ceil_div(A->N, 8);
    if (!g_tiles || A->N != B->N || A->N != C->N || nbk > 65535)
        return true;
    TileArgs a{};
    a.cost = g_tiles == 1 ? TILE_COST : 0.0;
    a.N = a.ncols = A->N;
    a.NG = b200_ceil_div(A->N, GR);
    a.nw = b200_ceil_div(nbk, 32);
    a.masked = 1;
    TileArgs b = a;
    a.Xv = A->d_value;
    a.Xi = A->d_index;
    a.Xn = A->d_nnz;
    a.ld = A->ld;
    b.Xv = B->d_value;
    b.Xi = B->d_index;
    b.Xn = B->d_nnz;
    b.ld = B->ld;
    a.Pi = P->d_index;
    a.Pn = P->d_nnz;
    a.ldp = P->ld;
    a.hw = b200_ceil_div(a.NG, 32);
    a.Cv = C->d_value;
    a.Ci = C->d_index;
    a.Cn = C->d_nnz;
    a.ldc = C->ld;
    a.Mc = C->M;
    return A->matrix_precision == double_real ? tile_masked_typed<double>(a, b, taken)
                                              : tile_masked_typed<float>(a, b, taken);
}

bool ell_general_tiles_by_rows(const bml_matrix_ellpack_t *A, const bml_matrix_ellpack_t *B,
                               const bml_matrix_ellpack_t *C, double threshold)
{
    return g_tiles == 1 && threshold >= 0.0 && A->N < FEW_ROWS && A->N == B->N && A->N == C->N &&
           general_may_pay(A, B, TILE_COST);
}

bool ell_general_tiles(bml_matrix_ellpack_t *A, bml_matrix_ellpack_t *B, bml_matrix_ellpack_t *C, double threshold,
                       const TileOutcome *known, double *trace, int *required_M, bool check_pre, bool *taken,
                       cudaEvent_t *timer)
{
    *taken = false;
    const int nbk = b200_ceil_div(A->N, 8);
    if (!g_tiles || !(threshold >= 0.0) || A->N != B->N || A->N != C->N || nbk > 65535)
        return true;
    TileArgs a{};
    a.cost = g_tiles == 1 ? TILE_COST : 0.0;
    if (known ? !general_pays(A->N, (double) known->counts.stored, (double) known->counts.products,
                              (double) known->counts.tiles2, a.cost)
              : !general_may_pay(A, B, a.cost))
        return true;
    const TileCounts *counts = known && known->complete ? &known->counts : nullptr;
    a.N = a.ncols = A->N;
    a.NG = b200_ceil_div(A->N, GR);
    a.nw = b200_ceil_div(nbk, 32);
    a.rw = b200_ceil_div(A->N, 128) * 4; // rows of 16-byte words
    if ((size_t) a.N * a.rw * sizeof(unsigned) > ((size_t) 2 << 30)) // bitmaps of B's rows: N up to 131072
        return true;
    a.general = 1;
    a.thr = threshold;
    TileArgs b = a;
    b.masked = 1;
    a.Xv = A->d_value;
    a.Xi = A->d_index;
    a.Xn = A->d_nnz;
    a.ld = A->ld;
    b.Xv = B->d_value;
    b.Xi = B->d_index;
    b.Xn = B->d_nnz;
    b.ld = B->ld;
    a.Cv = C->d_value;
    a.Ci = C->d_index;
    a.Cn = C->d_nnz;
    a.ldc = C->ld;
    a.Mc = C->M;
    a.check_pre = check_pre ? 1 : 0;
    return A->matrix_precision == double_real ? tile_general_typed<double>(a, b, counts, trace, required_M, taken, timer)
                                              : tile_general_typed<float>(a, b, counts, trace, required_M, taken, timer);
}

extern "C" BML_B200_API int bml_b200_set_tiles(int mode)
{
    const int old = g_tiles;
    g_tiles = mode < 0 ? 0 : mode > 2 ? 2 : mode;
    return old;
}
