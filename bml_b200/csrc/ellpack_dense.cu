// Dense tier of the unordered ELLPACK product C = A*B, for operands whose
// rows are a large share of N wide (the SP2 iterates of a metallic
// Hamiltonian fill in to dense rows within a few iterations).
//
// Same result set as the sparse products (ellpack/bml_multiply_ellpack_typed.c:
// 252-333 for X^2, :468-542 for A*B): A and B are scattered into zero-filled
// dense images, C = A B is formed by a register-tiled GEMM (each product a
// single rounded multiply-add; the products of one entry are summed in no
// fixed order, within the same bound as the unordered sparse kernel), and a
// compaction kernel applies the reference's keep rule row by row, in
// ascending column order: the diagonal when it is touched, another column
// when |c| > threshold (compared in the matrix precision).  A column that no
// structural product touches holds an exact zero in the image and is
// dropped by the rule, as the sparse kernels drop it, so only the diagonal
// needs the structure: it is touched when some j has A[i,j] and B[j,i]
// stored, found through a byte image of B's pattern (in a symmetric square
// through the image itself).  The traces are those of the sparse kernels: tr A
// from A's diagonal entries, tr C from the pre-threshold diagonal where touched.
//
// Symmetric squares (the image equal to its transpose) form the tiles on and
// above the diagonal only.  X^2 of 5001 full rows in FP64: 13.93 ms on the FMA
// pipe, as the FP32 GEMM below, with both triangles, 5.01 ms so.
//
// The FP32 GEMM: 128 x 128 tiles of C per CTA of 256 threads, each thread 8 x 8
// outputs (rows ty + 16 m, columns tx + 16 n) in registers; K in steps of 16
// staged through shared memory, the next step's operands loaded into
// registers while the current one is multiplied.  A's tile is stored
// transposed (k-major), so every inner step reads 8 values of A (two
// addresses per warp, broadcast) and 8 of B (16 consecutive per half warp).
// The images are padded to multiples of 128 with zeros, so the kernel has no
// edge cases.
#include "device_util.cuh"

#include <cstring>
#include <type_traits>

using namespace b200;

namespace {

constexpr int DT = 128;   // tile edge of C
constexpr int DK = 16;    // k step
constexpr int DTHREADS = 256;

struct DenseFlags
{
    int overflow;
    int max_width;
    int bad_input;
    int asym; // X^2: the image differs from its transpose
};

// image[i * ld + col] += value for every stored entry (duplicates add up, as
// they do in the sparse products; a strictly ascending row has none and is
// stored); rows padded with zeros.  One warp per row.
template <typename T>
__global__ void __launch_bounds__(256) dense_scatter_kernel(const T *v, const int *ix, const int *nz, int ldE, int nrows,
                                                            int ncols, T *img, size_t ld, DenseFlags *flags)
{
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nrows; i += warps)
    {
        const int n = nz[i];
        if (n < 0 || n > ldE)
        {
            if (lane == 0)
                atomicExch(&flags->bad_input, 1);
            continue;
        }
        bool desc = false;
#pragma unroll 4
        for (int p = lane; p + 1 < n; p += 32)
            desc |= ix[(size_t) i * ldE + p + 1] <= ix[(size_t) i * ldE + p];
        const bool sorted = !__any_sync(FULL, desc);
        for (int p = lane; p < n; p += 32)
        {
            const int c = ix[(size_t) i * ldE + p];
            if (c < 0 || c >= ncols)
            {
                atomicExch(&flags->bad_input, 1);
                continue;
            }
            if (sorted)
                img[(size_t) i * ld + c] = v[(size_t) i * ldE + p];
            else
                atomicAdd(&img[(size_t) i * ld + c], v[(size_t) i * ldE + p]);
        }
    }
}

// Pattern of B, transposed: pat[col * ld + row] = 1 for every stored entry.  One
// warp per row; nothing to do for a symmetric square (*asym == 0).  The bytes
// are a column apart: 0.2 ms of the 0.3 ms that the scatter took for 5001 full
// rows.
__global__ void __launch_bounds__(256) dense_pattern_kernel(const int *ix, const int *nz, int ldE, int nrows, int ncols,
                                                            unsigned char *pat, size_t ld, const int *asym)
{
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    if (asym && *asym == 0)
        return;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nrows; i += warps)
    {
        const int n = nz[i];
        if (n < 0 || n > ldE)
            continue;
        for (int p = lane; p < n; p += 32)
        {
            const int c = ix[(size_t) i * ldE + p];
            if (c >= 0 && c < ncols)
                pat[(size_t) c * ld + i] = 1;
        }
    }
}

// touched[i] = 1 when some stored A[i,j] meets a stored B[j,i]; dA[i] = sum of
// A's diagonal entries.  One warp per row of A.  In a symmetric square
// (*asym == 0) an entry of the image that is not zero has its mirror (a stored
// one may not: entries of one column add up, perhaps to zero); a row of zeros
// looks for one in the rows that it names.
template <typename T>
__global__ void __launch_bounds__(256) dense_diag_kernel(const T *v, const int *ix, const int *nz, int ldE, int nrows,
                                                         int ncols, const unsigned char *patBt, size_t ld,
                                                         const T *img, const int *asym, int *touched, double *dA)
{
    const bool sym = asym && *asym == 0;
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nrows; i += warps)
    {
        const int n = nz[i];
        int hit = 0;
        double d = 0.0;
        if (n >= 0 && n <= ldE)
        {
#pragma unroll 4
            for (int p = lane; p < n; p += 32)
                if (ix[(size_t) i * ldE + p] == i)
                    d += (double) v[(size_t) i * ldE + p];
            for (int p0 = 0; p0 < n && !__any_sync(FULL, hit); p0 += 32)
            {
                const int j = p0 + lane < n ? ix[(size_t) i * ldE + p0 + lane] : -1;
                // B[j,i] stored <=> patBt[i * ld + j]
                if (j >= 0 && j < ncols)
                    hit = sym ? img[(size_t) i * ld + j] != T(0) : i < ncols && patBt[(size_t) i * ld + j];
            }
        }
        if (sym && n > 0 && n <= ldE && !__any_sync(FULL, hit))
            for (int p = 0; p < n; ++p)
            {
                const int j = ix[(size_t) i * ldE + p];
                if (j < 0 || j >= nrows)
                    continue;
                const int m = nz[j];
                for (int q = lane; q < m && m <= ldE; q += 32)
                    if (ix[(size_t) j * ldE + q] == i)
                        hit = 1;
            }
        hit = __any_sync(FULL, hit);
        for (int o = 16; o; o >>= 1)
            d += __shfl_xor_sync(FULL, d, o);
        if (lane == 0)
        {
            touched[i] = hit;
            if (dA)
                dA[i] = d;
        }
    }
}

// C[Mp x Np] = A[Mp x Kp] B[Kp x Np], all row-major with leading dimension ld,
// every dimension a multiple of 128.  Dynamic shared memory: two stages of
// A^T (16 x 128) and B (16 x 128).
__global__ void __launch_bounds__(DTHREADS, 1) dense_gemm_kernel(const float *__restrict__ A, const float *__restrict__ B,
                                                                 float *__restrict__ Cm, size_t ld, int Kp,
                                                                 const int *asym)
{
    const bool sym = asym && *asym == 0;
    if (sym && blockIdx.x < blockIdx.y)
        return;
    extern __shared__ __align__(16) unsigned char dsm[];
    float(*As)[DK][DT] = reinterpret_cast<float(*)[DK][DT]>(dsm);
    float(*Bs)[DK][DT] = reinterpret_cast<float(*)[DK][DT]>(dsm + 2 * sizeof(float) * DK * DT);
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const size_t i0 = (size_t) blockIdx.y * DT, j0 = (size_t) blockIdx.x * DT;
    // loads: A tile 128 rows x 16 k, thread t takes row t >> 1 and the 8 k
    // from (t & 1) * 8; B tile 16 rows x 128, thread t takes row t >> 4 and
    // columns (t & 15) + 16 q, q < 8 (a half warp reads 16 consecutive)
    const int ar = tid >> 1, ak = (tid & 1) * 8;
    const int br = tid >> 4, bc = tid & 15;
    float ra[8], rb[8];
    auto load = [&](int k0) {
        const float *pa = A + (i0 + ar) * ld + k0 + ak;
        const float *pb = B + (size_t) (k0 + br) * ld + j0 + bc;
#pragma unroll
        for (int q = 0; q < 8; ++q)
        {
            ra[q] = __ldg(pa + q);
            rb[q] = __ldg(pb + 16 * q);
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
        {
            As[buf][ak + q][ar] = ra[q];
            Bs[buf][br][bc + 16 * q] = rb[q];
        }
    };
    float acc[8][8];
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int n = 0; n < 8; ++n)
            acc[m][n] = 0.0f;
    load(0);
    store(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < Kp; k0 += DK)
    {
        const bool more = k0 + DK < Kp;
        if (more)
            load(k0 + DK);
#pragma unroll
        for (int k = 0; k < DK; ++k)
        {
            float a[8], b[8];
#pragma unroll
            for (int m = 0; m < 8; ++m)
                a[m] = As[buf][k][ty + 16 * m];
#pragma unroll
            for (int n = 0; n < 8; ++n)
                b[n] = Bs[buf][k][tx + 16 * n];
#pragma unroll
            for (int m = 0; m < 8; ++m)
#pragma unroll
                for (int n = 0; n < 8; ++n)
                    acc[m][n] = fmaf(a[m], b[n], acc[m][n]);
        }
        if (more)
        {
            store(buf ^ 1);
            __syncthreads();
            buf ^= 1;
        }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int n = 0; n < 8; ++n)
        {
            Cm[(i0 + ty + 16 * m) * ld + j0 + tx + 16 * n] = acc[m][n];
            if (sym && blockIdx.x > blockIdx.y)
                Cm[(j0 + tx + 16 * n) * ld + i0 + ty + 16 * m] = acc[m][n];
        }
}

// -------------------------------------------------------------------------
// FP64 GEMM on the tensor instructions (mma.sync m8n8k4, 37 TFLOP/s; the FMA
// pipe reaches 34).  128 x 128 of C per CTA of 8 warps, each 64 x 32 (8 x 4
// accumulator tiles, 64 doubles per lane); k in steps of 16 through a ring of
// GS stages filled by 16-byte cp.async, so three steps are in flight while one
// is multiplied.  Rows of A's stage are 20 doubles apart and rows of B's 132:
// the 16 lanes of a half warp, (row, k) = (lane / 4, lane % 4) of A and (k,
// column) = (lane % 4, lane / 4) of B, then read 16 distinct bank pairs.
// 12 8-byte loads feed 32 MMAs, an eighth of the shared-memory rate.
// Symmetric C (A == B with equal mirrored entries, *asym == 0): only the
// tiles on and above the diagonal are formed and each is stored twice.
// -------------------------------------------------------------------------
constexpr int GS = 4;                  // stages
constexpr int GA = 20, GB = DT + 4;    // row strides of the stages, in doubles
constexpr int GSTAGE = DT * GA + DK * GB;

__device__ __forceinline__ void cp16(double *dst, const double *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned) __cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

__global__ void __launch_bounds__(DTHREADS, 1) dense_gemm_f64_kernel(const double *__restrict__ A,
                                                                     const double *__restrict__ B,
                                                                     double *__restrict__ Cm, size_t ld, int Kp,
                                                                     const int *asym)
{
    extern __shared__ __align__(16) unsigned char dsm[];
    double *st = reinterpret_cast<double *>(dsm);
    const bool sym = asym && *asym == 0;
    if (sym && blockIdx.x < blockIdx.y)
        return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 2) * 64, wn = (warp & 3) * 32;
    const size_t i0 = (size_t) blockIdx.y * DT, j0 = (size_t) blockIdx.x * DT;
    // thread t copies 8 chunks: A row t >> 3 (+ 32 u), k 2 (t & 7); B row t >> 6 (+ 4 u), columns 2 (t & 63)
    const double *pa = A + (i0 + (tid >> 3)) * ld + 2 * (tid & 7);
    const double *pb = B + (size_t) (tid >> 6) * ld + j0 + 2 * (tid & 63);
    const int sa = (tid >> 3) * GA + 2 * (tid & 7), sb = DT * GA + (tid >> 6) * GB + 2 * (tid & 63);
    auto fetch = [&](int step) {
        double *s = st + (step % GS) * GSTAGE;
        const double *a = pa + (size_t) step * DK, *b = pb + (size_t) step * DK * ld;
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            cp16(s + sa + 32 * u * GA, a + 32 * u * ld);
            cp16(s + sb + 4 * u * GB, b + 4 * u * ld);
        }
    };
    double acc[8][4][2];
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n)
            acc[m][n][0] = acc[m][n][1] = 0.0;
    const int steps = Kp / DK;
    for (int s = 0; s < GS - 1; ++s)
    {
        fetch(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int fa = (wm + (lane >> 2)) * GA + (lane & 3), fb = DT * GA + (lane & 3) * GB + wn + (lane >> 2);
    for (int step = 0; step < steps; ++step)
    {
        asm volatile("cp.async.wait_group %0;" ::"n"(GS - 2) : "memory");
        __syncthreads();
        if (step + GS - 1 < steps)
            fetch(step + GS - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double *s = st + (step % GS) * GSTAGE;
#pragma unroll
        for (int k = 0; k < DK; k += 4)
        {
            double a[8], b[4];
#pragma unroll
            for (int m = 0; m < 8; ++m)
                a[m] = s[fa + 8 * m * GA + k];
#pragma unroll
            for (int n = 0; n < 4; ++n)
                b[n] = s[fb + k * GB + 8 * n];
#pragma unroll
            for (int m = 0; m < 8; ++m)
#pragma unroll
                for (int n = 0; n < 4; ++n)
                    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                                 : "+d"(acc[m][n][0]), "+d"(acc[m][n][1])
                                 : "d"(a[m]), "d"(b[n]));
        }
    }
    const int r = lane >> 2, q = 2 * (lane & 3);
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n)
        {
            const size_t row = i0 + wm + 8 * m + r, col = j0 + wn + 8 * n + q;
            *reinterpret_cast<double2 *>(Cm + row * ld + col) = make_double2(acc[m][n][0], acc[m][n][1]);
            if (sym && blockIdx.x > blockIdx.y)
            {
                Cm[col * ld + row] = acc[m][n][0];
                Cm[(col + 1) * ld + row] = acc[m][n][1];
            }
        }
}

// *asym = 1 when some entry of the image differs from its mirror (a NaN
// differs from itself).  One CTA per pair of 32 x 32 blocks.
template <typename T> __global__ void __launch_bounds__(256) dense_sym_kernel(const T *A, size_t ld, int *asym)
{
    __shared__ T t[32][33];
    if (blockIdx.x < blockIdx.y || __syncthreads_or(*(volatile int *) asym)) // other CTAs set it meanwhile
        return;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const size_t i0 = (size_t) blockIdx.y * 32, j0 = (size_t) blockIdx.x * 32;
    for (int r = y; r < 32; r += 8)
        t[r][x] = A[(j0 + r) * ld + i0 + x];
    __syncthreads();
    int bad = 0;
    for (int r = y; r < 32; r += 8)
        bad |= A[(i0 + r) * ld + j0 + x] != t[x][r];
    if (__any_sync(FULL, bad) && x == 0)
        atomicExch(asym, 1);
}

template <typename T> __device__ __forceinline__ bool above_d(T x, double thr);
template <> __device__ __forceinline__ bool above_d<double>(double x, double thr) { return fabs(x) > thr; }
template <> __device__ __forceinline__ bool above_d<float>(float x, double thr) { return fabsf(x) > (float) thr; }

// Row i of C from the image: the diagonal when touched, other columns when
// above the threshold, ascending; one warp per row.
template <typename T>
__global__ void __launch_bounds__(256) dense_compact_kernel(const T *img, size_t ld, int nrows, int ncols,
                                                            const int *touched, double thr, T *Cv, int *Ci, int *Cn,
                                                            int ldc, int Mc, double *dC, DenseFlags *flags)
{
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nrows; i += warps)
    {
        const T *row = img + (size_t) i * ld;
        const bool dt = touched[i] != 0;
        int n = 0;
        for (int b = 0; b < ncols; b += 32)
        {
            const int k = b + lane;
            bool keep = false;
            T x = T(0);
            if (k < ncols)
            {
                x = row[k];
                keep = k == i ? dt : above_d<T>(x, thr);
            }
            const unsigned bal = __ballot_sync(FULL, keep);
            const int pos = n + __popc(bal & lanemask_lt());
            if (keep && pos < Mc)
            {
                Ci[(size_t) i * ldc + pos] = k;
                Cv[(size_t) i * ldc + pos] = x;
            }
            n += __popc(bal);
        }
        if (lane == 0)
        {
            Cn[i] = min(n, Mc);
            atomicMax(&flags->max_width, n);
            if (n > Mc)
                atomicExch(&flags->overflow, 1);
            if (dC)
                dC[i] = (dt && i < ncols) ? (double) row[i] : 0.0;
        }
    }
}

bool g_dense_tier = true;

template <typename T>
bool dense_typed(bml_matrix_ellpack_t *A, bml_matrix_ellpack_t *B, bml_matrix_ellpack_t *C, double thr,
                 double *trace, int *required_M)
{
    B200Context *c = b200_ctx();
    if (!c)
        return false;
    const int NA = A->N, ncols = B->N > C->N ? B->N : C->N;
    const int dim = NA > ncols ? NA : ncols;
    const size_t ld = (size_t) b200_round_up(dim > B->N ? dim : B->N, DT);
    const size_t img = ld * ld * sizeof(T);
    const bool same = A == B;
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t off_b = al(img);
    const size_t off_c = al(off_b + (same ? 0 : img));
    const size_t off_p = al(off_c + img);
    const size_t off_t = al(off_p + ld * ld);
    const size_t off_d = al(off_t + (size_t) NA * sizeof(int));
    const size_t total = al(off_d + (size_t) 2 * NA * sizeof(double));
    unsigned char *scr = static_cast<unsigned char *>(b200_scratch(total));
    if (!scr)
        return false;
    T *DA = reinterpret_cast<T *>(scr);
    T *DB = same ? DA : reinterpret_cast<T *>(scr + off_b);
    T *DC = reinterpret_cast<T *>(scr + off_c);
    unsigned char *pat = scr + off_p;
    int *touched = reinterpret_cast<int *>(scr + off_t);
    double *dA = reinterpret_cast<double *>(scr + off_d);
    double *dC = dA + NA;
    unsigned char *small = static_cast<unsigned char *>(c->d_small) + 20480;
    DenseFlags *flags = reinterpret_cast<DenseFlags *>(small);
    double *dtrace = reinterpret_cast<double *>(small + 64);
    if (!CUDA_OK(cudaMemsetAsync(small, 0, 128, c->stream)) ||
        !CUDA_OK(cudaMemsetAsync(DA, 0, img, c->stream)) ||
        (!same && !CUDA_OK(cudaMemsetAsync(DB, 0, img, c->stream))) ||
        !CUDA_OK(cudaMemsetAsync(pat, 0, ld * ld, c->stream)))
        return false;
    const int wgrid = max(1, min(b200_ceil_div(dim, 8), c->sm_count * 16));
    if (!same)
    {
        dense_scatter_kernel<T><<<wgrid, 256, 0, c->stream>>>(static_cast<const T *>(A->d_value), A->d_index, A->d_nnz,
                                                              A->ld, NA, B->N, DA, ld, flags);
        if (!LAUNCH_OK("dense_scatter_kernel"))
            return false;
    }
    dense_scatter_kernel<T><<<wgrid, 256, 0, c->stream>>>(static_cast<const T *>(B->d_value), B->d_index, B->d_nnz,
                                                          B->ld, B->N, ncols, DB, ld, flags);
    if (!LAUNCH_OK("dense_scatter_kernel"))
        return false;
    const int *asym = same ? &flags->asym : nullptr;
    if (same)
    {
        dense_sym_kernel<T><<<dim3((unsigned) (ld / 32), (unsigned) (ld / 32)), 256, 0, c->stream>>>(DA, ld, &flags->asym);
        if (!LAUNCH_OK("dense_sym_kernel"))
            return false;
    }
    dense_pattern_kernel<<<wgrid, 256, 0, c->stream>>>(B->d_index, B->d_nnz, B->ld, B->N, ncols, pat, ld, asym);
    if (!LAUNCH_OK("dense_pattern_kernel"))
        return false;
    dense_diag_kernel<T><<<wgrid, 256, 0, c->stream>>>(static_cast<const T *>(A->d_value), A->d_index, A->d_nnz,
                                                       A->ld, NA, B->N, pat, ld, DA, asym, touched,
                                                       trace ? dA : nullptr);
    if (!LAUNCH_OK("dense_diag_kernel"))
        return false;
    const dim3 grid((unsigned) (ld / DT), (unsigned) (ld / DT));
    const int kp = b200_round_up(B->N, DK); // the images are zero from there on (N >= 1024)
    if constexpr (std::is_same<T, double>::value)
    {
        const size_t smemG = GS * GSTAGE * sizeof(double);
        if (!CUDA_OK(cudaFuncSetAttribute(dense_gemm_f64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int) smemG)))
            return false;
        dense_gemm_f64_kernel<<<grid, DTHREADS, smemG, c->stream>>>(DA, DB, DC, ld, kp, asym);
    }
    else
    {
        const size_t smemG = 4 * sizeof(T) * DK * DT;
        if (!CUDA_OK(cudaFuncSetAttribute(dense_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int) smemG)))
            return false;
        dense_gemm_kernel<<<grid, DTHREADS, smemG, c->stream>>>(DA, DB, DC, ld, kp, asym);
    }
    if (!LAUNCH_OK("dense_gemm_kernel"))
        return false;
    dense_compact_kernel<T><<<wgrid, 256, 0, c->stream>>>(DC, ld, NA, ncols, touched, thr, static_cast<T *>(C->d_value),
                                                          C->d_index, C->d_nnz, C->ld, C->M, trace ? dC : nullptr,
                                                          flags);
    if (!LAUNCH_OK("dense_compact_kernel"))
        return false;
    if (trace)
    {
        b200_sum_rows_kernel<<<1, 1024, 0, c->stream>>>(dA, dC, NA, dtrace);
        if (!LAUNCH_OK("b200_sum_rows_kernel"))
            return false;
    }
    unsigned char *pin = static_cast<unsigned char *>(c->pinned) + 20480;
    if (!CUDA_OK(cudaMemcpyAsync(pin, small, 128, cudaMemcpyDeviceToHost, c->stream)) || !b200_sync())
        return false;
    const DenseFlags *hf = reinterpret_cast<const DenseFlags *>(pin);
    if (required_M)
        *required_M = hf->max_width;
    if (hf->bad_input)
    {
        b200_set_error(BML_B200_ERR_INVALID, "multiply: a column index or row length of an input is out of range");
        return false;
    }
    if (trace)
        memcpy(trace, pin + 64, 2 * sizeof(double));
    if (hf->overflow)
    {
        b200_set_error(BML_B200_ERR_ROW_OVERFLOW, "Number of non-zeroes per row > M, Increase M (need %d, M = %d)",
                       hf->max_width, C->M);
        return false;
    }
    return true;
}

} // namespace

// The dense tier applies when both operands' rows fill at least 40 % of
// their columns on average (there the GEMM beats the sparse kernels), the
// threshold is >= 0, and the three images (and B's pattern) take at most
// 64 GiB.  The row totals cost one small reduction and a synchronisation,
// and are only looked at when M allows rows that wide.
bool ell_dense_fits(bml_matrix_ellpack_t *A, bml_matrix_ellpack_t *B, bml_matrix_ellpack_t *C, double thr)
{
    if (!g_dense_tier || !(thr >= 0.0) || A->N < 1024)
        return false;
    const int ncols = B->N > C->N ? B->N : C->N;
    if ((double) A->M < 0.4 * ncols || (double) B->M < 0.4 * ncols)
        return false;
    const size_t ld = (size_t) b200_round_up(A->N > ncols ? A->N : ncols, DT);
    const size_t bytes = ld * ld * (3 * prec_size(A->matrix_precision) + 1);
    if (bytes > ((size_t) 64 << 30))
        return false;
    long long ta = 0, tb = 0;
    int wa = 0, wb = 0;
    if (!ell_nnz_total(A, &ta, &wa) || (B != A && !ell_nnz_total(B, &tb, &wb)))
        return false;
    if (B == A)
        tb = ta;
    return (double) ta >= 0.4 * (double) A->N * ncols && (double) tb >= 0.4 * (double) B->N * ncols;
}

bool ell_multiply_dense(bml_matrix_ellpack_t *A, bml_matrix_ellpack_t *B, bml_matrix_ellpack_t *C, double thr,
                        double *trace, int *required_M)
{
    return A->matrix_precision == double_real ? dense_typed<double>(A, B, C, thr, trace, required_M)
                                              : dense_typed<float>(A, B, C, thr, trace, required_M);
}

// Allows (1, the default) or forbids (0) the dense tier; returns the previous setting.
extern "C" BML_B200_API int bml_b200_set_dense_tier(int allow)
{
    const int old = g_dense_tier ? 1 : 0;
    g_dense_tier = allow != 0;
    return old;
}
