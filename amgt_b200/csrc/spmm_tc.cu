// Multi-right-hand-side mBSR SpMM with row-major multivectors:
//   Y (m x nvec) <- alpha * A * X (n x nvec) + beta * Y,  nvec <= 32,
// X[i * nvec + v], Y[i * nvec + v], fp64 in memory.  The batching form's
// operator: one pass over A's values for all right-hand sides (the
// reference's hook ignores num_vectors, AmgT_HYPRE/src/seq_mv/
// csr_matvec_device.c:2409-2437; its tensor-core SpMV is bsr_spmv_tc_fp64,
// :452-507).
//
// Tensor-core form (values in fp32 / fp16 / bf16): one warp takes two block
// rows b1, b2 at a time and walks their blocks in step (block t of each
// row); per step one mma.m16n8k8 (tf32 in, fp32 accumulate) per 16
// right-hand sides computes
//   D (16 rhs x 8 outputs) += Xg (16 rhs x 8) * Bop (8 x 8)
// with K = [the 4 columns of b1's block t | the 4 columns of b2's block t]
// and N = [b1's 4 rows | b2's 4 rows]: Bop = [A1^T 0; 0 A2^T] (block
// diagonal), Xg the gathered rows of X.  Half of Bop is zero, and in
// exchange every lane loads exactly one value per step (lane l < 16: entry
// l of b1's block, l >= 16: entry l - 16 of b2's block, which is the
// mma's B fragment element for that lane) and no shuffle is needed.  fp32
// accuracy on the tf32 units: values and x are split as v = hi + lo
// (hi = tf32(v), lo = tf32(v - hi)) and D accumulates hi*hi + lo*hi + hi*lo
// (fp16 / bf16 values are exact in tf32: two products).  The op stays
// bandwidth-bound, so the extra mma work is free.
//
// CUDA-core form (any precision, fp64 for fp64 values): see its kernel.
//
// Deterministic: every output sums its blocks in stored order.
#include "spmv_common.cuh"

#include "spmm.cuh"

namespace amgt {

__device__ __forceinline__ uint32_t to_tf32(float f)
{
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(f));
    return r;
}

__device__ __forceinline__ void mma_tf32(float d[4], const uint32_t a[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int PREC>
__device__ __forceinline__ float load_val1(const void *__restrict__ val, long long i)
{
    if constexpr (PREC == AMGT_FLOAT) return __ldcs(static_cast<const float *>(val) + i);
    else if constexpr (PREC == AMGT_HALF)
        return __half2float(__ushort_as_half(__ldcs(static_cast<const unsigned short *>(val) + i)));
    else return __bfloat162float(__ushort_as_bfloat16(__ldcs(static_cast<const unsigned short *>(val) + i)));
}

// NH halves of 16 right-hand sides (nvec <= 16 * NH); WPC warps per CTA.
template <int PREC, int NH, int WPC>
__global__ void __launch_bounds__(WPC * 32)
spmm_tc_kernel(int m, int n, int brow, const int *__restrict__ ptr, const int *__restrict__ idx,
               const void *__restrict__ val, double alpha, const double *__restrict__ X, int nvec, double beta,
               double *__restrict__ Y)
{
    grid_dependency_wait();
    constexpr bool kSplitA = PREC == AMGT_FLOAT;  // fp16 / bf16 values are exact in tf32
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int npairs = (brow + 1) >> 1;
    const bool upper = lane >= 16;  // this lane's block value comes from b2
    for (int p = warp; p < npairs; p += nwarps) {
        const int b1 = 2 * p, b2 = 2 * p + 1;
        const int s1 = ptr[b1], e1 = ptr[b1 + 1];
        const int s2 = b2 < brow ? ptr[b2] : 0, e2 = b2 < brow ? ptr[b2 + 1] : 0;
        const int len = max(e1 - s1, e2 - s2);
        const int ms = upper ? s2 : s1, me = upper ? e2 : e1;
        float acc[NH][4];
#pragma unroll
        for (int h = 0; h < NH; ++h)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[h][q] = 0.0f;
        for (int t = 0; t < len; ++t) {
            const int kb = ms + t;
            const bool mine = kb < me;
            const float a = mine ? load_val1<PREC>(val, 16LL * kb + (lane & 15)) : 0.0f;
            const int cm = mine ? __ldcs(idx + kb) : -1;
            const int c1 = __shfl_sync(FULL, cm, 0), c2 = __shfl_sync(FULL, cm, 16);
            const uint32_t ahi = to_tf32(a);
            const uint32_t b0h = upper ? 0u : ahi, b1h = upper ? ahi : 0u;
            uint32_t b0l = 0u, b1l = 0u;
            if constexpr (kSplitA) {
                const uint32_t alo = to_tf32(a - __uint_as_float(ahi));
                b0l = upper ? 0u : alo;
                b1l = upper ? alo : 0u;
            }
            const long long r1 = 4LL * c1 + tig, r2 = 4LL * c2 + tig;
            const bool ok1 = c1 >= 0 && r1 < n, ok2 = c2 >= 0 && r2 < n;
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                const int v0 = 16 * h + gid, v1 = v0 + 8;
                double xv[4];
                xv[0] = (ok1 && v0 < nvec) ? X[r1 * nvec + v0] : 0.0;
                xv[1] = (ok1 && v1 < nvec) ? X[r1 * nvec + v1] : 0.0;
                xv[2] = (ok2 && v0 < nvec) ? X[r2 * nvec + v0] : 0.0;
                xv[3] = (ok2 && v1 < nvec) ? X[r2 * nvec + v1] : 0.0;
                uint32_t xh[4], xl[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float f = (float)xv[q];
                    xh[q] = to_tf32(f);
                    xl[q] = to_tf32((float)(xv[q] - (double)__uint_as_float(xh[q])));
                }
                mma_tf32(acc[h], xh, b0h, b1h);
                mma_tf32(acc[h], xl, b0h, b1h);
                if constexpr (kSplitA) mma_tf32(acc[h], xh, b0l, b1l);
            }
        }
        // D fragment: (rhs gid, output 2 tig), (gid, 2 tig + 1), (gid + 8, 2 tig), (gid + 8, 2 tig + 1)
#pragma unroll
        for (int h = 0; h < NH; ++h)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int v = 16 * h + gid + ((q & 2) ? 8 : 0);
                const int o = 2 * tig + (q & 1);
                const int b = o < 4 ? b1 : b2;
                const int row = 4 * b + (o & 3);
                if (b < brow && row < m && v < nvec) {
                    double *yy = Y + (long long)row * nvec + v;
                    const double r = alpha * (double)acc[h][q];
                    *yy = (beta == 0.0) ? r : r + beta * *yy;
                }
            }
    }
}

// CUDA-core form: GL lanes per block row (4, 8 or 16 for up to 8, 16 or 32
// right-hand sides), two right-hand sides a lane.  A block's 16 values are
// read by every lane of the group (one broadcast access), its X rows only
// where the bitmap has an entry in their column, the next block's column and
// bitmap a step ahead.  A CTA takes consecutive block rows from first to
// last, so that the X rows of neighbouring block rows (the row's own line and
// the lines beside it) are found in L1: at 32 right-hand sides a block row
// reads 20 to 28 X rows of 256 bytes, and from L2 that traffic would be 463 MB
// a product of the 64^3 7-point operator, which itself is 151 MB.  Measured
// there (fp16 storage, 32 right-hand sides, calls back to back): 45.5 us, 3.3
// TB/s of the 151 MB; a warp per block row with values broadcast by shuffles
// 72, the tensor-core form 76.  Latency and registers bound it: one block at a
// time leaves the 64 registers of 1,024 threads per SM to the loads in flight
// (two at a time 47.4 us; 27 right-hand sides 52.5 against 60.2, with 8-byte
// values 68 against 117), except 8-byte values at strides known at compile
// time (100^3, 16 right-hand sides: two 144 us, one 161).
//
// Operators of few block rows: `split` parts of GL lanes take a block row's
// blocks in turn (their sums are added by shuffles, in the same order every
// time), while the GPU holds all threads at once, and the CTAs shrink until
// one lands on every SM.  27-point 10^3 (250 block rows), 8 right-hand sides,
// fp16: 13.1 -> 2.7 us (tensor cores 10.4); 4,921 block rows 15.4 -> 5.1 (13.8).
//
// The epilogues fuse the vector passes of the multi-right-hand-side cycle
// (multirhs.cu), with the arithmetic of the separate passes.
constexpr int kCcThreads = 512;

template <int PREC>
__device__ __forceinline__ void block_values(const void *__restrict__ val, long long k,
                                             typename ValTraits<PREC>::acc_t v[16])
{
    if constexpr (PREC == AMGT_DOUBLE) {
        const double2 *p = static_cast<const double2 *>(val) + 8 * k;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const double2 t = __ldcs(p + i);
            v[2 * i] = t.x;
            v[2 * i + 1] = t.y;
        }
    } else if constexpr (PREC == AMGT_FLOAT) {
        const float4 *p = static_cast<const float4 *>(val) + 4 * k;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 t = __ldcs(p + i);
            v[4 * i] = t.x;
            v[4 * i + 1] = t.y;
            v[4 * i + 2] = t.z;
            v[4 * i + 3] = t.w;
        }
    } else {
        const uint4 *p = static_cast<const uint4 *>(val) + 2 * k;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint4 t = __ldcs(p + i);
            const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float2 f;
                if constexpr (PREC == AMGT_HALF) f = __half22float2(*reinterpret_cast<const __half2 *>(&w[j]));
                else f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w[j]));
                v[8 * i + 2 * j] = f.x;
                v[8 * i + 2 * j + 1] = f.y;
            }
        }
    }
}

// Lane l's two right-hand sides of a row-major multivector's rows.  VEC 0: l
// and l + nvec / 2, two scalar accesses, each contiguous over the lanes (an odd
// count's middle one twice, stored once; 3: the same for a matrix without
// bitmaps); 1: 2 l and 2 l + 1, one 16-byte access; 2: the same for exactly 2 GL
// right-hand sides (strides known at compile time).  A lane without a
// right-hand side reads another's: a test in every load parts the loads.
template <int GL, int VEC>
struct MvCols {
    static constexpr bool pair = VEC == 1 || VEC == 2;
    int nvec, c0, second;
    bool on0, on1;
    __device__ __forceinline__ MvCols(int nv, int l)
    {
        nvec = VEC == 2 ? 2 * GL : nv;
        second = pair ? 1 : nv / 2;
        on0 = VEC == 2 || (pair ? 2 * l < nv : l < nv / 2);
        on1 = VEC == 2 || (pair ? on0 : l < nv - nv / 2);
        c0 = VEC == 2 ? 2 * l : pair ? min(2 * l, nv - 2) : min(l, nv - nv / 2 - 1);
    }
    __device__ __forceinline__ double2 load(const double *__restrict__ X, long long row) const
    {
        const double *p = X + row * nvec + c0;
        if constexpr (pair) return *reinterpret_cast<const double2 *>(p);
        else return make_double2(p[0], p[second]);
    }
    __device__ __forceinline__ void store(double *__restrict__ Y, long long row, double2 t) const
    {
        double *p = Y + row * nvec + c0;
        if constexpr (pair) {
            if (on0) *reinterpret_cast<double2 *>(p) = t;
        } else {
            if (on0) p[0] = t.x;
            if (on1) p[second] = t.y;
        }
    }
};

// SPLIT 1: one part a block row, known at compile time; 0: a.split parts.
template <int PREC, int GL, int VEC, int EPI, int SPLIT>
__global__ void __launch_bounds__(kCcThreads, 2)
spmm_cc_kernel(const __grid_constant__ MvArgs a)
{
    grid_dependency_wait();
    using acc_t = typename ValTraits<PREC>::acc_t;
    constexpr int U = PREC == AMGT_DOUBLE && VEC == 2 ? 2 : 1;  // blocks in flight
    constexpr bool kDot = EPI == MV_DOT || EPI == MV_JACOBI;
    __shared__ double sred[kDot ? kCcThreads / 32 : 1][32];
    const int l = threadIdx.x % GL;
    const MvCols<GL, VEC> mv(a.nvec, l);
    // a block row's lanes: `split` parts of GL (a power of two, within a warp)
    const int split = SPLIT ? SPLIT : a.split, part = threadIdx.x / GL & (split - 1);
    const unsigned lanes = GL * split == 32 ? FULL : ((1u << (GL * split)) - 1u) << (threadIdx.x & 31 & ~(GL * split - 1));
    const int groups = blockDim.x / (GL * split);
    const int per = (a.brow + gridDim.x - 1) / gridDim.x;
    const int bend = min(a.brow, (int)(blockIdx.x + 1) * per);
    double2 dot = make_double2(0.0, 0.0);
    for (int b = blockIdx.x * per + threadIdx.x / (GL * split); b < bend; b += groups) {
        acc_t acc[4][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = (acc_t)0;
        const int k1 = a.ptr[b + 1];
        // the next blocks' columns and bitmaps are read a step ahead (a set
        // bit also says that the X row exists)
        uint32_t mpn[U];
        int cn[U];
        auto head = [&](int k) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                mpn[u] = 0u;
                cn[u] = 0;
                if (k + u < k1) {
                    cn[u] = __ldcs(a.idx + k + u);
                    if constexpr (VEC == 3) mpn[u] = 0x1111u * ((1u << min(4, a.n - 4 * cn[u])) - 1u);  // full blocks
                    else mpn[u] = a.map[k + u];
                }
            }
        };
        int k = a.ptr[b] + U * part;
        head(k);
        for (; k < k1; k += U * split) {
            uint32_t mp[U];
            int c[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                mp[u] = mpn[u];
                c[u] = cn[u];
            }
            head(k + U * split);
            double2 x[U][4];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    const long long r = 4LL * c[u] + cc;
                    x[u][cc] = make_double2(0.0, 0.0);
                    if (mp[u] & (0x1111u << cc)) {
                        x[u][cc] = mv.load(a.X, r);
                        if constexpr (EPI == MV_RESID0) {  // the zero-guess sweep's u, entry by entry
                            const double li = __ldg(a.inv_l1 + r);
                            x[u][cc].x = a.alpha * x[u][cc].x * li;
                            x[u][cc].y = a.alpha * x[u][cc].y * li;
                        }
                    }
                }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (u > 0 && k + u >= k1) break;  // the same for the group; a re-read block's infinity would meet zero x
                acc_t v[16];
                block_values<PREC>(a.val, k + u, v);
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) {
                        acc[r][0] = fma(v[4 * r + cc], (acc_t)x[u][cc].x, acc[r][0]);
                        acc[r][1] = fma(v[4 * r + cc], (acc_t)x[u][cc].y, acc[r][1]);
                    }
            }
        }
        // the parts' sums, in the same order every time; part p writes the
        // rows r = p mod split
        for (int o = GL; o < GL * split; o <<= 1)
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) acc[r][c] += __shfl_xor_sync(lanes, acc[r][c], o);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const long long row = 4LL * b + r;
            if (row >= a.m || ((r ^ part) & (split - 1)) != 0) continue;
            const double2 ax = make_double2((double)acc[r][0], (double)acc[r][1]);
            double2 t;
            if constexpr (EPI == MV_SPMM) {
                t = make_double2(a.alpha * ax.x, a.alpha * ax.y);
                if (a.beta != 0.0) {
                    const double2 y = mv.load(a.Y, row);
                    t.x += a.beta * y.x;
                    t.y += a.beta * y.y;
                }
            } else if constexpr (EPI == MV_RESID || EPI == MV_RESID0) {
                const double2 f = mv.load(a.F, row);
                t = make_double2(f.x - ax.x, f.y - ax.y);
            } else if constexpr (EPI == MV_CORRECT) {
                const double2 f = mv.load(a.F, row);
                const double li = __ldg(a.inv_l1 + row);
                t = make_double2(ax.x + a.alpha * f.x * li, ax.y + a.alpha * f.y * li);
            } else if constexpr (EPI == MV_JACOBI) {
                const double2 f = mv.load(a.F, row), u = mv.load(a.X, row);
                const double li = __ldg(a.inv_l1 + row);
                t = make_double2(u.x + a.alpha * (f.x - ax.x) * li, u.y + a.alpha * (f.y - ax.y) * li);
                dot.x += f.x * t.x;
                dot.y += f.y * t.y;
            } else {
                const double2 u = mv.load(a.X, row);
                t = ax;
                dot.x += u.x * t.x;
                dot.y += u.y * t.y;
            }
            mv.store(a.Y, row, t);
        }
    }
    if constexpr (kDot) {
        if (!a.part) return;  // the same for every thread
        // fixed order: groups of a warp, then warps
#pragma unroll
        for (int o = GL; o < 32; o <<= 1) {
            dot.x += __shfl_xor_sync(FULL, dot.x, o);
            dot.y += __shfl_xor_sync(FULL, dot.y, o);
        }
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (lane < 16) sred[warp][2 * lane] = sred[warp][2 * lane + 1] = 0.0;
        __syncwarp();
        if (lane < GL) {
            if (mv.on0) sred[warp][mv.c0] = dot.x;
            if (mv.on1) sred[warp][mv.c0 + mv.second] = dot.y;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            double t = 0.0;
            for (int w = 0; w < (int)blockDim.x / 32; ++w) t += sred[w][threadIdx.x];
            a.part[blockIdx.x * 32 + threadIdx.x] = t;
        }
    }
}

// ---------------------------------------------------------------- launch
// Launch shape of the CUDA-core form.
struct CcShape {
    int gl, split, threads, grid;
};
static CcShape cc_shape(const amgt_bsr *A, int nvec, int wpc, int sm_count)
{
    CcShape c{nvec <= 8 ? 4 : nvec <= 16 ? 8 : 16, 1, 64 * wpc, 1};
    const double avg = (double)A->blc_num / A->blc_row;
    // parts of a block row: as many as keep two blocks each on average, while
    // the GPU holds all their threads at once
    while (2 * c.split * c.gl <= 32 && avg > 2 * c.split &&
           2LL * c.split * c.gl * A->blc_row <= 1024LL * sm_count)
        c.split *= 2;
    // CTAs small enough to land on every SM
    while (c.threads > 64 && (long long)c.gl * c.split * A->blc_row < (long long)c.threads * sm_count) c.threads /= 2;
    c.grid = grid_for(c.threads / (c.gl * c.split), A->blc_row, sm_count, 1024 / (64 * wpc));
    return c;
}

template <int PREC, int EPI>
static int launch_cc(const amgt_bsr *A, const void *val, int nvec, int wpc, MvArgs a, cudaStream_t s, int sm_count)
{
    const CcShape c = cc_shape(A, nvec, wpc, sm_count);
    a.m = A->row;
    a.n = A->col;
    a.brow = A->blc_row;
    a.nvec = nvec;
    a.split = c.split;
    a.ptr = A->blcPtr;
    a.idx = A->blcIdx;
    a.map = A->blcMap;
    a.val = val;
    // two right-hand sides in one 16-byte access: rows of an even count at
    // 16-byte aligned bases
    const bool vec = nvec % 2 == 0 && (((uintptr_t)a.X | (uintptr_t)a.Y | (uintptr_t)a.F) % 16) == 0;
    const int form = !a.map ? 3 : !vec ? 0 : nvec == 2 * c.gl ? 2 : 1;
#define AMGT_CC_CASE(GL, VEC, SPLIT)                                                                    \
    if (c.gl == GL && form == VEC && (SPLIT == 0 || c.split == SPLIT)) {                                \
        AMGT_LAUNCH_PDL((spmm_cc_kernel<PREC, GL, VEC, EPI, SPLIT>), c.grid, c.threads, 0, s, a);        \
        return AMGT_OK;                                                                                 \
    }
    if constexpr (EPI == MV_SPMM) {  // the multi-right-hand-side cycle's operators have bitmaps
        AMGT_CC_CASE(4, 3, 0)
        AMGT_CC_CASE(8, 3, 0)
        AMGT_CC_CASE(16, 3, 0)
    }
    if constexpr (PREC == AMGT_DOUBLE) {  // one part, known at compile time: 3 to 5 % at 8-byte values, none at others
        AMGT_CC_CASE(4, 0, 1)
        AMGT_CC_CASE(8, 0, 1)
        AMGT_CC_CASE(16, 0, 1)
        AMGT_CC_CASE(16, 1, 1)
        AMGT_CC_CASE(16, 2, 1)
    }
    AMGT_CC_CASE(4, 0, 0)
    AMGT_CC_CASE(4, 1, 0)
    AMGT_CC_CASE(4, 2, 0)
    AMGT_CC_CASE(8, 0, 0)
    AMGT_CC_CASE(8, 1, 0)
    AMGT_CC_CASE(8, 2, 0)
    AMGT_CC_CASE(16, 0, 0)
    AMGT_CC_CASE(16, 1, 0)
    AMGT_CC_CASE(16, 2, 0)
#undef AMGT_CC_CASE
    return AMGT_ERR_INVALID;
}

// kind: 0 CUDA cores, 1 tensor cores; wpc: warps per CTA (4 or 8).
template <int PREC, int WPC>
static int launch_rm(int kind, const amgt_bsr *A, const void *val, double alpha, const double *X, int nvec,
                     double beta, double *Y, cudaStream_t s, int sm_count)
{
    const int brow = A->blc_row;
    if (kind == 1) {
        if constexpr (PREC == AMGT_DOUBLE) {
            return AMGT_ERR_UNSUPPORTED;
        } else {
            const int grid = grid_for(WPC, (brow + 1) / 2, sm_count, 16);
            if (nvec <= 16)
                AMGT_LAUNCH_PDL((spmm_tc_kernel<PREC, 1, WPC>), grid, WPC * 32, 0, s, A->row, A->col, brow, A->blcPtr,
                                A->blcIdx, val, alpha, X, nvec, beta, Y);
            else
                AMGT_LAUNCH_PDL((spmm_tc_kernel<PREC, 2, WPC>), grid, WPC * 32, 0, s, A->row, A->col, brow, A->blcPtr,
                                A->blcIdx, val, alpha, X, nvec, beta, Y);
            return AMGT_OK;
        }
    }
    MvArgs a{};
    a.alpha = alpha;
    a.beta = beta;
    a.X = X;
    a.Y = Y;
    return launch_cc<PREC, MV_SPMM>(A, val, nvec, WPC, a, s, sm_count);
}

template <int PREC>
static int launch_rm_prec(int kind, int wpc, const amgt_bsr *A, const void *val, double alpha, const double *X,
                          int nvec, double beta, double *Y, cudaStream_t s, int sm_count)
{
    return wpc == 8 ? launch_rm<PREC, 8>(kind, A, val, alpha, X, nvec, beta, Y, s, sm_count)
                    : launch_rm<PREC, 4>(kind, A, val, alpha, X, nvec, beta, Y, s, sm_count);
}

static const void *rm_values(const amgt_bsr *A, int prec)
{
    switch (prec) {
    case AMGT_DOUBLE: return A->blcVal;
    case AMGT_FLOAT: return A->blcVal_fp32;
    case AMGT_HALF: return A->blcVal_fp16;
    case AMGT_BF16: return A->blcVal_bf16;
    default: return nullptr;
    }
}

// The storage read for `prec`: fp32 requests read an exact fp16 shadow
// (same inputs, half the bytes); fp64 keeps 8-byte values here.
static int rm_storage(const amgt_bsr *A, int prec)
{
    if (prec == AMGT_FLOAT && A->exact_prec == AMGT_HALF && A->blcVal_fp16) return AMGT_HALF;
    return prec;
}

int spmm_rowmajor(int prec, int kind, int wpc, const amgt_bsr *A, double alpha, const double *X, int nvec,
                  double beta, double *Y, cudaStream_t s, int sm_count)
{
    const int mode = rm_storage(A, prec);
    const void *val = rm_values(A, mode);
    if (!val) return AMGT_ERR_INVALID;
    if (mode == AMGT_DOUBLE && kind == 1) kind = 0;  // fp64 values: CUDA cores
    switch (mode) {
    case AMGT_DOUBLE: return launch_rm_prec<AMGT_DOUBLE>(kind, wpc, A, val, alpha, X, nvec, beta, Y, s, sm_count);
    case AMGT_FLOAT: return launch_rm_prec<AMGT_FLOAT>(kind, wpc, A, val, alpha, X, nvec, beta, Y, s, sm_count);
    case AMGT_HALF: return launch_rm_prec<AMGT_HALF>(kind, wpc, A, val, alpha, X, nvec, beta, Y, s, sm_count);
    default: return launch_rm_prec<AMGT_BF16>(kind, wpc, A, val, alpha, X, nvec, beta, Y, s, sm_count);
    }
}

int mv_apply_grid(const amgt_bsr *A, int nvec, int sm_count) { return cc_shape(A, nvec, 8, sm_count).grid; }

template <int EPI>
static int launch_apply(int prec, const amgt_bsr *A, int nvec, const MvArgs &a, cudaStream_t s, int sm_count)
{
    const int mode = rm_storage(A, prec);
    const void *val = rm_values(A, mode);
    if (!val) return AMGT_ERR_INVALID;
    if constexpr (EPI == MV_RESID) {  // the refinement's residual: fp64 values only
        return mode == AMGT_DOUBLE ? launch_cc<AMGT_DOUBLE, EPI>(A, val, nvec, 8, a, s, sm_count) : AMGT_ERR_INVALID;
    } else
    switch (mode) {
    case AMGT_DOUBLE: return launch_cc<AMGT_DOUBLE, EPI>(A, val, nvec, 8, a, s, sm_count);
    case AMGT_FLOAT: return launch_cc<AMGT_FLOAT, EPI>(A, val, nvec, 8, a, s, sm_count);
    case AMGT_HALF: return launch_cc<AMGT_HALF, EPI>(A, val, nvec, 8, a, s, sm_count);
    default: return launch_cc<AMGT_BF16, EPI>(A, val, nvec, 8, a, s, sm_count);
    }
}

int mv_apply(int prec, int epi, const amgt_bsr *A, int nvec, const MvArgs &a, cudaStream_t s, int sm_count)
{
    switch (epi) {
    case MV_SPMM: return launch_apply<MV_SPMM>(prec, A, nvec, a, s, sm_count);
    case MV_RESID: return launch_apply<MV_RESID>(prec, A, nvec, a, s, sm_count);
    case MV_RESID0: return launch_apply<MV_RESID0>(prec, A, nvec, a, s, sm_count);
    case MV_CORRECT: return launch_apply<MV_CORRECT>(prec, A, nvec, a, s, sm_count);
    case MV_JACOBI: return launch_apply<MV_JACOBI>(prec, A, nvec, a, s, sm_count);
    case MV_DOT: return launch_apply<MV_DOT>(prec, A, nvec, a, s, sm_count);
    default: return AMGT_ERR_INVALID;
    }
}

}  // namespace amgt
