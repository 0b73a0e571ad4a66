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
// read by every lane of the group (one broadcast access), its X rows as
// 16-byte loads of two right-hand sides, only those whose column the bitmap
// has an entry in; two blocks in flight.  A CTA takes consecutive block rows
// from first to last, so that the X rows of neighbouring block rows (the
// row's own line and the lines beside it) are found in L1: at 32 right-hand
// sides a block row reads 20 to 28 X rows of 256 bytes, and from L2 that
// traffic would be 463 MB a product of the 64^3 7-point operator, which itself
// is 151 MB.  Measured there (fp16 storage, 32 right-hand sides): 50.6 us, 3.0
// TB/s of the 151 MB; the warp-per-block-row form with values broadcast by
// shuffles that this replaces took 73 us, the tensor-core form 76.  Latency
// bounds it (ncu: 51 % issue, 9.6 of 14.6 stall cycles on global loads): the
// columns read a pair ahead and strides known at compile time took it from 100
// us, 24 warps or fewer registers per SM gave 60 and 68 us.
//
// The epilogues fuse the vector passes of the multi-right-hand-side cycle
// (multirhs.cu), with the arithmetic of the separate passes.
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

// Access to right-hand sides v0, v0 + 1 of a row-major multivector's rows:
// VEC 0 two scalars, 1 one 16-byte access, 2 the same for exactly 32
// right-hand sides (constant strides; bitmaps present).
template <int VEC>
__device__ __forceinline__ double2 mv_load(const double *__restrict__ X, long long row, int nvec, int v0)
{
    const double *p = X + row * (VEC == 2 ? 32 : nvec) + v0;
    if constexpr (VEC == 2) return *reinterpret_cast<const double2 *>(p);
    else if constexpr (VEC == 1) return v0 < nvec ? *reinterpret_cast<const double2 *>(p) : make_double2(0.0, 0.0);
    else return make_double2(v0 < nvec ? p[0] : 0.0, v0 + 1 < nvec ? p[1] : 0.0);
}
template <int VEC>
__device__ __forceinline__ void mv_store(double *__restrict__ Y, long long row, int nvec, int v0, double2 t)
{
    double *p = Y + row * (VEC == 2 ? 32 : nvec) + v0;
    if constexpr (VEC == 2) {
        *reinterpret_cast<double2 *>(p) = t;
    } else if constexpr (VEC == 1) {
        if (v0 < nvec) *reinterpret_cast<double2 *>(p) = t;
    } else {
        if (v0 < nvec) p[0] = t.x;
        if (v0 + 1 < nvec) p[1] = t.y;
    }
}

template <int PREC, int GL, int VEC, int EPI, int WPC>
__global__ void __launch_bounds__(WPC * 64, 16 / WPC)
spmm_cc_kernel(const __grid_constant__ MvArgs a)
{
    grid_dependency_wait();
    using acc_t = typename ValTraits<PREC>::acc_t;
    constexpr int GROUPS = WPC * 64 / GL;
    constexpr bool kDot = EPI == MV_DOT || EPI == MV_JACOBI;
    __shared__ double sred[kDot ? WPC * 2 : 1][32];
    const int l = threadIdx.x % GL, v0 = 2 * l, nvec = a.nvec;
    const int per = (a.brow + gridDim.x - 1) / gridDim.x;
    const int bend = min(a.brow, (int)(blockIdx.x + 1) * per);
    double2 dot = make_double2(0.0, 0.0);
    for (int b = blockIdx.x * per + threadIdx.x / GL; b < bend; b += GROUPS) {
        acc_t acc[4][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = (acc_t)0;
        const int k1 = a.ptr[b + 1];
        // the next pair's columns and bitmaps are read a pair ahead (a set
        // bit also says that the X row exists)
        uint32_t mpn[2];
        int cn[2];
        auto head = [&](int k) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                mpn[u] = 0u;
                cn[u] = 0;
                if (k + u < k1) {
                    cn[u] = __ldcs(a.idx + k + u);
                    if (VEC == 2 || a.map) mpn[u] = a.map[k + u];
                    else mpn[u] = 0x1111u * ((1u << min(4, a.n - 4 * cn[u])) - 1u);  // no bitmaps: full blocks
                }
            }
        };
        int k = a.ptr[b];
        head(k);
        for (; k < k1; k += 2) {
            uint32_t mp[2];
            int c[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                mp[u] = mpn[u];
                c[u] = cn[u];
            }
            head(k + 2);
            double2 x[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    const long long r = 4LL * c[u] + cc;
                    x[u][cc] = make_double2(0.0, 0.0);
                    if (mp[u] & (0x1111u << cc)) {
                        x[u][cc] = mv_load<VEC>(a.X, r, nvec, v0);
                        if constexpr (EPI == MV_RESID0) {  // the zero-guess sweep's u, entry by entry
                            const double li = __ldg(a.inv_l1 + r);
                            x[u][cc].x = a.alpha * x[u][cc].x * li;
                            x[u][cc].y = a.alpha * x[u][cc].y * li;
                        }
                    }
                }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
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
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const long long row = 4LL * b + r;
            if (row >= a.m) continue;
            const double2 ax = make_double2((double)acc[r][0], (double)acc[r][1]);
            double2 t;
            if constexpr (EPI == MV_SPMM) {
                t = make_double2(a.alpha * ax.x, a.alpha * ax.y);
                if (a.beta != 0.0) {
                    const double2 y = mv_load<VEC>(a.Y, row, nvec, v0);
                    t.x += a.beta * y.x;
                    t.y += a.beta * y.y;
                }
            } else if constexpr (EPI == MV_RESID || EPI == MV_RESID0) {
                const double2 f = mv_load<VEC>(a.F, row, nvec, v0);
                t = make_double2(f.x - ax.x, f.y - ax.y);
            } else if constexpr (EPI == MV_CORRECT) {
                const double2 f = mv_load<VEC>(a.F, row, nvec, v0);
                const double li = __ldg(a.inv_l1 + row);
                t = make_double2(ax.x + a.alpha * f.x * li, ax.y + a.alpha * f.y * li);
            } else if constexpr (EPI == MV_JACOBI) {
                const double2 f = mv_load<VEC>(a.F, row, nvec, v0), u = mv_load<VEC>(a.X, row, nvec, v0);
                const double li = __ldg(a.inv_l1 + row);
                t = make_double2(u.x + a.alpha * (f.x - ax.x) * li, u.y + a.alpha * (f.y - ax.y) * li);
                dot.x += f.x * t.x;
                dot.y += f.y * t.y;
            } else {
                const double2 u = mv_load<VEC>(a.X, row, nvec, v0);
                t = ax;
                dot.x += u.x * t.x;
                dot.y += u.y * t.y;
            }
            mv_store<VEC>(a.Y, row, nvec, v0, t);
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
            sred[warp][v0] = dot.x;
            sred[warp][v0 + 1] = dot.y;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            double t = 0.0;
            for (int w = 0; w < WPC * 2; ++w) t += sred[w][threadIdx.x];
            a.part[blockIdx.x * 32 + threadIdx.x] = t;
        }
    }
}

// ---------------------------------------------------------------- launch
// The CUDA-core form's CTAs: 2 x 512 or 4 x 256 threads per SM.
template <int WPC>
static int cc_grid(const amgt_bsr *A, int nvec, int sm_count)
{
    const int gl = nvec <= 8 ? 4 : nvec <= 16 ? 8 : 16;
    return grid_for(WPC * 64 / gl, A->blc_row, sm_count, 16 / WPC);
}

template <int PREC, int EPI, int WPC>
static int launch_cc(const amgt_bsr *A, const void *val, int nvec, MvArgs a, cudaStream_t s, int sm_count)
{
    a.m = A->row;
    a.n = A->col;
    a.brow = A->blc_row;
    a.nvec = nvec;
    a.ptr = A->blcPtr;
    a.idx = A->blcIdx;
    a.map = A->blcMap;
    a.val = val;
    const int grid = cc_grid<WPC>(A, nvec, sm_count);
    // two right-hand sides in one 16-byte access: rows of an even count at
    // 16-byte aligned bases
    const bool vec = nvec % 2 == 0 && (((uintptr_t)a.X | (uintptr_t)a.Y | (uintptr_t)a.F) % 16) == 0;
#define AMGT_CC_CASE(GL)                                                                                    \
    if (vec) AMGT_LAUNCH_PDL((spmm_cc_kernel<PREC, GL, 1, EPI, WPC>), grid, WPC * 64, 0, s, a);               \
    else AMGT_LAUNCH_PDL((spmm_cc_kernel<PREC, GL, 0, EPI, WPC>), grid, WPC * 64, 0, s, a);                   \
    return AMGT_OK
    if (nvec <= 8) {
        AMGT_CC_CASE(4);
    }
    if (nvec <= 16) {
        AMGT_CC_CASE(8);
    }
    if (vec && nvec == 32 && A->blcMap) {
        AMGT_LAUNCH_PDL((spmm_cc_kernel<PREC, 16, 2, EPI, WPC>), grid, WPC * 64, 0, s, a);
        return AMGT_OK;
    }
    AMGT_CC_CASE(16);
#undef AMGT_CC_CASE
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
    return launch_cc<PREC, MV_SPMM, WPC>(A, val, nvec, a, s, sm_count);
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

int mv_apply_grid(const amgt_bsr *A, int nvec, int sm_count) { return cc_grid<8>(A, nvec, sm_count); }

template <int EPI>
static int launch_apply(int prec, const amgt_bsr *A, int nvec, const MvArgs &a, cudaStream_t s, int sm_count)
{
    const int mode = rm_storage(A, prec);
    const void *val = rm_values(A, mode);
    if (!val) return AMGT_ERR_INVALID;
    switch (mode) {
    case AMGT_DOUBLE: return launch_cc<AMGT_DOUBLE, EPI, 8>(A, val, nvec, a, s, sm_count);
    case AMGT_FLOAT: return launch_cc<AMGT_FLOAT, EPI, 8>(A, val, nvec, a, s, sm_count);
    case AMGT_HALF: return launch_cc<AMGT_HALF, EPI, 8>(A, val, nvec, a, s, sm_count);
    default: return launch_cc<AMGT_BF16, EPI, 8>(A, val, nvec, a, s, sm_count);
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
