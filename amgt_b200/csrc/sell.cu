// Sliced sparse copies of the AMG cycle's operators, and the cycle's
// products on them.
//
// A solve reads each operator of its hierarchy two or three times per
// iteration, and an mBSR block carries 16 values for about 4 stored ones
// (7-point 4.0, 27-point 4.1, HMIS coarse levels 4): the dense-block kernels
// stream 3 to 4 times the bytes the product needs, at the memory's speed.
// The setup therefore keeps, beside the mBSR form, a copy of the larger
// operators with only the stored entries, 16-bit column offsets and the
// narrowest storage that the level's precision reads, and the cycle's
// products (residual, l1-Jacobi, restriction, interpolation, A p) run on it.
// Measured (B200, 7-point 128^3 with BoomerAMG's hierarchy): see the kernel.
#include <algorithm>
#include <type_traits>

#include "sell.cuh"
#include "spmv_common.cuh"

namespace amgt {

// Below this many blocks the dense form's product is launch latency (about
// 3 us at 0.1-8 MB), and a copy would only lengthen the setup.
constexpr int kSellMinBlocks = 65536;
constexpr int kSellThreads = 256;

struct SellDesc {
    const int *ptr, *idx;
    const uint16_t *map;
    int4 *hdr;
    void *sidx;
    int64_t *meas;
    int m, n, brow, nslices, log_t, idx32;
};
// Row lengths -> slice widths, offsets, column bases and the mask of rows that
// have entries.  A warp per slice: the slice's block rows (8 >> log_t of them)
// share the lanes evenly (4 << log_t lanes each); a lane walks every (4 <<
// log_t)-th block of its row and counts the stored entries of the four scalar
// rows.
__global__ void __launch_bounds__(kSellThreads) sell_measure_kernel(const __grid_constant__ SellDesc d)
{
    __shared__ int wsum[kSellThreads / 32], wbase;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lt = d.log_t, gl = 4 << lt;  // lanes per block row
    for (int s0 = blockIdx.x * (kSellThreads / 32); s0 < d.nslices; s0 += gridDim.x * (kSellThreads / 32)) {
        const int s = s0 + warp;
        const bool on = s < d.nslices;
        const int b = s * (8 >> lt) + lane / gl;
        const int k0 = on && b < d.brow ? d.ptr[b] : 0, k1 = on && b < d.brow ? d.ptr[b + 1] : 0;
        // entries of two scalar rows in the halves of one word (at most 65,532
        // each: sell_wanted); unsigned, the upper half uses its top bit
        uint32_t cnt01 = 0, cnt23 = 0;
        int lo = 0x7FFFFFFF, hi = -1;
#pragma unroll 4
        for (int k = k0 + lane % gl; k < k1; k += gl) {
            const uint32_t mp = d.map[k];
            const int c = 4 * d.idx[k];
            if (mp) {
                lo = min(lo, c);
                hi = max(hi, min(c + 3, d.n - 1));
            }
            cnt01 += __popc(mp & 0xFu) | (__popc(mp & 0xF0u) << 16);
            cnt23 += __popc(mp & 0xF00u) | (__popc(mp & 0xF000u) << 16);
        }
        for (int o = 1; o < gl; o <<= 1) {
            cnt01 += __shfl_xor_sync(FULL, cnt01, o);
            cnt23 += __shfl_xor_sync(FULL, cnt23, o);
        }
        // rows with entries: bit i for the slice's row i
        const uint32_t have = ((cnt01 & 0xFFFFu) ? 1u : 0u) | ((cnt01 >> 16) ? 2u : 0u) |
                              ((cnt23 & 0xFFFFu) ? 4u : 0u) | ((cnt23 >> 16) ? 8u : 0u);
        const uint32_t rows = __reduce_or_sync(FULL, have << (4 * (lane / gl)));
        const int len = (int)__reduce_max_sync(FULL, max(max(cnt01 & 0xFFFFu, cnt01 >> 16),
                                                         max(cnt23 & 0xFFFFu, cnt23 >> 16)));
        lo = __reduce_min_sync(FULL, lo);
        hi = __reduce_max_sync(FULL, hi);
        const int w = max(1, (len + (1 << lt) - 1) >> lt);  // the product reads a slice's first step
        // the CTA's slices take consecutive steps from one counter: their
        // place in memory varies from run to run, their sums do not
        if (lane == 0) wsum[warp] = on ? w : 0;
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
            for (int i = 0; i < kSellThreads / 32; ++i) {
                const int v = wsum[i];
                wsum[i] = t;
                t += v;
            }
            wbase = (int)atomicAdd((unsigned long long *)d.meas, (unsigned long long)t);
        }
        __syncthreads();
        if (on && lane == 0) {
            d.hdr[s] = make_int4(wbase + wsum[warp], w, hi < 0 ? 0 : lo, (int)rows);
            if (hi >= 0 && hi - lo > 0xFFFF) atomicMax((unsigned long long *)(d.meas + 1), (unsigned long long)(hi - lo));
            const int last = min(d.m - s * (32 >> lt), 32 >> lt);  // the slice's rows
            if (rows != (last < 32 ? (1u << last) - 1u : FULL)) d.meas[3] = 1;
            if (w > 64) atomicMax((unsigned long long *)(d.meas + 2), (unsigned long long)w);
        }
        __syncthreads();
    }
}

// Entries, for one storage type: a lane per scalar row (the four lanes of a
// block row read the same block; the lanes of a warp write the same step of
// neighbouring rows), its blocks in order, kFillU blocks' columns, bitmaps
// and first values in flight.  The rest of the row is filled with zero values
// at the row's own last column, so that a product reads no x entry that the row
// does not multiply anyway (a slice may hold rows of two systems of a batch,
// and 0 * NaN is NaN); an empty row, which has none, is masked in the product.
// with_idx: write the columns too.  A row that the size pass found shorter
// than it is raises the error word and writes nothing beyond its slice (one
// test per kFillU blocks; a test per entry took 5 % longer).
constexpr int kFillU = 4;

template <typename V>
__global__ void __launch_bounds__(kSellThreads) sell_fill_kernel(const __grid_constant__ SellDesc d,
                                                                const V *__restrict__ src, V *__restrict__ dst,
                                                                int with_idx, int *__restrict__ err)
{
    const int lt = d.log_t, tm = (1 << lt) - 1;
    for (int row = blockIdx.x * kSellThreads + threadIdx.x; row < ((d.m + 31) & ~31); row += gridDim.x * kSellThreads) {
        const int b = row >> 2, q = row & 3;
        const int s = row >> (5 - lt);
        if (s >= d.nslices) continue;
        const int k0 = b < d.brow ? d.ptr[b] : 0, k1 = b < d.brow ? d.ptr[b + 1] : 0;
        // position of the row's entry j: row0 + 32 (j >> lt) + (j & tm)
        const int4 hd = d.hdr[s];
        const long long row0 = 32LL * hd.x + ((row & ((32 >> lt) - 1)) << lt);
        const int w = hd.y << lt, cb = hd.z;
        int *i32 = with_idx && d.idx32 ? static_cast<int *>(d.sidx) + row0 : nullptr;
        unsigned short *i16 = with_idx && !d.idx32 ? static_cast<unsigned short *>(d.sidx) + row0 : nullptr;
        V *vr = dst + row0;
        int j = 0, last = cb;
        auto put = [&](int col, V v) {
            const int e = 32 * (j >> lt) + (j & tm);
            if (i16) i16[e] = (unsigned short)(col - cb);
            else if (i32) i32[e] = col;
            vr[e] = v;
            last = col;
            ++j;
        };
        const V *sq = src + 4 * q;
        for (int k = k0; k < k1; k += kFillU) {
            uint32_t nib[kFillU];
            int col[kFillU];
            V v0[kFillU];
#pragma unroll
            for (int u = 0; u < kFillU; ++u) {
                nib[u] = 0;
                col[u] = 0;
                if (k + u < k1) {
                    nib[u] = (d.map[k + u] >> (4 * q)) & 0xFu;
                    col[u] = 4 * d.idx[k + u];
                }
            }
            int n = j;
#pragma unroll
            for (int u = 0; u < kFillU; ++u) n += __popc(nib[u]);
            if (n > w) {
                raise_error(err, DEV_ERR_CAPACITY);
                break;
            }
#pragma unroll
            for (int u = 0; u < kFillU; ++u)
                if (nib[u]) v0[u] = __ldg(sq + (16LL * (k + u) + __ffs(nib[u]) - 1));
#pragma unroll
            for (int u = 0; u < kFillU; ++u) {
                uint32_t nb = nib[u];
                if (!nb) continue;
                put(col[u] + __ffs(nb) - 1, v0[u]);
                for (nb &= nb - 1; nb; nb &= nb - 1) {
                    const int c = __ffs(nb) - 1;
                    put(col[u] + c, __ldg(sq + (16LL * (k + u) + c)));
                }
            }
        }
        while (j < w) put(last, (V)0);
    }
}

// ---------------------------------------------------------------- products
enum { SEPI_SPMV = 0, SEPI_RESID = 1, SEPI_JACOBI = 2, SEPI_RESTRICT_JACOBI0 = 3, SEPI_DOT = 4 };

struct SellArgs {
    const int4 *hdr;
    const void *idx, *val;
    int m, nslices, log_t;
    double alpha, beta;    // SPMV; alpha: the weight of JACOBI and RESTRICT_JACOBI0
    const double *x;       // multiplied vector (u of RESID / JACOBI / DOT)
    const double *f;       // RESID, JACOBI
    const double *inv_l1;  // JACOBI, RESTRICT_JACOBI0
    double *out;           // result
    double *out2;          // RESTRICT_JACOBI0: w out ./ l1; DOT: partials, one per CTA
};

// Stored value e in its storage type, and widened.
template <int MODE>
struct SellVal {
    using raw_t = unsigned short;
};
template <>
struct SellVal<AMGT_DOUBLE> {
    using raw_t = double;
};
template <>
struct SellVal<AMGT_FLOAT> {
    using raw_t = float;
};
template <>
struct SellVal<kExact32> {
    using raw_t = float;
};
template <int MODE>
__device__ __forceinline__ typename ValTraits<MODE>::acc_t sell_widen(typename SellVal<MODE>::raw_t v)
{
    if constexpr (MODE == AMGT_HALF || MODE == kExact16) return __half2float(__ushort_as_half(v));
    else if constexpr (MODE == AMGT_BF16) return __bfloat162float(__ushort_as_bfloat16(v));
    else return v;
}

// Steps in flight per warp and CTAs per SM.  Measured on the 128^3 7-point
// BoomerAMG hierarchy and a batch of 2D systems: the interpolation's rows (2
// to 4 entries) do best with four steps (fp64 values 13.3 us a pass over the
// first three levels against 18.0 with six; 2D fp16 batch 38 us against 46
// with eight), the operators' (7 and more) with six 8-byte values (20.0 us a
// residual against 21.2 with four) or eight narrower ones (28 us against 29).
template <int MODE, int EPI>
struct SellShape {
    static constexpr bool wide = sizeof(typename SellVal<MODE>::raw_t) == 8;
    static constexpr int steps = EPI == SEPI_SPMV ? 4 : wide ? 6 : 8;
    static constexpr int ctas = EPI == SEPI_SPMV ? (wide ? 5 : 6) : 4;
};

// One warp per slice, a batch of steps at a time: while a batch's x entries
// are gathered (the lanes of a step hold neighbouring rows, whose columns lie
// close together) and added in entry order, the next batch's columns and
// values (of this slice, or of the warp's next one, whose header was read a
// slice earlier) go in flight.  A slice's last batch reads its last step
// again instead of predicating each step off (the predicated form compiled to
// about 340 instructions a slice of seven steps and 36 us a level-0 residual).
// One wave of CTAs, so that every warp walks several slices.
// HOLES (the operator has rows without entries) masks their sums by the bits
// in the slice's header; done for every operator it cost the batch's solve
// 1.3 % (9.43 against 9.54 ms).
//
// Bound by HBM bytes: an entry is 2 + {8, 4, 2} bytes, each vector 8 bytes a
// row.  128^3 7-point, fp64 from exact fp16 storage, residual: 109 MB in 28
// us (3.9 TB/s; the block kernel: 183 MB in 41 us); BoomerAMG's level 1 (1.05
// M rows, 17.6 M entries, 8-byte values): 202 MB in 38 us (5.3 TB/s) against
// 93 us on 593 MB of blocks.
template <int MODE, bool IDX32, int EPI, bool HOLES>
__global__ void __launch_bounds__(kSellThreads, SellShape<MODE, EPI>::ctas)
sell_kernel(const __grid_constant__ SellArgs a)
{
    using acc_t = typename ValTraits<MODE>::acc_t;
    using raw_t = typename SellVal<MODE>::raw_t;
    using idx_t = typename std::conditional<IDX32, int, unsigned short>::type;
    constexpr int U = SellShape<MODE, EPI>::steps;
    __shared__ double sred[kSellThreads / 32];
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * kSellThreads) >> 5;
    const int lt = a.log_t, rps = 32 >> lt;
    const idx_t *idx = static_cast<const idx_t *>(a.idx) + lane;
    const raw_t *val = static_cast<const raw_t *>(a.val) + lane;
    double dot = 0.0;
    int s = (blockIdx.x * kSellThreads + threadIdx.x) >> 5;
    // the setup that wrote the matrix has ended with a synchronisation: its
    // first loads need not wait for the kernels before
    const int4 none = make_int4(0, 1, 0, 0);
    int4 h = s < a.nslices ? __ldg(a.hdr + s) : none, hn = s + nw < a.nslices ? __ldg(a.hdr + s + nw) : none;
    int c[U];   // columns of the batch to gather next
    raw_t v[U];  // values of the batch to add next
    const idx_t *ip = idx + 32LL * h.x;
    const raw_t *vp = val + 32LL * h.x;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        c[u] = __ldcs(ip + 32 * min(u, h.y - 1));
        v[u] = __ldcs(vp + 32 * min(u, h.y - 1));
    }
    grid_dependency_wait();
    for (; s < a.nslices; s += nw) {
        const double *xb = a.x + (IDX32 ? 0 : h.z);
        const int row = s * rps + (lane >> lt);
        const bool mine = (lane & ((1 << lt) - 1)) == 0 && row < a.m;
        double fv = 0.0, uv = 0.0, lv = 0.0;
        if (mine) {
            if constexpr (EPI == SEPI_RESID || EPI == SEPI_JACOBI) fv = a.f[row];
            if constexpr (EPI == SEPI_JACOBI || EPI == SEPI_DOT) uv = a.x[row];
            if constexpr (EPI == SEPI_JACOBI || EPI == SEPI_RESTRICT_JACOBI0) lv = a.inv_l1[row];
            if constexpr (EPI == SEPI_SPMV)
                if (a.beta != 0.0) fv = a.out[row];
        }
        const int4 hnn = s + 2 * nw < a.nslices ? __ldg(a.hdr + s + 2 * nw) : none;
        acc_t sum = 0;
        int rem = h.y;  // steps left, this batch included (warp-uniform)
        do {
            double xv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) xv[u] = __ldg(xb + c[u]);
            // the next batch: of this slice, else of the warp's next one
            const bool more = rem > U;
            const int nrem = more ? rem - U : hn.y;
            ip = more ? ip + 32 * U : idx + 32LL * hn.x;
            vp = more ? vp + 32 * U : val + 32LL * hn.x;
#pragma unroll
            for (int u = 0; u < U; ++u) c[u] = __ldcs(ip + 32 * min(u, nrem - 1));
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (u < rem) sum = fma(sell_widen<MODE>(v[u]), (acc_t)xv[u], sum);
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = __ldcs(vp + 32 * min(u, nrem - 1));
            rem = more ? nrem : 0;
        } while (rem > 0);
        for (int o = 1; o < (1 << lt); o <<= 1) sum += __shfl_xor_sync(FULL, sum, o);
        if (mine) {
            double ax = (double)sum;
            if constexpr (HOLES) ax = (h.w >> (lane >> lt)) & 1 ? ax : 0.0;  // an empty row's slots are not its own
            if constexpr (EPI == SEPI_SPMV) {
                const double t = a.alpha * ax;
                a.out[row] = a.beta == 0.0 ? t : t + a.beta * fv;
            } else if constexpr (EPI == SEPI_RESID) {
                a.out[row] = fv - ax;
            } else if constexpr (EPI == SEPI_JACOBI) {
                a.out[row] = uv + a.alpha * (fv - ax) * lv;
            } else if constexpr (EPI == SEPI_RESTRICT_JACOBI0) {
                a.out[row] = ax;
                a.out2[row] = a.alpha * ax * lv;
            } else {
                a.out[row] = ax;
                dot += uv * ax;
            }
        }
        h = hn;
        hn = hnn;
    }
    if constexpr (EPI == SEPI_DOT) {
        // fixed-order reduction: lanes, then warps (deterministic for a fixed grid)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(FULL, dot, o);
        if (lane == 0) sred[threadIdx.x >> 5] = dot;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int i = 0; i < kSellThreads / 32; ++i) t += sred[i];
            a.out2[blockIdx.x] = t;
        }
    }
}

template <int EPI>
static int launch_sell(const SellMat &S, int mode, SellArgs a, cudaStream_t s, int sm_count)
{
    a.hdr = S.hdr;
    a.idx = S.idx;
    a.val = S.val[sell_storage(mode)];
    a.m = S.m;
    a.nslices = S.nslices;
    a.log_t = S.log_t;
#define AMGT_SELL_CASE(M)                                                                              \
    case M: {                                                                                          \
        const int grid = grid_for(kSellThreads / 32, S.nslices, sm_count, SellShape<M, EPI>::ctas);    \
        if (S.idx32 && S.holes) AMGT_LAUNCH_PDL((sell_kernel<M, true, EPI, true>), grid, kSellThreads, 0, s, a); \
        else if (S.idx32) AMGT_LAUNCH_PDL((sell_kernel<M, true, EPI, false>), grid, kSellThreads, 0, s, a);      \
        else if (S.holes) AMGT_LAUNCH_PDL((sell_kernel<M, false, EPI, true>), grid, kSellThreads, 0, s, a);      \
        else AMGT_LAUNCH_PDL((sell_kernel<M, false, EPI, false>), grid, kSellThreads, 0, s, a);                  \
        return AMGT_OK;                                                                                \
    }
    switch (mode) {
        AMGT_SELL_CASE(AMGT_DOUBLE)
        AMGT_SELL_CASE(AMGT_FLOAT)
        AMGT_SELL_CASE(AMGT_HALF)
        AMGT_SELL_CASE(AMGT_BF16)
        AMGT_SELL_CASE(kExact32)
        AMGT_SELL_CASE(kExact16)
    default: return AMGT_ERR_INVALID;
    }
#undef AMGT_SELL_CASE
}

int sell_storage(int mode)
{
    switch (mode) {
    case AMGT_DOUBLE: return 0;
    case AMGT_FLOAT: case kExact32: return 1;
    case AMGT_HALF: case kExact16: return 2;
    default: return 3;
    }
}

bool sell_has(const SellMat &S, int mode) { return S.hdr && S.val[sell_storage(mode)]; }

bool sell_wanted(const amgt_bsr *A)
{
    // rows of at most 65,535 entries: the passes count them in 16 bits
    return A->blc_num >= kSellMinBlocks && A->row > 0 && A->col > 0 && A->csr_nnz > 0 && A->max_blc_per_row > 0 &&
           A->max_blc_per_row <= 16383;
}

// Lanes per row: one, where that gives every SM 24 warps (neighbouring rows
// in a step keep the gathers of x together), else the fewest that do, with at
// least two entries a lane.
static int pick_log_t(const amgt_bsr *A, int sm_count)
{
    const double avg = (double)A->csr_nnz / A->row;
    int lt = 0;
    while (lt < 3 && (((long long)A->row << lt) / 32) < 24LL * sm_count && avg >= (4 << lt)) ++lt;
    return lt;
}

static SellDesc describe(const SellJob &j)
{
    const amgt_bsr *A = j.A;
    const SellMat &S = *j.out;
    SellDesc d{};
    d.ptr = A->blcPtr;
    d.idx = A->blcIdx;
    d.map = A->blcMap;
    d.hdr = S.hdr;
    d.sidx = S.idx;
    d.m = S.m;
    d.n = S.n;
    d.brow = A->blc_row;
    d.nslices = S.nslices;
    d.log_t = S.log_t;
    d.idx32 = S.idx32 ? 1 : 0;
    return d;
}

int sell_measure(const std::vector<SellJob> &jobs, int64_t *meas, cudaStream_t s, int sm_count)
{
    for (size_t j = 0; j < jobs.size(); ++j) {
        SellMat &S = *jobs[j].out;
        S.m = jobs[j].A->row;
        S.n = jobs[j].A->col;
        S.log_t = pick_log_t(jobs[j].A, sm_count);
        const int rows = 32 >> S.log_t;
        S.nslices = (S.m + rows - 1) / rows;
        if (alloc_n(&S.hdr, (size_t)S.nslices, s)) continue;  // no memory: no copy
        SellDesc d = describe(jobs[j]);
        d.meas = meas + kSellMeas * j;
        AMGT_LAUNCH(sell_measure_kernel, grid_for(kSellThreads / 32, S.nslices, sm_count, 8), kSellThreads, 0, s, d);
    }
    return AMGT_OK;
}

// A long row among short ones is a serial chain on both forms: one warp adds
// its slice step after step (0.45 us a step beyond a warp's ordinary share
// where the copy streams from HBM, 0.15 where half of L2 holds it), lpr lanes
// walk its blocks (2 / lpr us a block).  True when the chain loses more than
// the smaller copy wins in bytes (5 TB/s, 10 from L2).  Measured, us a
// product, copy against blocks: 128 x 128 x 64 7-point with four rows of 135
// entries 70 against 76, of 263 127 against 106, of 1,032 465 against 293
// (without 23 against 46); its next level with the latter 453 against 190;
// 64^3 with rows of 263 43 against 73, of 1,030 151 against 259.
static bool slice_too_long(const SellJob &j, long long steps, long long longest, int sm_count)
{
    const int vbytes = (j.storages & 1u) ? 8 : (j.storages & 2u) ? 4 : 2;  // the widest storage read
    const double bytes = 32.0 * steps * ((j.out->idx32 ? 4 : 2) + vbytes), blocks = (16.0 * vbytes + 6) * j.A->blc_num;
    const bool l2 = bytes < 64e6;
    const double share = (double)steps / (8.0 * SellShape<AMGT_DOUBLE, SEPI_RESID>::ctas * sm_count);
    const double chain = (longest - share) * (l2 ? 0.15 : 0.45) - 2.0 * j.A->max_blc_per_row / spmv_lanes(j.A);
    return longest > 0 && chain > (blocks - bytes) / (l2 ? 10e6 : 5e6);
}

int sell_fill(const std::vector<SellJob> &jobs, const int64_t *meas_host, cudaStream_t s, int sm_count)
{
    DeviceState *st;
    AMGT_TRY(device_state(&st));
    for (size_t j = 0; j < jobs.size(); ++j) {
        SellMat &S = *jobs[j].out;
        if (!S.hdr) continue;
        const long long steps = meas_host[kSellMeas * j], longest = meas_host[kSellMeas * j + 2];
        S.idx32 = meas_host[kSellMeas * j + 1] > 0xFFFF;
        S.holes = meas_host[kSellMeas * j + 3] != 0;
        // blocks of many entries: the copy, 2 or 4 bytes an entry for its column,
        // would be no smaller than the blocks (7-point 80^3 nodes of full 4x4
        // blocks: 105 us a product against 90 at fp64, 81 against 52 at fp16; of 4
        // entries 44 against 91 and 29 against 53); long rows among short ones:
        // the padding would outweigh the blocks' zeros (and 32 steps is the unit
        // of 32-bit offsets), or one warp would walk a slice for longer than the
        // bytes saved win
        const int narrow = (jobs[j].storages & 12u) ? 2 : (jobs[j].storages & 2u) ? 4 : 8;  // the narrowest storage read
        if (32LL * steps * ((S.idx32 ? 4 : 2) + narrow) >= (16LL * narrow + 6) * jobs[j].A->blc_num ||
            32LL * steps > 2LL * jobs[j].A->csr_nnz + 65536 || steps > 0x3FFFFFFF ||
            slice_too_long(jobs[j], steps, longest, sm_count)) {
            sell_free(S, s);
            continue;
        }
        const size_t ne = (size_t)(32 * steps);
        unsigned char *p = nullptr;
        int rc = alloc_n(&p, ne * (S.idx32 ? 4 : 2), s);
        S.idx = p;
        const int width[4] = {8, 4, 2, 2};
        for (int k = 0; k < 4 && !rc; ++k)
            if (jobs[j].storages & (1u << k)) {
                rc = alloc_n(&p, ne * width[k], s);
                S.val[k] = p;
            }
        if (rc) {  // no memory: the products stay on the blocks
            sell_free(S, s);
            continue;
        }
        const SellDesc d = describe(jobs[j]);
        const int grid = grid_for(kSellThreads, S.m, sm_count, 16);
        const amgt_bsr *A = jobs[j].A;
        int with_idx = 1;  // the first storage type's pass writes the columns
        if (S.val[0]) {
            AMGT_LAUNCH(sell_fill_kernel<double>, grid, kSellThreads, 0, s, d, (const double *)A->blcVal,
                        (double *)S.val[0], with_idx, st->err);
            with_idx = 0;
        }
        if (S.val[1]) {
            AMGT_LAUNCH(sell_fill_kernel<float>, grid, kSellThreads, 0, s, d, (const float *)A->blcVal_fp32,
                        (float *)S.val[1], with_idx, st->err);
            with_idx = 0;
        }
        for (int k = 2; k < 4; ++k)
            if (S.val[k]) {
                AMGT_LAUNCH(sell_fill_kernel<unsigned short>, grid, kSellThreads, 0, s, d,
                            (const unsigned short *)(k == 2 ? A->blcVal_fp16 : A->blcVal_bf16),
                            (unsigned short *)S.val[k], with_idx, st->err);
                with_idx = 0;
            }
    }
    return AMGT_OK;
}

void sell_free(SellMat &S, cudaStream_t s)
{
    free_ptr(S.hdr, s);
    free_ptr(S.idx, s);
    for (auto &v : S.val) free_ptr(v, s);
}

int sell_spmv(const SellMat &S, int mode, double alpha, const double *x, double beta, double *y, cudaStream_t s,
              int sm_count)
{
    SellArgs a{};
    a.alpha = alpha;
    a.beta = beta;
    a.x = x;
    a.out = y;
    return launch_sell<SEPI_SPMV>(S, mode, a, s, sm_count);
}

int sell_residual(const SellMat &S, int mode, const double *f, const double *u, double *r, cudaStream_t s,
                  int sm_count)
{
    SellArgs a{};
    a.x = u;
    a.f = f;
    a.out = r;
    return launch_sell<SEPI_RESID>(S, mode, a, s, sm_count);
}

int sell_jacobi(const SellMat &S, int mode, const double *inv_l1, double w, const double *f, const double *u,
                double *u_out, cudaStream_t s, int sm_count)
{
    SellArgs a{};
    a.alpha = w;
    a.x = u;
    a.f = f;
    a.inv_l1 = inv_l1;
    a.out = u_out;
    return launch_sell<SEPI_JACOBI>(S, mode, a, s, sm_count);
}

int sell_restrict_jacobi0(const SellMat &S, int mode, const double *t, double *f, const double *inv_l1, double w,
                          double *u, cudaStream_t s, int sm_count)
{
    SellArgs a{};
    a.alpha = w;
    a.x = t;
    a.inv_l1 = inv_l1;
    a.out = f;
    a.out2 = u;
    return launch_sell<SEPI_RESTRICT_JACOBI0>(S, mode, a, s, sm_count);
}

int sell_dot_grid(const SellMat &S, int sm_count)
{
    return grid_for(kSellThreads / 32, S.nslices, sm_count, SellShape<AMGT_DOUBLE, SEPI_DOT>::ctas);
}

int sell_dot(const SellMat &S, int mode, const double *u, double *out, double *partial, cudaStream_t s, int sm_count)
{
    SellArgs a{};
    a.x = u;
    a.out = out;
    a.out2 = partial;
    return launch_sell<SEPI_DOT>(S, mode, a, s, sm_count);
}

}  // namespace amgt
