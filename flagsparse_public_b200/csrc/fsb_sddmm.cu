// fsb_sddmm.cu -- sampled dense-dense matrix multiplication on a CSR pattern:
//     out[p] = alpha * dot(x[row(p)], y[col(p)]) + beta * data[p]
// for every stored position p (FlagSparse's flagsparse_sddmm_csr,
// sddmm_csr.py:350-422, kernel _sddmm_csr_real_kernel :108-152).
//
// A sub-group of LPN lanes computes kSddmmU positions at a time (consecutive
// ones, in sub-groups of one or two lanes ones a warp's width apart), each lane covering VW consecutive elements of K per step (16-byte vectors
// where x and y allow).  The positions' indices come as vector loads, their y
// rows are loaded back to back (random gathers, latency bound), and x is
// loaded once where the positions of every sub-group lie in one row each.  The
// dot products are reduced together: each halving step exchanges half of the
// sums (5 shuffles for 4 products over 16 lanes where one reduction each took
// 16), and the lanes that end with them store neighbouring results.
// float32 accumulates in float32, float64 in float64, as FlagSparse's baseline
// kernel does.
#include "fsb_dispatch.cuh"

namespace fsb {

constexpr int kSddmmThreads = 256;
constexpr int kSddmmU = 4;  // positions per sub-group and batch

// The indices of a batch from position p0 on (clamped to the last of n; 16-byte loads
// where they are aligned and all inside).
template <class I>
__device__ __forceinline__ void load_indices(const I* __restrict__ a, int64_t p0, int64_t n, bool vec_ok,
                                             I (&out)[kSddmmU]) {
    if (vec_ok && p0 + kSddmmU <= n) {
        constexpr int M = 16 / (int)sizeof(I) < kSddmmU ? 16 / (int)sizeof(I) : kSddmmU;
#pragma unroll
        for (int i = 0; i < kSddmmU; i += M) {
            const vec_t<I, M> t = ld_stream<I, M>(a + p0 + i);
#pragma unroll
            for (int j = 0; j < M; ++j) out[i + j] = t.v[j];
        }
    } else {
#pragma unroll
        for (int u = 0; u < kSddmmU; ++u) out[u] = a[p0 + u < n ? p0 + u : n - 1];
    }
}

// What bounds it: y rows in flight per SM.  Power-law pattern, 3.1 M
// positions, before (a reduction per position, x loaded per position) -> now:
// float32 K = 64 144 -> 119 us (its gathers alone: 68); 3.2 M positions,
// float32 K = 33 (single elements) 357 -> 265, K = 128 303 -> 255, K = 200 749 -> 503;
// float64 K = 64 435 -> 283, K = 200 1185 -> 811.  Eight positions per batch: 151 us
// at 2 CTAs (128 registers), 186 at 3 (spills); 3 or 5 CTAs with four: 166 and
// 136 (all three with the loop over K that one step has since replaced below
// 32 lanes).
// Sub-groups of one or two lanes (K up to two vectors) take positions NPAR
// apart: with neighbouring ones per lane every index load and store of the
// warp spreads over four times the lines (3 M positions, kernel us, a
// reduction per position / neighbouring / apart: float64 K = 1 15.6 / 24 /
// 15.7, float32 K = 4 16.6 / 18 / 16.1, K = 2 16.4 / 17.1 / 14.5).
// Below 32 lanes the lanes cover K in one step: without the loop the compiler
// spends no registers on unrolling it (float32 K = 64 114 -> 101 us on even
// rows, K = 2 21.6 -> 14.5).
template <class V, class A, class I, int VW, int LPN_LOG2>
__global__ void __launch_bounds__(kSddmmThreads, 4)
k_sddmm(const I* __restrict__ col, const int32_t* __restrict__ row_ids, int64_t nnz, const V* __restrict__ x,
        int64_t ldx, const V* __restrict__ y, int64_t ldy, int64_t k, const V* __restrict__ data,
        V* __restrict__ out, A alpha, A beta, int vec_ok) {
    constexpr int LPN = 1 << LPN_LOG2;
    constexpr int NPAR = 32 >> LPN_LOG2;
    constexpr int U = kSddmmU;
    constexpr int HALVINGS = LPN_LOG2 < 2 ? LPN_LOG2 : 2;  // log2 U at most
    constexpr int LEFT = U >> HALVINGS;  // results per storing lane
    constexpr bool kApart = LPN_LOG2 <= 1;
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int sub = lane >> LPN_LOG2, cl = lane & (LPN - 1);
    const int64_t warp = ((int64_t)blockIdx.x * kSddmmThreads + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * kSddmmThreads) >> 5;
    for (int64_t base = warp * (NPAR * U); base < nnz; base += n_warps * (NPAR * U)) {
        // the sub-group's positions: U consecutive ones, or (kApart) NPAR apart
        const int64_t p0 = base + (kApart ? sub : sub * U);
        I c[U];
        int32_t r[U];
        bool one_row = false;
        if constexpr (kApart) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int64_t p = p0 + u * NPAR < nnz ? p0 + u * NPAR : nnz - 1;
                c[u] = col[p];
                r[u] = row_ids[p];
            }
        } else {
            load_indices<I>(col, p0, nnz, vec_ok, c);
            load_indices<int32_t>(row_ids, p0, nnz, vec_ok, r);
            bool same = true;
#pragma unroll
            for (int u = 1; u < U; ++u) same = same && r[u] == r[0];
            one_row = __all_sync(full, same);
        }
        A acc[U];
#pragma unroll
        for (int u = 0; u < U; ++u) acc[u] = A(0);
        auto step = [&](int64_t kk) {
            vec_t<V, VW> yv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) yv[u] = ld_ro<V, VW>(y + idx(c[u]) * ldy + kk);
            if (one_row) {
                const vec_t<V, VW> xv = ld_ro<V, VW>(x + (int64_t)r[0] * ldx + kk);
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int w = 0; w < VW; ++w) acc[u] = fma((A)xv.v[w], (A)yv[u].v[w], acc[u]);
            } else {
                vec_t<V, VW> xv[U];
#pragma unroll
                for (int u = 0; u < U; ++u) xv[u] = ld_ro<V, VW>(x + (int64_t)r[u] * ldx + kk);
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int w = 0; w < VW; ++w) acc[u] = fma((A)xv[u].v[w], (A)yv[u].v[w], acc[u]);
            }
        };
        if constexpr (LPN_LOG2 < 5) {  // the lanes cover k in one step
            if (cl * VW < k) step(cl * VW);
        } else {
            for (int64_t kk = (int64_t)cl * VW; kk < k; kk += (int64_t)LPN * VW) step(kk);
        }
        // halving steps: the upper half of the lanes keeps the upper half of
        // the sums, the lower half the lower
        int first = 0;
#pragma unroll
        for (int h = 0; h < HALVINGS; ++h) {
            const int o = LPN >> (h + 1), n = U >> (h + 1);
            const bool upper = (cl & o) != 0;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const A send = upper ? acc[i] : acc[i + n];
                const A keep = upper ? acc[i + n] : acc[i];
                acc[i] = keep + __shfl_xor_sync(full, send, o);
            }
            if (upper) first += n;
        }
#pragma unroll
        for (int o = LPN >> (HALVINGS + 1); o > 0; o >>= 1) acc[0] += __shfl_xor_sync(full, acc[0], o);
        if ((cl & ((LPN >> HALVINGS) - 1)) == 0) {
#pragma unroll
            for (int i = 0; i < LEFT; ++i) {
                const int64_t p = p0 + (first + i) * (kApart ? NPAR : 1);
                if (p < nnz) {
                    A v = alpha * acc[i];
                    if (data) v += (A)data[p] * beta;
                    out[p] = (V)v;
                }
            }
        }
    }
}

template <class V, class A, class I, int VW>
int launch_sddmm_vw(int lpn_log2, const I* col, const int32_t* rows, int64_t nnz, const V* x, int64_t ldx, const V* y,
                    int64_t ldy, int64_t k, const V* data, V* out, A alpha, A beta, cudaStream_t st) {
    const int npar = 32 >> lpn_log2;
    const int vec_ok = aligned16(col) && aligned16(rows);
    const int64_t warps = ceil_div(nnz, (int64_t)npar * kSddmmU);
    int64_t blocks = ceil_div(warps, (int64_t)(kSddmmThreads / 32));
    if (blocks > 148 * 64) blocks = 148 * 64;  // grid-stride beyond ~64 waves of CTAs
#define FSB_SDDMM(L)                                                                                           \
    case L:                                                                                                    \
        k_sddmm<V, A, I, VW, L><<<(unsigned)blocks, kSddmmThreads, 0, st>>>(col, rows, nnz, x, ldx, y, ldy, k, \
                                                                             data, out, alpha, beta, vec_ok);  \
        break;
    switch (lpn_log2) {
        FSB_SDDMM(0)
        FSB_SDDMM(1)
        FSB_SDDMM(2)
        FSB_SDDMM(3)
        FSB_SDDMM(4)
        FSB_SDDMM(5)
        default:
            fsb_host::set_error("fsb_sddmm_csr: bad lane count");
            return FSB_ERR_INVALID;
    }
#undef FSB_SDDMM
    return fsb_host::check_launch("k_sddmm");
}

}  // namespace fsb

extern "C" int fsb_sddmm_csr(const void* col_idx, int index_dtype, const int32_t* row_ids, int64_t nnz, int64_t n_rows,
                             int64_t n_cols, const void* x, int64_t ldx, const void* y, int64_t ldy, int64_t k,
                             const void* data, void* out, int value_dtype, double alpha, double beta, void* stream) {
    if (nnz < 0 || k < 0 || n_rows < 0 || n_cols < 0 || ldx < k || ldy < k) {
        fsb_host::set_error("fsb_sddmm_csr: bad sizes");
        return FSB_ERR_INVALID;
    }
    if (nnz == 0) return FSB_OK;
    if (!col_idx || !row_ids || !out || (k > 0 && (!x || !y))) {
        fsb_host::set_error("fsb_sddmm_csr: null pointer");
        return FSB_ERR_INVALID;
    }
    if (value_dtype != FSB_F32 && value_dtype != FSB_F64) {
        fsb_host::set_error("fsb_sddmm_csr: values must be float32 or float64");
        return FSB_ERR_UNSUPPORTED;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return fsb::dispatch_idx(index_dtype, [&](auto ti) -> int {
        using I = typename decltype(ti)::type;
        auto run = [&](auto tv) -> int {
            using V = typename decltype(tv)::type;
            using A = V;
            constexpr int kVW = 16 / (int)sizeof(V);
            const V* xv = static_cast<const V*>(x);
            const V* yv = static_cast<const V*>(y);
            const bool vec = k % kVW == 0 && ldx % kVW == 0 && ldy % kVW == 0 && ((uintptr_t)xv) % 16 == 0 &&
                             ((uintptr_t)yv) % 16 == 0;
            const int vw = vec ? kVW : 1;
            int lpn_log2 = 0;
            while ((int64_t)(vw << lpn_log2) < k && lpn_log2 < 5) ++lpn_log2;
            const I* col = static_cast<const I*>(col_idx);
            const V* d = static_cast<const V*>(data);
            V* o = static_cast<V*>(out);
            if (vec)
                return fsb::launch_sddmm_vw<V, A, I, kVW>(lpn_log2, col, row_ids, nnz, xv, ldx, yv, ldy, k, d, o,
                                                          (A)alpha, (A)beta, st);
            return fsb::launch_sddmm_vw<V, A, I, 1>(lpn_log2, col, row_ids, nnz, xv, ldx, yv, ldy, k, d, o, (A)alpha,
                                                    (A)beta, st);
        };
        if (value_dtype == FSB_F32) return run(fsb::tag<float>{});
        return run(fsb::tag<double>{});
    });
}
