// fsb_spmm_common.cuh -- pieces shared by the SpMM kernel files: C-row stores,
// accumulator reset and the merge-path carry fix-up.
#pragma once
#include "fsb_dispatch.cuh"

namespace fsb {

constexpr int kSpmmThreads = 128;

template <class O, class A, int VW>
__device__ __forceinline__ void store_row(O* __restrict__ C, int64_t ldc, int64_t out_row, int64_t c0,
                                          const A (&acc)[VW]) {
    if constexpr (VW > 1 && sizeof(O) * VW == 32) {
        // two 16-byte halves
        constexpr int H = VW / 2;
        vec_t<O, H> lo, hi;
#pragma unroll
        for (int w = 0; w < H; ++w) {
            lo.v[w] = Out<O, A>::cvt(acc[w]);
            hi.v[w] = Out<O, A>::cvt(acc[H + w]);
        }
        st_stream<O, H>(C + out_row * ldc + c0, lo);
        st_stream<O, H>(C + out_row * ldc + c0 + H, hi);
    } else if constexpr (VW > 1 && (sizeof(O) * VW == 16 || sizeof(O) * VW == 8 || sizeof(O) * VW == 4)) {
        vec_t<O, VW> o;
#pragma unroll
        for (int w = 0; w < VW; ++w) o.v[w] = Out<O, A>::cvt(acc[w]);
        st_stream<O, VW>(C + out_row * ldc + c0, o);
    } else {
#pragma unroll
        for (int w = 0; w < VW; ++w) C[out_row * ldc + c0 + w] = Out<O, A>::cvt(acc[w]);
    }
}

template <class A> struct is_comp_acc { static constexpr bool value = false; };
template <> struct is_comp_acc<comp_t> { static constexpr bool value = true; };

template <class A, int VW>
__device__ __forceinline__ void zero_acc(A (&acc)[VW]) {
#pragma unroll
    for (int w = 0; w < VW; ++w) acc[w] = A{};
}

// The first unit of each run carrying the same open row folds the run's carries
// (unit order) and the ending unit's head partial: one warp for all columns,
// or, where the run goes on for kFixupLong units, one warp per 64 columns
// (blockIdx.y).  A long run is one chain of additions per column, bound by the
// latency of its loads: its end is looked for 128 units at a time and 64 bytes
// of carries per lane are loaded ahead; 48 registers, since matrices of short
// runs need the resident warps.  One row over 780 units at 1 / 33 / 128 columns,
// a warp per run with four loads ahead -> this form, us: float32 26 / 36 / 90 ->
// 17 / 23 / 29, float64 35 / 51 / 141 -> 29 / 39 / 60, complex128 44 / 78 / 191 ->
// 44 / 68 / 91.  9600 rows over two units each: as before (float32 and float64
// 6.3 at 33 columns, 8.3 at 128); a warp per 32 columns takes 7 - 8 and 10.4
// there, 64 registers 6.6 and 8.8.
constexpr int kFixupLong = 16;

template <class A, class O, class I, class P>
__global__ void __launch_bounds__(kSpmmThreads, 10)
k_spmm_merge_fixup(const int64_t* __restrict__ carry_row, const A* __restrict__ carry_val,
                   const A* __restrict__ head_val, int64_t n_units, int64_t n_dense, const P* __restrict__ ptr,
                   const I* __restrict__ row_map, O* __restrict__ C, int64_t ldc) {
    constexpr int kAhead = 64 / (int)sizeof(A);
    const int64_t t = (int64_t)blockIdx.x * (kSpmmThreads / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= n_units) return;
    const int64_t r = carry_row[t];
    if (r < 0) return;
    if (t > 0 && carry_row[t - 1] == r) return;
    const bool is_long = t + kFixupLong < n_units && carry_row[t + kFixupLong] == r;
    if (blockIdx.y > 0 && !is_long) return;
    // end of the run of units carrying row r, by ballot (the run is one piece:
    // full ballots, then its end, then none)
    int64_t u_end = t + 1;
    unsigned in = 0xffffffffu;
    while (in == 0xffffffffu) {
        bool same[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t u = u_end + i * 32 + lane;
            same[i] = u < n_units && carry_row[u] == r;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            in = __ballot_sync(0xffffffffu, same[i]);
            u_end += __popc(in);
        }
    }
    const int64_t out_row = row_map ? idx(row_map[idx(ptr[r])]) : r;
    const int64_t step = is_long ? (int64_t)gridDim.y * 32 : 32;
    for (int64_t c = (int64_t)blockIdx.y * 32 + lane; c < n_dense; c += step) {
        // loads ahead, adds in unit order (deterministic)
        A sum = carry_val[t * n_dense + c];
        int64_t u = t + 1;
        for (; u + kAhead <= u_end; u += kAhead) {
            A a[kAhead];
#pragma unroll
            for (int i = 0; i < kAhead; ++i) a[i] = carry_val[(u + i) * n_dense + c];
#pragma unroll
            for (int i = 0; i < kAhead; ++i) sum = acc_add(sum, a[i]);
        }
        for (; u < u_end; ++u) sum = acc_add(sum, carry_val[u * n_dense + c]);
        if (u_end < n_units) sum = acc_add(sum, head_val[u_end * n_dense + c]);
        C[out_row * ldc + c] = Out<O, A>::cvt(sum);
    }
}

// Grid of k_spmm_merge_fixup.
inline dim3 fixup_grid(int64_t n_units, int64_t n_dense) {
    const int64_t groups = ceil_div(n_dense, (int64_t)64);
    return dim3((unsigned)ceil_div(n_units, (int64_t)(kSpmmThreads / 32)), (unsigned)(groups < 65535 ? groups : 65535));
}

// FSB_ALGO_GATHER launch (fsb_spmm_gather.cu), dtype dispatch included.
int spmm_gather_dispatch(const fsb_csr* A, const void* B, int64_t ldb, int64_t n_dense, void* C, int64_t ldc,
                         int out_dtype, int acc_mode, const fsb_plan* plan, void* workspace, int64_t workspace_bytes,
                         cudaStream_t st);

}  // namespace fsb
