// fsb_spmv.cu -- CSR SpMV on sm_100a: y = A x.
//
// Two kernel families, chosen per matrix by the host plan:
//   * k_spmv_rows  : a group of 2^k lanes per row (k = 0..5), 128-bit streaming
//                    loads of values and column indices, read-only cached
//                    gathers of x, xor-butterfly reduction inside the group.
//                    Up to 16 lanes take the aligned chunks that cover the row,
//                    the elements outside it masked; a whole warp per row takes
//                    the aligned body and single elements at its two ends.
//   * k_spmv_merge : merge-path units of equal (row ends + nonzeros) whatever
//                    the row-length skew (Merrill & Garland, SC'16), a warp per
//                    unit.  Each lane sums 8 consecutive nonzeros in order and
//                    stores the rows that lie inside them; one segmented warp
//                    scan per 256 nonzeros joins the lanes' open sums.  Rows
//                    that cross units are finished by k_spmv_merge_fixup.
//
// FlagSparse computes the same products in _spmv_csr_real_kernel
// (spmv_csr.py:158-184), _spmv_csr_complex_kernel (:187-219), the CSR-vector
// bucket kernels (:225-343) and the COO row-run kernels (spmv_coo.py:131-226).
#include <algorithm>
#include <cstring>
#include <cmath>
#include <mutex>

#include "fsb_partition.cuh"

namespace fsb {

constexpr int kRowsThreads = 256;
constexpr int kMergeThreads = 128;
constexpr int kMergeMaxItemsPerThread = 8;
constexpr int kMergeMaxTile = kMergeThreads * kMergeMaxItemsPerThread;
// FSB_PLAN_OVERLAP_LAUNCH applies to grids of at most one wave at four
// resident CTAs per SM (a waiting successor then takes no slot a later wave
// of this kernel would need)
constexpr int64_t kOverlapMaxBlocks = 148 * 4;

// The nonzeros [kb, kb + VEC) of the streams, kb a multiple of VEC: 16-byte
// loads where the whole vector lies inside the arrays (the last one of the
// matrix may not), single elements otherwise.
template <class V, class I, int VEC>
__device__ __forceinline__ void load_chunk(const V* __restrict__ val, const I* __restrict__ col, int64_t kb,
                                           int64_t nnz, vec_t<V, VEC>& vv, vec_t<I, VEC>& cc) {
    if (kb + VEC <= nnz) {
        vv = ld_stream<V, VEC>(val + kb);
        cc = ld_stream<I, VEC>(col + kb);
    } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            vv.v[j] = vzero<V>();
            cc.v[j] = 0;
            if (kb + j < nnz) {
                vv.v[j] = ld_stream1(val + kb + j);
                cc.v[j] = ld_stream1(col + kb + j);
            }
        }
    }
}

// Partial sum of row nonzeros [s, e) handled by `lane` of a T-lane group: the
// aligned VEC-wide chunks covering the row, the elements outside it skipped.
// One loop and one chain of loads per row (chunk, x) where a scalar head, an
// aligned body and a scalar tail made three; two chunks per lane in flight.
// What bounds it is the loads of x (about one line per cycle and SM) and, for
// short rows, the chain of loads per row: few lanes per row with a whole
// chunk each beat many (see spmv_row_lanes).
template <class V, class A, class I>
__device__ __forceinline__ A row_partial(const V* __restrict__ val, const I* __restrict__ col,
                                         const V* __restrict__ x, int64_t s, int64_t e, int64_t nnz,
                                         int lane, int T, bool vec_ok) {
    constexpr int VV = VecWidth<V>::value;
    constexpr int VI = VecWidth<I>::value;
    constexpr int VEC = VV < VI ? VV : VI;
    A acc = Acc<V, A>::zero();
    if (VEC > 1 && vec_ok) {
        for (int64_t kb = (s & ~(int64_t)(VEC - 1)) + (int64_t)lane * VEC; kb < e; kb += 2 * (int64_t)T * VEC) {
            const int64_t k2 = kb + (int64_t)T * VEC;
            const bool two = k2 < e;
            vec_t<V, VEC> v0, v1;
            vec_t<I, VEC> c0, c1;
            V x0[VEC], x1[VEC];
            load_chunk<V, I, VEC>(val, col, kb, nnz, v0, c0);
            if (two) load_chunk<V, I, VEC>(val, col, k2, nnz, v1, c1);
#pragma unroll
            for (int j = 0; j < VEC; ++j)
                if (kb + j >= s && kb + j < e) x0[j] = ld_ro1(x + idx(c0.v[j]));
            if (two) {
#pragma unroll
                for (int j = 0; j < VEC; ++j)
                    if (k2 + j < e) x1[j] = ld_ro1(x + idx(c1.v[j]));
            }
            // four short chains, then their sum: a lane with several chunks
            // rounds no more often than many lanes with one each
            A t[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) t[q] = Acc<V, A>::zero();
#pragma unroll
            for (int j = 0; j < VEC; ++j)
                if (kb + j >= s && kb + j < e) t[j & 1] = Acc<V, A>::fma(v0.v[j], x0[j], t[j & 1]);
            if (two) {
#pragma unroll
                for (int j = 0; j < VEC; ++j)
                    if (k2 + j < e) t[2 + (j & 1)] = Acc<V, A>::fma(v1.v[j], x1[j], t[2 + (j & 1)]);
            }
            acc = acc_add(acc, acc_add(acc_add(t[0], t[1]), acc_add(t[2], t[3])));
        }
    } else {
#pragma unroll 4
        for (int64_t k = s + lane; k < e; k += T)
            acc = Acc<V, A>::fma(ld_stream1(val + k), ld_ro1(x + idx(ld_stream1(col + k))), acc);
    }
    return acc;
}

// The same for a whole warp per row (32 lanes), which rows of hundreds of
// nonzeros take: scalar head, aligned body, scalar tail. With 128 nonzeros per
// step the masked chunks above cost more than the two extra loops, and fewer
// registers leave more warps to hide the loads (400000 banded rows, one in a
// hundred of 8192 nonzeros: float32 263 us here, 273 with the chunks, float64
// 355 and 451, bfloat16 232 and 304).
template <class V, class A, class I>
__device__ __forceinline__ A row_partial_wide(const V* __restrict__ val, const I* __restrict__ col,
                                              const V* __restrict__ x, int64_t s, int64_t e,
                                              int lane, int T, bool vec_ok) {
    constexpr int VV = VecWidth<V>::value;
    constexpr int VI = VecWidth<I>::value;
    constexpr int VEC = VV < VI ? VV : VI;
    A acc = Acc<V, A>::zero();
    if (VEC > 1 && vec_ok) {
        int64_t a0 = (s + VEC - 1) & ~(int64_t)(VEC - 1);
        if (a0 > e) a0 = e;
        int64_t a1 = e & ~(int64_t)(VEC - 1);
        if (a1 < a0) a1 = a0;
        for (int64_t k = s + lane; k < a0; k += T)
            acc = Acc<V, A>::fma(ld_stream1(val + k), ld_ro1(x + idx(ld_stream1(col + k))), acc);
#pragma unroll 2
        for (int64_t kb = a0 + (int64_t)lane * VEC; kb < a1; kb += (int64_t)T * VEC) {
            vec_t<V, VEC> vv = ld_stream<V, VEC>(val + kb);
            vec_t<I, VEC> cc = ld_stream<I, VEC>(col + kb);
            V xv[VEC];
#pragma unroll
            for (int j = 0; j < VEC; ++j) xv[j] = ld_ro1(x + idx(cc.v[j]));
#pragma unroll
            for (int j = 0; j < VEC; ++j) acc = Acc<V, A>::fma(vv.v[j], xv[j], acc);
        }
        for (int64_t k = a1 + lane; k < e; k += T)
            acc = Acc<V, A>::fma(ld_stream1(val + k), ld_ro1(x + idx(ld_stream1(col + k))), acc);
    } else {
#pragma unroll 4
        for (int64_t k = s + lane; k < e; k += T)
            acc = Acc<V, A>::fma(ld_stream1(val + k), ld_ro1(x + idx(ld_stream1(col + k))), acc);
    }
    return acc;
}

template <class A> struct is_comp { static constexpr bool value = false; };
template <> struct is_comp<comp_t> { static constexpr bool value = true; };

// WIDE: 32 lanes per row (lanes_log2 = 5).
template <class V, class A, class O, class I, class P, bool WIDE>
__global__ void __launch_bounds__(kRowsThreads)
k_spmv_rows(const V* __restrict__ val, const I* __restrict__ col, const P* __restrict__ ptr,
            const I* __restrict__ row_map, const V* __restrict__ x, O* __restrict__ y,
            int64_t n_rows, int64_t nnz, int64_t row_cap, int64_t comp_threshold, int lanes_log2, int vec_ok,
            int overlap) {
    // programmatic dependent launch: wait until the previous kernel on the
    // stream has completed and its writes are visible -- nothing is read
    // before -- and let the next launch start once this CTA's rows are done
    if (overlap) asm volatile("griddepcontrol.wait;" ::: "memory");
    const int T = 1 << lanes_log2;
    const int wl = threadIdx.x & 31;
    const int lane = wl & (T - 1);
    const unsigned mask = segment_mask(wl, T);
    const int64_t stride = ((int64_t)gridDim.x * blockDim.x) >> lanes_log2;
    for (int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> lanes_log2; row < n_rows;
         row += stride) {
        const int64_t s = idx(ptr[row]);
        int64_t e = idx(ptr[row + 1]);
        if (row_cap > 0 && e - s > row_cap) e = s + row_cap;
        auto partial = [&](auto ta) {
            using B = typename decltype(ta)::type;
            if constexpr (WIDE) return row_partial_wide<V, B, I>(val, col, x, s, e, lane, T, vec_ok);
            else return row_partial<V, B, I>(val, col, x, s, e, nnz, lane, T, vec_ok);
        };
        A acc;
        if constexpr (is_comp<A>::value) {
            if (e - s > comp_threshold) {
                acc = partial(tag<comp_t>{});
            } else {
                acc = comp_t{partial(tag<float>{}), 0.f};
            }
        } else {
            acc = partial(tag<A>{});
        }
        acc = segment_reduce(mask, acc, 1, T);
        if (lane == 0) {
            const int64_t out_row = row_map ? idx(row_map[s]) : row;
            y[out_row] = Out<O, A>::cvt(acc);
        }
    }
    if (overlap) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------- merge path ----
// unit_coords[2u], [2u+1] = (rows ended, nonzeros consumed) at the start of unit u.
// Scratch per unit: carry_row (row still open at the unit end, -1 if none),
// carry_val (its partial), head_val (partial of the unit's first finished row
// when that row began in an earlier unit).
//
// What bounds it: the random loads of x.  Each lane's load of x is its own
// line, and an SM takes about one line per cycle: 24 M nonzeros cost 84 us on
// 148 SMs.  A CTA per 512- or 1024-item tile (products in shared memory, a
// binary search and a serial walk per thread, two barriers) kept loads in
// flight a third of the time; with a warp per unit nothing waits for other
// warps.  Zipf rows, 24 M nonzeros over 1.5 M rows: float64 354 -> 146 us,
// float32 137 -> 122, float32 with float64 sums 268 -> 125; 0.8 M rows of
// 40 (12 M nonzeros, skewed): warp-per-row groups 230, this form 62.  Loading
// the next chunk's columns and row offsets a chunk ahead: 150 us (float64).
// 8 resident CTAs (64 registers) for values below 8 bytes, 6 (80) else: 173 us
// with 8 for float64.

// N consecutive elements from an address that is a multiple of 16 bytes (or of
// the N elements where those are fewer bytes), in streaming vector loads.
template <class T, int N>
__device__ __forceinline__ void load_group(const T* p, T (&out)[N]) {
    constexpr int M = (int)sizeof(T) * N <= 16 ? N : 16 / (int)sizeof(T);
#pragma unroll
    for (int i = 0; i < N; i += M) {
        const vec_t<T, M> t = ld_stream<T, M>(p + i);
#pragma unroll
        for (int j = 0; j < M; ++j) out[i + j] = t.v[j];
    }
}

template <class V, class A, class O, class I, class P>
__global__ void __launch_bounds__(kMergeThreads, sizeof(V) >= 8 ? 6 : 8)
k_spmv_merge(const V* __restrict__ val, const I* __restrict__ col, const P* __restrict__ ptr,
             const I* __restrict__ row_map, const V* __restrict__ x, O* __restrict__ y,
             int64_t n_rows, int64_t nnz, int vec_ok, const int64_t* __restrict__ coords, int64_t n_units,
             int64_t* __restrict__ carry_row, A* __restrict__ carry_val, A* __restrict__ head_val) {
    constexpr int E = sizeof(V) <= 8 ? 8 : 4;  // nonzeros per lane and chunk
    constexpr int CH = 32 * E;
    constexpr int kWarps = kMergeThreads / 32;
    constexpr unsigned full = 0xffffffffu;
    constexpr unsigned kAll = (1u << E) - 1u;
    __shared__ int sm_row[kWarps][CH];  // number of the row that starts at a nonzero (where the flag is set)
    __shared__ __align__(8) unsigned char sm_flag[kWarps][CH];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t unit = (int64_t)blockIdx.x * kWarps + warp;
    if (unit >= n_units) return;
    int* s_row = sm_row[warp];
    unsigned char* s_flag = sm_flag[warp];
    // rows are numbered from 1 at the unit's first row, nonzeros from 0 at k0
    const int64_t r0 = coords[2 * unit], k0 = coords[2 * unit + 1];
    const int n_ends = (int)(coords[2 * unit + 2] - r0);  // rows ending in the unit
    const int nk = (int)(coords[2 * unit + 3] - k0);
    const int n_rel = n_ends + (r0 + n_ends < n_rows ? 1 : 0);
    // start of row i + 1, clamped to [-1, nk + 1]
    auto start_of = [&](int i) -> int {
        const int64_t s = idx(ptr[r0 + i]) - k0;
        return s < 0 ? -1 : (s > nk ? nk + 1 : (int)s);
    };
    const bool continued = n_rel > 0 && start_of(0) < 0;
    auto put = [&](int rel, A v) {
        if (rel == 1 && continued) {
            head_val[unit] = v;
        } else {
            const int64_t r = r0 + (rel - 1);
            y[row_map ? idx(row_map[idx(ptr[r])]) : r] = Out<O, A>::cvt(v);
        }
    };
    // Chunks start at multiples of E in the arrays (aligned vector loads); the
    // first one reaches `lead` nonzeros before the unit.
    const int lead = (int)(k0 & (E - 1));
    int rb = 0;                            // rows whose start has been passed
    int open_row = continued ? 1 : 0;      // row open before the chunk, 0: none
    A open_acc = Acc<V, A>::zero();        // its sum so far
    auto valid_of = [&](int g) -> unsigned {  // the lane's nonzeros g .. g + E - 1 that are the unit's
        const int lo = g < 0 ? -g : 0, hi = nk - g < E ? nk - g : E;
        return hi > lo ? (kAll >> (E - hi)) & (kAll << lo) : 0u;
    };
    auto load = [&](auto* base, int g, unsigned valid, auto& out) {
        if (vec_ok && valid && k0 + g + E <= nnz) {
            load_group(base + k0 + g, out);
        } else {
#pragma unroll
            for (int u = 0; u < E; ++u)
                if ((valid >> u) & 1u) out[u] = ld_stream1(base + k0 + g + u);
        }
    };
    for (int kc = -lead;; kc += CH) {
        const bool last = kc + CH >= nk;
        const int g = kc + lane * E;  // the lane's first nonzero
        const unsigned valid = valid_of(g);
        V v[E];
        I c[E];
        load(val, g, valid, v);
        load(col, g, valid, c);
        if constexpr (E == 8) *reinterpret_cast<uint2*>(s_flag + lane * E) = make_uint2(0u, 0u);
        else *reinterpret_cast<uint32_t*>(s_flag + lane * E) = 0u;
        __syncwarp();
        const int end = last ? nk : kc + CH;
        for (;;) {
            const int row = rb + lane;
            const bool in = row < n_rel;
            const int s = in ? start_of(row) : 0, e = in ? start_of(row + 1) : 0;
            const bool take = in && (s < end || (last && row < n_ends));
            if (take && e > s && s >= (kc < 0 ? 0 : kc) && s < end) {
                s_row[s - kc] = row + 1;
                s_flag[s - kc] = 1;
            }
            if (take && e == s && row < n_ends) {  // an empty row
                const int64_t r = r0 + row;
                y[row_map ? idx(row_map[idx(ptr[r])]) : r] = Out<O, A>::cvt(Acc<V, A>::zero());
            }
            const int cnt = __popc(__ballot_sync(full, take));
            rb += cnt;
            if (cnt < 32) break;
        }
        V xv[E];
        const bool whole = __all_sync(full, valid == kAll);
#pragma unroll
        for (int u = 0; u < E; ++u)
            if (whole || ((valid >> u) & 1u)) xv[u] = ld_ro1(x + idx(c[u]));
        __syncwarp();
        // the lane's nonzeros in order; a flag ends the row before it
        uint32_t fl[E / 4];
#pragma unroll
        for (int i = 0; i < E / 4; ++i) fl[i] = reinterpret_cast<const uint32_t*>(s_flag + lane * E)[i];
        A acc = Acc<V, A>::zero(), head = Acc<V, A>::zero();
        int rcur = 0;
        bool broke = false;
        uint32_t any_flag = fl[0];
        if constexpr (E == 8) any_flag |= fl[1];
        if (any_flag == 0u) {
            // no row starts here: pairs, then their tree (a long row's sum
            // rounds as often as if many lanes shared it)
            A t[E / 2];
#pragma unroll
            for (int i = 0; i < E / 2; ++i) t[i] = Acc<V, A>::zero();
#pragma unroll
            for (int u = 0; u < E; ++u)
                if (whole || ((valid >> u) & 1u)) t[u / 2] = Acc<V, A>::fma(v[u], xv[u], t[u / 2]);
#pragma unroll
            for (int n = E / 2; n > 1; n /= 2)
#pragma unroll
                for (int i = 0; i < n / 2; ++i) t[i] = acc_add(t[2 * i], t[2 * i + 1]);
            acc = t[0];
        } else {
#pragma unroll
            for (int u = 0; u < E; ++u) {
                if (fl[u / 4] & (1u << (8 * (u % 4)))) {
                    if (broke) put(rcur, acc);
                    else head = acc;
                    broke = true;
                    rcur = s_row[lane * E + u];
                    acc = Acc<V, A>::zero();
                }
                if (whole || ((valid >> u) & 1u)) acc = Acc<V, A>::fma(v[u], xv[u], acc);
            }
        }
        // lanes in order: the open row's sum enters at lane 0, each lane's tail
        // passes on to the lanes up to (and into) the next one holding a break
        if (lane == 0) {
            if (broke) head = acc_add(open_acc, head);
            else acc = acc_add(open_acc, acc);
        }
        const unsigned breaks = __ballot_sync(full, broke);
        const unsigned upto = breaks & (0xffffffffu >> (31 - lane));
        const int seg = upto ? 31 - __clz(upto) : 0;  // the lane whose tail the row began in (lane 0: open_row)
        const int from = __shfl_sync(full, rcur, seg);
        const int row_t = upto ? from : open_row;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const A up = shfl_up(full, acc, o);
            if (lane - o >= seg) acc = acc_add(up, acc);
        }
        const A in = shfl_up(full, acc, 1);
        const int in_row = __shfl_up_sync(full, row_t, 1);
        if (broke) {
            const A total = lane > 0 ? acc_add(in, head) : head;
            const int rel = lane > 0 ? in_row : open_row;
            if (rel > 0) put(rel, total);
        }
        open_acc = shfl_idx(full, acc, 31, 32);
        open_row = __shfl_sync(full, row_t, 31);
        __syncwarp();  // flags and rows are overwritten by the next chunk
        if (last) break;
    }
    if (lane == 0) {
        bool open = false;
        if (nk > 0 && n_rel > n_ends) {
            const int s1 = start_of(n_ends);
            open = nk > (s1 > 0 ? s1 : 0);
        }
        // (a continued row without a nonzero here ends with an empty head partial)
        if (open) carry_val[unit] = open_acc;
        else if (open_row > 0) put(open_row, open_acc);
        carry_row[unit] = open ? r0 + n_ends : -1;
    }
}

// One lane per unit: the first unit of each run of units carrying the same open
// row sums the run's carries, adds the partial held by the unit where the row
// ends and writes the row once.  A run of more than kFixupLaneRun further units
// (a row of many units' nonzeros) is summed by the whole warp: every lane takes
// each 32nd carry, four loads of each array in flight, then the lanes' sums
// meet in a fixed order.  One lane alone takes the carries one dependent load
// after the other: 100000 rows of 2 and one of 100000 nonzeros (782 units),
// a prepared call float32 117 us -> 21, float64 111 -> 21 (25 and 39 with units
// of 1024 and 512 items and one lane).
constexpr int kFixupLaneRun = 4;
constexpr int kFixupThreads = 256;

template <class A, class O, class I, class P>
__global__ void __launch_bounds__(kFixupThreads)
k_spmv_merge_fixup(const int64_t* __restrict__ carry_row, const A* __restrict__ carry_val,
                   const A* __restrict__ head_val, int64_t n_units, const P* __restrict__ ptr,
                   const I* __restrict__ row_map, O* __restrict__ y) {
    constexpr unsigned full = 0xffffffffu;
    constexpr int kSteps = 4;
    const int64_t t = (int64_t)blockIdx.x * kFixupThreads + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int64_t r = t < n_units ? carry_row[t] : -1;
    const bool first = r >= 0 && !(t > 0 && carry_row[t - 1] == r);
    A sum = Acc<A, A>::zero();
    int64_t u = t + 1;  // the run's next unit
    if (first) {
        sum = carry_val[t];
        for (int i = 0; i < kFixupLaneRun && u < n_units && carry_row[u] == r; ++i, ++u)
            sum = acc_add(sum, carry_val[u]);
    }
    unsigned more = __ballot_sync(full, first && u < n_units && carry_row[u] == r);
    while (more) {
        const int owner = __ffs(more) - 1;
        more &= more - 1;
        const int64_t row = __shfl_sync(full, r, owner);
        int64_t base = __shfl_sync(full, u, owner);
        A part = Acc<A, A>::zero();
        unsigned in = full;
        while (in == full) {
            bool same[kSteps];
            A v[kSteps];
#pragma unroll
            for (int i = 0; i < kSteps; ++i) {
                const int64_t w = base + i * 32 + lane;
                same[i] = w < n_units && carry_row[w] == row;
                v[i] = w < n_units ? carry_val[w] : Acc<A, A>::zero();
            }
#pragma unroll
            for (int i = 0; i < kSteps; ++i) {
                if (same[i]) part = acc_add(part, v[i]);
                in = __ballot_sync(full, same[i]);  // the run is one piece: full, then its end, then none
                base += __popc(in);
            }
        }
        part = segment_reduce(full, part, 1, 32);
        if (lane == owner) {
            sum = acc_add(sum, part);
            u = base;
        }
    }
    if (first) {
        if (u < n_units) sum = acc_add(sum, head_val[u]);
        y[row_map ? idx(row_map[idx(ptr[r])]) : r] = Out<O, A>::cvt(sum);
    }
}

}  // namespace fsb

using namespace fsb;

extern "C" int fsb_spmv_csr(const fsb_csr* A, const void* x, void* y, int out_dtype, int acc_mode,
                            const fsb_plan* plan, void* workspace, int64_t workspace_bytes, void* stream) {
    if (!A || !plan) {
        fsb_host::set_error("fsb_spmv_csr: null matrix or plan");
        return FSB_ERR_INVALID;
    }
    if (A->n_rows < 0 || A->nnz < 0) {
        fsb_host::set_error("fsb_spmv_csr: negative size");
        return FSB_ERR_INVALID;
    }
    if (A->n_rows == 0) return FSB_OK;
    if (!A->row_ptr || !y || (A->nnz > 0 && (!A->values || !A->col_idx || !x))) {
        fsb_host::set_error("fsb_spmv_csr: null data pointer");
        return FSB_ERR_INVALID;
    }
    if (A->row_map && A->row_map_dtype != A->index_dtype) {
        fsb_host::set_error("fsb_spmv_csr: row_map dtype must equal index dtype");
        return FSB_ERR_INVALID;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int vdt = A->value_dtype;
    return dispatch_vao(vdt, acc_mode, out_dtype, [&](auto tv, auto ta, auto to) -> int {
        using V = typename decltype(tv)::type;
        using Ac = typename decltype(ta)::type;
        using O = typename decltype(to)::type;
        return dispatch_idx(A->index_dtype, [&](auto ti) -> int {
            using I = typename decltype(ti)::type;
            return dispatch_idx(A->ptr_dtype, [&](auto tp) -> int {
                using P = typename decltype(tp)::type;
                const V* val = static_cast<const V*>(A->values);
                const I* col = static_cast<const I*>(A->col_idx);
                const P* ptr = static_cast<const P*>(A->row_ptr);
                const I* rmap = static_cast<const I*>(A->row_map);
                const V* xv = static_cast<const V*>(x);
                O* yv = static_cast<O*>(y);
                if (plan->algo == FSB_ALGO_ROWS) {
                    int lanes = plan->lanes;
                    if (lanes < 1 || lanes > 32 || (lanes & (lanes - 1))) {
                        fsb_host::set_error("fsb_spmv_csr: lanes=%d is not a power of two in [1, 32]", lanes);
                        return FSB_ERR_INVALID;
                    }
                    int lg = 0;
                    while ((1 << lg) < lanes) ++lg;
                    const int vec_ok = aligned16(val) && aligned16(col);
                    const int64_t rows_per_block = kRowsThreads / lanes;
                    int64_t grid = ceil_div(A->n_rows, rows_per_block);
                    if (plan->grid_blocks > 0 && grid > plan->grid_blocks) grid = plan->grid_blocks;
                    if (grid > 0x7fffffffLL) grid = 0x7fffffffLL;
                    const int64_t thr = plan->comp_threshold > 0 ? plan->comp_threshold : 0;
                    const int overlap = (plan->flags & FSB_PLAN_OVERLAP_LAUNCH) && grid <= kOverlapMaxBlocks;
                    auto kern = lg == 5 ? k_spmv_rows<V, Ac, O, I, P, true> : k_spmv_rows<V, Ac, O, I, P, false>;
                    if (!overlap) {
                        kern<<<(unsigned)grid, kRowsThreads, 0, st>>>(
                            val, col, ptr, rmap, xv, yv, A->n_rows, A->nnz, plan->row_cap, thr, lg, vec_ok, 0);
                        return fsb_host::check_launch("k_spmv_rows");
                    }
                    cudaLaunchConfig_t cfg = {};
                    cfg.gridDim = dim3((unsigned)grid);
                    cfg.blockDim = dim3(kRowsThreads);
                    cfg.stream = st;
                    cudaLaunchAttribute attr[1];
                    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
                    attr[0].val.programmaticStreamSerializationAllowed = 1;
                    cfg.attrs = attr;
                    cfg.numAttrs = 1;
                    const int64_t nr = A->n_rows, nz = A->nnz, rc_cap = plan->row_cap;
                    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, val, col, ptr, rmap,
                                                             xv, yv, nr, nz, rc_cap, thr, lg, vec_ok, 1);
                    if (e != cudaSuccess) {
                        fsb_host::set_error("k_spmv_rows (overlapped launch): %s", cudaGetErrorString(e));
                        return FSB_ERR_LAUNCH;
                    }
                    return fsb_host::check_launch("k_spmv_rows");
                }
                if (plan->algo != FSB_ALGO_MERGE) {
                    fsb_host::set_error("fsb_spmv_csr: unknown algo %d", plan->algo);
                    return FSB_ERR_INVALID;
                }
                const int ipt = plan->items_per_unit / kMergeThreads;
                if (plan->items_per_unit % kMergeThreads || ipt < 1 || ipt > kMergeMaxItemsPerThread) {
                    fsb_host::set_error("fsb_spmv_csr: items_per_unit=%d must be %d x [1, %d]", plan->items_per_unit,
                                        kMergeThreads, kMergeMaxItemsPerThread);
                    return FSB_ERR_INVALID;
                }
                const int64_t n_units = plan->n_units;
                if (n_units != ceil_div(A->n_rows + A->nnz, plan->items_per_unit) || !plan->unit_coords) {
                    fsb_host::set_error("fsb_spmv_csr: merge plan does not match the matrix");
                    return FSB_ERR_INVALID;
                }
                if (plan->row_cap > 0) {
                    fsb_host::set_error("fsb_spmv_csr: row_cap needs the rows algorithm");
                    return FSB_ERR_INVALID;
                }
                const int64_t need = merge_scratch_bytes(n_units, 1, (int)sizeof(Ac));
                if (!workspace || workspace_bytes < need) {
                    fsb_host::set_error("fsb_spmv_csr: workspace %lld bytes < %lld", (long long)workspace_bytes,
                                        (long long)need);
                    return FSB_ERR_WORKSPACE;
                }
                MergeScratch ms = merge_scratch_carve(workspace, n_units, 1, (int)sizeof(Ac));
                if (n_units > 0x7fffffffLL) {
                    fsb_host::set_error("fsb_spmv_csr: too many merge tiles");
                    return FSB_ERR_LIMIT;
                }
                k_spmv_merge<V, Ac, O, I, P><<<(unsigned)ceil_div(n_units, kMergeThreads / 32), kMergeThreads, 0, st>>>(
                    val, col, ptr, rmap, xv, yv, A->n_rows, A->nnz, aligned16(val) && aligned16(col),
                    plan->unit_coords, n_units, ms.carry_row,
                    static_cast<Ac*>(ms.carry_val), static_cast<Ac*>(ms.head_val));
                int rc = fsb_host::check_launch("k_spmv_merge");
                if (rc) return rc;
                k_spmv_merge_fixup<Ac, O, I, P><<<(unsigned)ceil_div(n_units, kFixupThreads), kFixupThreads, 0, st>>>(
                    ms.carry_row, static_cast<const Ac*>(ms.carry_val), static_cast<const Ac*>(ms.head_val),
                    n_units, ptr, rmap, yv);
                return fsb_host::check_launch("k_spmv_merge_fixup");
            });
        });
    });
}

// ------------------------------------------------------ one-shot SpMV ----
// fsb_spmv_csr_checked: structural check, one device->host read of its
// figures, the heuristic plan from them, the product -- one host call.

namespace {
int64_t check_bytes(const fsb_csr* A) { return align_up(fsb_csr_check_workspace_bytes(A->n_rows, A->nnz), 256); }

// Elements of one 16-byte step of a lane: the smaller of the value and the
// index vector.
int spmv_chunk(int value_bytes, int index_bytes) {
    return 16 / std::max(1, std::min(16, std::max(value_bytes, index_bytes)));
}

// Lanes of a row group: a lane should have a few whole steps of `chunk`
// elements of its row, and a row of hundreds of nonzeros a whole warp:
//   chunk 4 (32-bit indices, values up to 4 bytes): 2 lanes, 4 from 12 (24
//           where the rows alone fill the chip) nonzeros on average, 8 from
//           80, 16 from 200, 32 from 512;
//   chunk 2 (8-byte values or indices): 2, 4 from 12, 8 from 80, 32 from 128;
//   chunk 1 (16-byte values): 2, 4 from 12, 8 from 24, 16 from 64, 32 from 128;
// doubled while the whole grid would hold at most 1024 threads per SM and the
// lanes' steps stay below twice the row.
// Measured, kernel us at lanes 2 / 4 / 8 / 16 / 32 (rows x mean, Poisson):
//   float32  10^6 x 4 32 / 48 / 86 / 166 / 285, 10^6 x 16 78 / 85 / 111 / 190 / 366,
//            10^5 x 12 8.8 / 8.7 / 10.7 / 17.6 / 36, 10^5 x 64 36 / 30 / 29 / 32 / 45,
//            10^5 x 150 80 / 62 / 59 / 60 / 73, 10^5 x 300 154 / 113 / 109 / 102 / 109,
//            20000 x 1000 95 / 54 / 54 / 44 / 42, 5000 x 3000 - / 94 / 56 / 34 / 33;
//   float16  10^6 x 12 64 / 76 / 109 / 199 / 368, 20000 x 1000 107 / 60 / 59 / 47 / 37;
//            64-bit indices: 20000 x 1000 179 / 95 / 58 / 54 / 43;
//   float64  10^5 x 32 28 / 22 / 23 / 27 / 39, 10^5 x 100 81 / 60 / 57 / 59 / 66,
//            50000 x 150 52 / 51 / 41 / 42 / 39, 20000 x 1000 235 / 122 / 126 / 93 / 56;
//   complex128 10^5 x 12 12 / 11 / 12 / 16 / 27, 50000 x 32 17 / 13 / 12 / 13 / 18,
//            10^5 x 64 60 / 48 / 41 / 40 / 48, 10^5 x 300 266 / 192 / 166 / 153 / 146.
// Four lanes for every row from 12 on (no step up with the mean) took up to
// 2.1 times the time of 32 on rows of 1000 (10^4 rows, 16-bit values, 64-bit
// indices: 50 us, 25 with 32 lanes).
// Rows that a few long ones dominate (skewed, off the merge path) take a whole
// warp.  default_spmv_plan in _plan.py follows the same rule.
int spmv_row_lanes(int64_t n_rows, double mean, int chunk, bool skewed) {
    if (skewed) return 32;
    int lanes;
    if (chunk >= 4) lanes = mean >= 512.0 ? 32 : (mean >= 200.0 ? 16 : (mean >= 80.0 ? 8 : 4));
    else if (chunk == 2) lanes = mean >= 128.0 ? 32 : (mean >= 80.0 ? 8 : 4);
    else lanes = mean >= 128.0 ? 32 : (mean >= 64.0 ? 16 : (mean >= 24.0 ? 8 : 4));
    const bool filled = n_rows * 2 >= 148 * 2048;  // with two lanes per row
    if (mean < 12.0 || (filled && mean < 6.0 * chunk)) lanes = 2;
    while (lanes < 32 && n_rows * lanes * 2 <= 148 * 1024 && 2.0 * lanes * chunk <= 2.0 * mean) lanes *= 2;
    return lanes;
}

// Merge-path unit: (rows + nonzeros) over 16 warps per SM, 128 to 1024 items
// (Zipf rows, 256 / 512 / 1024 items: 0.18 M items 8.1 / 9.9 / 13.6 us, 1.2 M
// 15.9 / 13.3 / 15.3, 3.4 M 27 / 25 / 23, 25 M 154 / 131 / 125).
int32_t spmv_merge_items(const fsb_csr* A) {
    double v = (double)(A->n_rows + A->nnz) / (148.0 * 16.0);
    if (v < 1.0) v = 1.0;
    const int64_t items = (int64_t)1 << (int)std::nearbyint(std::log2(v));
    return (int32_t)(items < 128 ? 128 : (items > 1024 ? 1024 : items));
}

// Row groups or merge path from the check's figures: merge path for skewed
// rows (the longest above 8 times the mean + 256) of less than 32 nonzeros on
// average, or of less than 128 where the matrix has at least 2^21 nonzeros or
// the longest row more than 32 steps of a whole warp (Zipf rows of 40, 12 M
// nonzeros: row groups 227 us, merge path 61).  A small matrix without such a
// row stays with the row groups there: the merge path's second launch and its
// workspace cost more than the balance gains (a prepared call, 2000 rows of 100
// with the longest at 2000: float32 14.7 us, 21.4 on the merge path, complex128
// 25 and 21; with the longest at 20000 the kernels alone 57 us and 9).
void checked_plan(const fsb_csr* A, const int64_t* fig, fsb_plan* plan) {
    memset(plan, 0, sizeof(*plan));
    const int chunk = spmv_chunk(elem_size(A->value_dtype), elem_size(A->index_dtype));
    const double mean = A->n_rows ? (double)A->nnz / (double)A->n_rows : 0.0;
    const bool skewed = (double)fig[5] > 8.0 * (mean > 1.0 ? mean : 1.0) + 256.0;
    if (A->n_rows > 0 && skewed &&
        (mean < 32.0 || (mean < 128.0 && (A->nnz >= (1 << 21) || fig[5] > 32 * 32 * chunk)))) {
        plan->algo = FSB_ALGO_MERGE;
        plan->items_per_unit = spmv_merge_items(A);
        plan->n_units = ceil_div(A->n_rows + A->nnz, plan->items_per_unit);
        return;
    }
    plan->algo = FSB_ALGO_ROWS;
    plan->lanes = A->n_rows ? spmv_row_lanes(A->n_rows, mean, chunk, skewed) : 32;
    plan->flags = FSB_PLAN_OVERLAP_LAUNCH;
}

int64_t checked_merge_bytes(const fsb_csr* A, int acc_mode, int out_dtype) {
    fsb_plan mp;
    memset(&mp, 0, sizeof(mp));
    mp.algo = FSB_ALGO_MERGE;
    mp.items_per_unit = spmv_merge_items(A);
    mp.n_units = ceil_div(A->n_rows + A->nnz, mp.items_per_unit);
    const int64_t coords = align_up((mp.n_units + 1) * 2 * (int64_t)sizeof(int64_t), 256);
    return coords + fsb_workspace_bytes(0, A, 1, acc_mode, out_dtype, &mp);
}
}  // namespace

extern "C" int64_t fsb_spmv_csr_checked_workspace_bytes(const fsb_csr* A, int acc_mode, int out_dtype) {
    if (!A || A->n_rows < 0 || A->nnz < 0) return 0;
    return check_bytes(A) + checked_merge_bytes(A, acc_mode, out_dtype);
}

extern "C" int fsb_spmv_csr_checked(const fsb_csr* A, const void* x, void* y, int out_dtype, int acc_mode,
                                    void* workspace, int64_t workspace_bytes, int64_t* figures, fsb_plan* plan_out,
                                    void* stream) {
    if (!A || !figures || A->n_rows < 0 || A->nnz < 0) {
        fsb_host::set_error("fsb_spmv_csr_checked: bad arguments");
        return FSB_ERR_INVALID;
    }
    const int64_t need = fsb_spmv_csr_checked_workspace_bytes(A, acc_mode, out_dtype);
    if (!workspace || workspace_bytes < need) {
        fsb_host::set_error("fsb_spmv_csr_checked: workspace %lld bytes < %lld", (long long)workspace_bytes,
                            (long long)need);
        return FSB_ERR_WORKSPACE;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // the check's kernels write the figures straight into a pinned buffer of
    // this host thread: no copy-engine work to queue behind uploads
    static thread_local int64_t* staged = nullptr;
    if (!staged && cudaHostAlloc(reinterpret_cast<void**>(&staged), 8 * sizeof(int64_t),
                                 cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
        staged = nullptr;
        return fsb_host::check_launch("fsb_spmv_csr_checked: pinned figure buffer");
    }
    const int64_t cb = check_bytes(A);
    int rc = fsb_csr_check(A->row_ptr, A->ptr_dtype, A->n_rows, A->col_idx, A->index_dtype, A->nnz, staged,
                           workspace, cb, stream);
    if (rc) return rc;
    if (cudaStreamSynchronize(st) != cudaSuccess) return fsb_host::check_launch("fsb_spmv_csr_checked: check");
    memcpy(figures, staged, 8 * sizeof(int64_t));
    if (figures[0] != 0 || figures[1] != A->nnz || figures[2] != 0 ||
        (A->nnz > 0 && (figures[3] != 0 || figures[4] >= A->n_cols))) {
        fsb_host::set_error("fsb_spmv_csr_checked: malformed CSR structure (figures returned)");
        return FSB_ERR_INVALID;
    }
    fsb_plan plan;
    checked_plan(A, figures, &plan);
    if (plan_out) *plan_out = plan;
    if (A->n_rows == 0) return FSB_OK;
    char* rest = static_cast<char*>(workspace) + cb;
    int64_t rest_bytes = workspace_bytes - cb;
    if (plan.algo == FSB_ALGO_MERGE) {
        int64_t* coords = reinterpret_cast<int64_t*>(rest);
        const int64_t cb = align_up((plan.n_units + 1) * 2 * (int64_t)sizeof(int64_t), 256);
        rc = fsb_merge_partition(A->row_ptr, A->ptr_dtype, A->n_rows, A->nnz, plan.items_per_unit, 0, coords,
                                 plan.n_units, stream);
        if (rc) return rc;
        plan.unit_coords = coords;
        rest += cb;
        rest_bytes -= cb;
    }
    return fsb_spmv_csr(A, x, y, out_dtype, acc_mode, &plan, rest, rest_bytes, stream);
}

// --------------------------------------------------- allocation-free SpMV ----
// fsb_spmv_csr_noalloc: the merge-path SpMV for callers that cannot allocate
// device memory -- a C program or plug-in that receives device pointers from
// a host framework owning all device memory, or a latency-critical loop in
// which cudaMalloc's implicit device-wide synchronisation is not acceptable.
// The caller still passes the matrix, x and y; the scratch this algorithm
// needs (merge-path tile coordinates and per-tile carries) lives in the
// file-scope device array below, of a fixed size, held by every GPU that loads
// this library until the process exits.
//
// Limit: at most kNoAllocMaxTiles merge-path tiles, i.e.
// n_rows + nnz <= kNoAllocMaxTiles * items_per_unit (16384 tiles: 16.7 M path
// items at 1024 items per tile); larger matrices are rejected with
// FSB_ERR_LIMIT.  Every call on a device shares the one array: two calls whose
// kernels overlap on the GPU (for example on two streams) race on it, so
// callers must order such calls.  Nothing in the array has to start at zero:
// each call writes the coordinates and every tile's carry slot before they
// are read.  The first call in a CUDA context (the device's primary context,
// or a host framework's own context current on the calling thread) resolves
// the array's device address in that context (cudaGetSymbolAddress) and
// caches it per context; that first call should come before any stream
// capture.
constexpr int64_t kNoAllocMaxTiles = 16384;
constexpr int64_t kNoAllocCoordBytes = ((kNoAllocMaxTiles + 1) * 2 * 8 + 255) / 256 * 256;
constexpr int64_t kNoAllocBytes = kNoAllocCoordBytes + (kNoAllocMaxTiles * 8 + 255) / 256 * 256 +
                                  2 * ((kNoAllocMaxTiles * 16 + 255) / 256 * 256);
static __device__ __align__(256) unsigned char g_spmv_noalloc_scratch[kNoAllocBytes];

namespace {
// The array's device address belongs to the CUDA context that was current
// when it was resolved: a plug-in may run inside its host framework's own
// driver context rather than the device's primary context.  Addresses are
// therefore cached per context (cuCtxGetCurrent, reached through the
// runtime's driver entry-point query), not per device ordinal.
using CtxGetCurrentFn = int (*)(void**);
constexpr int kMaxContexts = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_ctx[kMaxContexts] = {};
void* g_noalloc_ptr[kMaxContexts] = {};
int g_noalloc_used = 0;

CtxGetCurrentFn ctx_get_current() {
    static std::once_flag once;
    static CtxGetCurrentFn fn = nullptr;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<CtxGetCurrentFn>(p);
    });
    return fn;
}

// Device address of the scratch array in the current context (resolved on
// the first call made in that context).
int noalloc_scratch(void** out) {
    CtxGetCurrentFn get_ctx = ctx_get_current();
    if (!get_ctx) {
        fsb_host::set_error("fsb_spmv_csr_noalloc: cuCtxGetCurrent is not available");
        return FSB_ERR_LAUNCH;
    }
    void* ctx = nullptr;
    if (get_ctx(&ctx) != 0) ctx = nullptr;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (ctx) {
        for (int i = 0; i < g_noalloc_used; ++i) {
            if (g_noalloc_ctx[i] == ctx) {
                *out = g_noalloc_ptr[i];
                return FSB_OK;
            }
        }
    }
    // First call in this context (or no context current yet: the runtime
    // then makes the current device's primary context current here).
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_spmv_noalloc_scratch);
    if (e != cudaSuccess || !p) {
        fsb_host::set_error("fsb_spmv_csr_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        return FSB_ERR_LAUNCH;
    }
    if (!ctx && (get_ctx(&ctx) != 0 || !ctx)) {
        fsb_host::set_error("fsb_spmv_csr_noalloc: no current CUDA context");
        return FSB_ERR_LAUNCH;
    }
    if (g_noalloc_used < kMaxContexts) {
        g_noalloc_ctx[g_noalloc_used] = ctx;
        g_noalloc_ptr[g_noalloc_used] = p;
        ++g_noalloc_used;
    }
    *out = p;
    return FSB_OK;
}
}  // namespace

extern "C" int fsb_spmv_csr_noalloc(const fsb_csr* A, const void* x, void* y, int out_dtype, int acc_mode,
                                    int32_t items_per_unit, void* stream) {
    if (!A) {
        fsb_host::set_error("fsb_spmv_csr_noalloc: null matrix");
        return FSB_ERR_INVALID;
    }
    if (A->n_rows < 0 || A->nnz < 0) {
        fsb_host::set_error("fsb_spmv_csr_noalloc: negative size");
        return FSB_ERR_INVALID;
    }
    if (items_per_unit % kMergeThreads || items_per_unit < kMergeThreads || items_per_unit > kMergeMaxTile) {
        fsb_host::set_error("fsb_spmv_csr_noalloc: items_per_unit=%d must be %d x [1, %d]", items_per_unit,
                            kMergeThreads, kMergeMaxItemsPerThread);
        return FSB_ERR_INVALID;
    }
    if (A->n_rows == 0) return FSB_OK;
    const int64_t n_tiles = ceil_div(A->n_rows + A->nnz, items_per_unit);
    if (n_tiles > kNoAllocMaxTiles) {
        fsb_host::set_error("fsb_spmv_csr_noalloc: %lld tiles exceed the fixed scratch of %lld tiles "
                            "(n_rows + nnz must be <= %lld at items_per_unit=%d)",
                            (long long)n_tiles, (long long)kNoAllocMaxTiles,
                            (long long)(kNoAllocMaxTiles * items_per_unit), items_per_unit);
        return FSB_ERR_LIMIT;
    }
    if (!A->row_ptr || !y || (A->nnz > 0 && (!A->values || !A->col_idx || !x))) {
        fsb_host::set_error("fsb_spmv_csr_noalloc: null data pointer");
        return FSB_ERR_INVALID;
    }
    if (A->row_map && A->row_map_dtype != A->index_dtype) {
        fsb_host::set_error("fsb_spmv_csr_noalloc: row_map dtype must equal index dtype");
        return FSB_ERR_INVALID;
    }
    void* scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    int64_t* coords = static_cast<int64_t*>(scratch);
    void* carries = static_cast<unsigned char*>(scratch) + kNoAllocCoordBytes;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return dispatch_vao(A->value_dtype, acc_mode, out_dtype, [&](auto tv, auto ta, auto to) -> int {
        using V = typename decltype(tv)::type;
        using Ac = typename decltype(ta)::type;
        using O = typename decltype(to)::type;
        return dispatch_idx(A->index_dtype, [&](auto ti) -> int {
            using I = typename decltype(ti)::type;
            return dispatch_idx(A->ptr_dtype, [&](auto tp) -> int {
                using P = typename decltype(tp)::type;
                const P* ptr = static_cast<const P*>(A->row_ptr);
                k_merge_partition<P><<<(unsigned)ceil_div(n_tiles + 1, 256), 256, 0, st>>>(
                    ptr, A->n_rows, A->nnz, items_per_unit, 0, coords, n_tiles);
                int rc2 = fsb_host::check_launch("k_merge_partition (noalloc)");
                if (rc2) return rc2;
                MergeScratch ms = merge_scratch_carve(carries, n_tiles, 1, (int)sizeof(Ac));
                O* yv = static_cast<O*>(y);
                const I* rmap = static_cast<const I*>(A->row_map);
                k_spmv_merge<V, Ac, O, I, P><<<(unsigned)ceil_div(n_tiles, kMergeThreads / 32), kMergeThreads, 0, st>>>(
                    static_cast<const V*>(A->values), static_cast<const I*>(A->col_idx), ptr, rmap,
                    static_cast<const V*>(x), yv, A->n_rows, A->nnz,
                    aligned16(A->values) && aligned16(A->col_idx), coords, n_tiles, ms.carry_row,
                    static_cast<Ac*>(ms.carry_val), static_cast<Ac*>(ms.head_val));
                rc2 = fsb_host::check_launch("k_spmv_merge (noalloc)");
                if (rc2) return rc2;
                k_spmv_merge_fixup<Ac, O, I, P><<<(unsigned)ceil_div(n_tiles, kFixupThreads), kFixupThreads, 0, st>>>(
                    ms.carry_row, static_cast<const Ac*>(ms.carry_val), static_cast<const Ac*>(ms.head_val),
                    n_tiles, ptr, rmap, yv);
                return fsb_host::check_launch("k_spmv_merge_fixup (noalloc)");
            });
        });
    });
}
