// fsb_spmm_walk.cuh -- the range-walk form of the batched merge-path SpMM
// (FSB_ALGO_SEQ with FSB_PLAN_WALK; instantiated per value type in
// fsb_spmm_walk_*.cu), the form the heuristics, the selector and the batch use
// for all but narrow operands with long rows (spmm_form in _plan.py).
//
// One warp per (merge-path unit, column tile), as in fsb_spmm_seq.cuh.  The
// unit's nonzeros pass through shared memory in chunks of kWalkChunk: columns,
// values, and one bit per nonzero that tells where a row starts.  Each of the
// warp's NPAR = 32 / LPN sub-groups walks its own contiguous part of the chunk
// in batches of U nonzeros whose B-row loads are issued back to back; columns
// and values come as broadcast 16-byte shared-memory loads.  A sub-group
// stores its rows itself where their bits say so: no reduction across the warp
// per row and no replay of a batch per row, which is what k_spmm_seq spends
// most of its instructions on when rows are short (26 warp instructions per
// nonzero on the power-law matrix at N = 64; 10 here).  Sub-groups meet once
// per chunk, in a segmented scan of their open partials; a range's first row,
// begun before the range, waits for that in shared memory.  Sums are
// deterministic: batches of U, rows in order, sub-groups in order, units in
// order (tickets or the fix-up kernel, as in fsb_spmm_seq.cuh).
//
// What bounds it: the B rows in flight per SM.  Measured, cold-to-warm L2
// back to back, k_spmm_seq -> this form at their best unit sizes:
//   power law 262144^2, 3.1 M nonzeros, float32: N = 64 133 -> 82 us (the
//   gathers alone take 68 us), N = 32 104 -> 55, N = 8 87 -> 41, N = 128
//   264 -> 164, N = 64 with float64 sums 210 -> 134 us;
//   64 uneven matrices, 33 M nonzeros, N = 32: 540 -> 326 us;
//   50021 x 25013, 1.2 M nonzeros, N = 33, float64 sums: 119 -> 51 us.
#pragma once
#include "fsb_spmm_seq.cuh"

namespace fsb {

// Nonzeros staged per warp.  128 spends more on staging and on the sub-groups'
// meeting (64 matrices: 367 us against 325).
constexpr int kWalkChunk = 256;

// Resident CTAs of 128 threads per SM requested from the compiler.  For
// accumulators of 16 bytes per lane, power law at N = 64: 5 CTAs (96
// registers) 95 us, 6 (80) 81, 7 (72) 90, 8 (64, spills) 101; 4 CTAs with 16
// loads in flight per lane 92.  32 bytes per lane (float64 sums, N = 64): 5 CTAs
// 134, 4 CTAs 138 us at 256 items.
template <class V, class A, int VW> struct WalkMinBlocks {
    static constexpr int acc_bytes = (int)sizeof(A) * VW;
    static constexpr int value = acc_bytes <= 16 ? 6 : (acc_bytes <= 32 ? 5 : 4);
};

// N values from 16-byte aligned shared memory, in the widest loads.
template <class T, int N>
__device__ __forceinline__ void lds_vec(const T* p, T (&out)[N]) {
    constexpr int BY = (int)sizeof(T) * N;
    if constexpr (BY >= 16) {
#pragma unroll
        for (int i = 0; i < BY / 16; ++i) {
            const uint4 q = reinterpret_cast<const uint4*>(p)[i];
            memcpy(reinterpret_cast<char*>(out) + 16 * i, &q, 16);
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) out[i] = p[i];
    }
}

// As seq_finish_row / seq_unit_tickets, for lane columns CS apart (CS = 1: VW
// consecutive ones).
template <class A, class O, class I, class P, int VW, int CS>
__device__ __forceinline__ void walk_finish_row(int64_t first, int64_t last, int64_t row, const A* carry_val,
                                                const A* head_val, int64_t n_dense, int64_t c0, const P* ptr,
                                                const I* row_map, O* C, int64_t ldc) {
    if constexpr (CS == 1) {
        seq_finish_row<A, O, I, P, VW>(first, last, row, carry_val, head_val, n_dense, c0, ptr, row_map, C, ldc);
    } else {
#pragma unroll
        for (int w = 0; w < VW; ++w)
            if (c0 + w * CS < n_dense)
                seq_finish_row<A, O, I, P, 1>(first, last, row, carry_val, head_val, n_dense, c0 + w * CS, ptr,
                                              row_map, C, ldc);
    }
}

template <class A, class O, class I, class P, int VW, int CS>
__device__ __noinline__ void walk_unit_tickets(int64_t unit, int64_t r0, int64_t r1, bool head, bool open, int lane,
                                               bool finisher_lane, int64_t c0, const int64_t* runs, int* tix,
                                               const A* carry_val, const A* head_val, int64_t n_dense, const P* ptr,
                                               const I* row_map, O* C, int64_t ldc) {
    for (int job = 0; job < 2; ++job) {
        int64_t first = -1, last = -1, row = 0;
        if (job == 0 && head) {
            first = runs[2 * unit - 2];
            last = unit;
            row = r0;
        } else if (job == 1 && open) {
            first = runs[2 * unit];
            last = runs[2 * unit + 1];
            row = r1;
        }
        if (first >= 0 && last > first && seq_take_ticket(tix + first, (int)(last - first + 1), lane) &&
            finisher_lane)
            walk_finish_row<A, O, I, P, VW, CS>(first, last, row, carry_val, head_val, n_dense, c0, ptr, row_map, C,
                                                ldc);
    }
}

template <class V, class A, class O, class I, int VW, int LPN_LOG2, bool STRIDED>
__global__ void __launch_bounds__(kSpmmThreads, WalkMinBlocks<V, A, VW>::value)
k_spmm_walk(const V* __restrict__ val, const I* __restrict__ col, const void* __restrict__ ptr, int ptr64,
            const V* __restrict__ B, uint32_t ldb_bytes, O* __restrict__ C, uint32_t ldc_bytes, int64_t n_rows,
            int64_t n_dense, const int64_t* __restrict__ coords, int64_t n_units, int64_t* __restrict__ carry_row,
            A* __restrict__ carry_val, A* __restrict__ head_val, const int64_t* __restrict__ runs,
            int* __restrict__ tickets) {
    constexpr int LPN = 1 << LPN_LOG2;
    constexpr int NPAR = 32 >> LPN_LOG2;
    constexpr int U = VW * (int)sizeof(V) * 8 <= 192 ? 8 : 4;  // B loads in flight per lane
    constexpr int CH = kWalkChunk;
    constexpr int WORDS = CH / 32;
    constexpr int kWarps = kSpmmThreads / 32;
    constexpr unsigned full = 0xffffffffu;
    __shared__ __align__(16) uint32_t sm_col[kWarps][CH];
    __shared__ __align__(16) int sm_row[kWarps][CH];  // row (relative + 1) of each row start, at its first nonzero
    __shared__ __align__(16) V sm_val[kWarps][CH];
    __shared__ __align__(16) uint32_t sm_brk[kWarps][WORDS];  // bit per nonzero: a row starts here
    __shared__ __align__(16) A sm_head[kSpmmThreads][VW];  // a range's first row, finished before its part from earlier
    __shared__ __align__(16) A sm_open[kSpmmThreads][VW];  // the open row's sum before the chunk (first sub-group)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* s_col = sm_col[warp];
    int* s_row = sm_row[warp];
    V* s_val = sm_val[warp];
    const unsigned char* s_brk = reinterpret_cast<const unsigned char*>(sm_brk[warp]);
    const int sub = lane >> LPN_LOG2, lig = lane & (LPN - 1);
    // the lane's columns: VW consecutive ones, or (STRIDED) VW of them LPN apart
    const int64_t c0 = (int64_t)blockIdx.y * (LPN * VW) + (STRIDED ? lig : lig * VW);
    const bool col_ok = c0 < n_dense;
    const char* Bl = reinterpret_cast<const char*>(B + (col_ok ? c0 : 0));
    const uint64_t keep_b = policy_evict_last();
    auto row_ptr = [&](int64_t r) -> int64_t {
        return ptr64 ? static_cast<const int64_t*>(ptr)[r] : (int64_t)static_cast<const int32_t*>(ptr)[r];
    };
    auto load_b = [&](uint32_t c) -> vec_t<V, VW> {
        const V* p = reinterpret_cast<const V*>(Bl + (uint64_t)c * ldb_bytes);
        if constexpr (!STRIDED) {
            return ld_keep<V, VW>(p, keep_b);
        } else {
            vec_t<V, VW> v;
#pragma unroll
            for (int w = 0; w < VW; ++w) {
                v.v[w] = vzero<V>();
                if (c0 + w * LPN < n_dense) v.v[w] = ld_keep<V, 1>(p + w * LPN, keep_b).v[0];
            }
            return v;
        }
    };
    auto put_partial = [&](A* base, int64_t unit, const A (&a)[VW]) {
        A* dst = base + unit * n_dense + c0;
#pragma unroll
        for (int w = 0; w < VW; ++w) {
            if constexpr (STRIDED) {
                if (c0 + w * LPN < n_dense) dst[w * LPN] = a[w];
            } else {
                dst[w] = a[w];
            }
        }
    };

    const int64_t unit_stride = (int64_t)gridDim.x * kWarps;
    for (int64_t unit = (int64_t)blockIdx.x * kWarps + warp; unit < n_units; unit += unit_stride) {
        // everything below is relative to the unit's first row and nonzero
        // (a unit holds at most 2^24 rows and nonzeros); rows are numbered
        // from 1
        const int64_t r0 = coords[2 * unit], k0 = coords[2 * unit + 1];
        const int n_ends = (int)(coords[2 * unit + 2] - r0);  // rows ending in the unit
        const int nk = (int)(coords[2 * unit + 3] - k0);
        const int n_rel = n_ends + (r0 + n_ends < n_rows ? 1 : 0);  // rows touched, the one open at the end included
        // start of row i + 1, relative to k0 (clamped to [-1, nk + 1])
        auto start_of = [&](int i) -> int {
            const int64_t s = row_ptr(r0 + i) - k0;
            return s < 0 ? -1 : (s > nk ? nk + 1 : (int)s);
        };
        const bool continued = n_rel > 0 && start_of(0) < 0;
        char* Cl = reinterpret_cast<char*>(C + c0) + (r0 - 1) * (int64_t)ldc_bytes;

        A acc[VW];
        zero_acc<A, VW>(acc);
        auto put_row = [&](int rel, const A (&a)[VW]) {
            O* dst = reinterpret_cast<O*>(Cl + (uint64_t)(uint32_t)rel * ldc_bytes);
            if constexpr (STRIDED) {
#pragma unroll
                for (int w = 0; w < VW; ++w)
                    if (c0 + w * LPN < n_dense) dst[w * LPN] = Out<O, A>::cvt(a[w]);
            } else {
                if (col_ok) store_row<O, A, VW>(dst, 0, 0, 0, a);
            }
        };
        // a finished row: its C row, or the head partial of a row that began
        // in an earlier unit
        auto finish = [&](int rel, const A (&a)[VW]) {
            if (rel == 1 && continued) {
                if (col_ok) put_partial(head_val, unit, a);
            } else {
                put_row(rel, a);
            }
        };
        // a continued row that ends where the unit begins: nothing left to add
        if (continued && n_ends > 0 && start_of(1) == 0 && sub == 0 && col_ok) put_partial(head_val, unit, acc);

        if (sub == 0) {
#pragma unroll
            for (int w = 0; w < VW; ++w) sm_open[threadIdx.x][w] = acc[w];
        }
        int rb = 0;        // rows whose start has been passed
        int open_row = 1;  // row open at the chunk's start
        for (int kc = 0;; kc += CH) {
            const int n = nk - kc < CH ? nk - kc : CH;
            const bool last = kc + n == nk;
            // ---- stage the chunk: values, columns, row starts
            {
                V tv[WORDS];
                I tc[WORDS];
#pragma unroll
                for (int i = 0; i < WORDS; ++i) {
                    const int j = lane + 32 * i;
                    tv[i] = vzero<V>();
                    tc[i] = 0;
                    if (j < n) {
                        tv[i] = ld_stream1(val + (k0 + kc) + j);
                        tc[i] = ld_stream1(col + (k0 + kc) + j);
                    }
                }
                uint32_t brk[WORDS];
#pragma unroll
                for (int i = 0; i < WORDS; ++i) brk[i] = 0u;
                for (;;) {
                    const int row = rb + lane;
                    const bool in = row < n_rel;
                    const int s = in ? start_of(row) - kc : 0, e = in ? start_of(row + 1) - kc : 0;
                    const bool take = in && (s < n || (last && row < n_ends));
                    const bool mark = take && e > s && s >= 0 && s < n;
                    if (mark) s_row[s] = row + 1;
#pragma unroll
                    for (int i = 0; i < WORDS; ++i)
                        brk[i] |= __reduce_or_sync(full, mark && (s >> 5) == i ? 1u << (s & 31) : 0u);
                    // empty rows are written here
                    const unsigned empty = __ballot_sync(full, take && e == s && row < n_ends);
                    if (empty) {
                        A z[VW];
                        zero_acc<A, VW>(z);
                        for (int i = 0; i < 32; i += NPAR)
                            if ((empty >> (i + sub)) & 1u) put_row(rb + i + sub + 1, z);
                    }
                    const int cnt = __popc(__ballot_sync(full, take));
                    rb += cnt;
                    if (cnt < 32) break;
                }
                if (lane == 0) {
#pragma unroll
                    for (int i = 0; i < WORDS; ++i) sm_brk[warp][i] = brk[i];
                }
#pragma unroll
                for (int i = 0; i < WORDS; ++i) {
                    s_val[lane + 32 * i] = tv[i];
                    s_col[lane + 32 * i] = (uint32_t)tc[i];
                }
            }
            __syncwarp();
            if (n > 0) {
                // ---- walk.  Whole batches of U are dealt out evenly and in
                // order; what does not divide makes one ragged round.
                const int nb = n / U, base = nb / NPAR, extra = nb - base * NPAR;
                const int e_lo = U * (sub * base + (sub < extra ? sub : extra));
                const int ragged = sub < extra ? U : (sub == NPAR - 1 ? n - nb * U : 0);
                const bool some = base > 0 || ragged > 0;
                auto brk_bits = [&](int e) -> uint32_t {
                    if constexpr (U == 8) return s_brk[e >> 3];
                    else return (uint32_t)(s_brk[e >> 3] >> (e & 4)) & 15u;
                };
                // the range's first row began before it (cont: and is not finished yet)
                const bool has_open = kc > 0 || continued;
                bool joined = true;
                int rcur = has_open ? open_row : 0;  // 0: no row open yet
                uint32_t first_mask = ~0u;
                if (sub > 0 || !has_open) {
                    const bool starts = some && (brk_bits(e_lo) & 1u);
                    joined = !starts;
                    if (starts) rcur = s_row[e_lo];
                    first_mask = ~1u;  // the first nonzero of a range ends nothing
                }
                bool cont = joined;
                zero_acc<A, VW>(acc);
                auto batch = [&](int e, int cnt, bool whole) {
                    vec_t<V, VW> bv[U];
                    if (whole) {
#pragma unroll
                        for (int u = 0; u < U; u += 4) {
                            uint32_t c[4];
                            lds_vec(s_col + e + u, c);
#pragma unroll
                            for (int q = 0; q < 4; ++q) bv[u + q] = load_b(c[q]);
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < U; ++u) {
#pragma unroll
                            for (int w = 0; w < VW; ++w) bv[u].v[w] = vzero<V>();
                            if (u < cnt) bv[u] = load_b(s_col[e + u]);
                        }
                    }
                    uint32_t bits = cnt > 0 ? brk_bits(e) & first_mask : 0u;
                    if (!whole) bits &= (1u << cnt) - 1u;
                    first_mask = ~0u;
                    V a[U];
                    if (whole) {
                        lds_vec(s_val + e, a);
                    } else {
#pragma unroll
                        for (int u = 0; u < U; ++u) a[u] = u < cnt ? s_val[e + u] : vzero<V>();
                    }
                    // a batch's products are summed on their own, in two chains,
                    // and enter the row's sum once
                    A t[2][VW];
                    zero_acc<A, VW>(t[0]);
                    zero_acc<A, VW>(t[1]);
                    auto join = [&]() {
#pragma unroll
                        for (int w = 0; w < VW; ++w) acc[w] = acc_add(acc[w], acc_add(t[0][w], t[1][w]));
                    };
                    if (!__any_sync(full, bits != 0u)) {
#pragma unroll
                        for (int u = 0; u < U; ++u)
#pragma unroll
                            for (int w = 0; w < VW; ++w) t[u & 1][w] = Acc<V, A>::fma(a[u], bv[u].v[w], t[u & 1][w]);
                    } else {
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            if (bits & (1u << u)) {
                                join();
                                if (cont) {
#pragma unroll
                                    for (int w = 0; w < VW; ++w) sm_head[threadIdx.x][w] = acc[w];
                                    cont = false;
                                } else {
                                    put_row(rcur, acc);
                                }
                                rcur = s_row[e + u];
                                zero_acc<A, VW>(acc);
                                zero_acc<A, VW>(t[0]);
                                zero_acc<A, VW>(t[1]);
                            }
#pragma unroll
                            for (int w = 0; w < VW; ++w) t[u & 1][w] = Acc<V, A>::fma(a[u], bv[u].v[w], t[u & 1][w]);
                        }
                    }
                    join();
                };
                for (int it = 0; it < base; ++it) batch(e_lo + it * U, U, true);
                if (nb * U < n || extra > 0) batch(e_lo + base * U, ragged, false);

                // ---- the sub-groups' open partials, in order: f = the tail
                // holds no part of the previous sub-group's row
                const bool broke = joined && !cont;
                if (sub == 0 && has_open) {  // the chunk's sum joins the open row's once
#pragma unroll
                    for (int w = 0; w < VW; ++w) {
                        const A o = sm_open[threadIdx.x][w];
                        if (broke) sm_head[threadIdx.x][w] = acc_add(o, sm_head[threadIdx.x][w]);
                        else acc[w] = acc_add(o, acc[w]);
                    }
                }
                int f = (sub > 0 && joined && !broke) ? 0 : 1;
                int row_t = rcur;
#pragma unroll
                for (int o = LPN; o < 32; o <<= 1) {
                    const int fu = __shfl_up_sync(full, f, o), ru = __shfl_up_sync(full, row_t, o);
                    const bool add = lane >= o && !f;
#pragma unroll
                    for (int w = 0; w < VW; ++w) {
                        const A up = shfl_up(full, acc[w], o);
                        if (add) acc[w] = acc_add(up, acc[w]);
                    }
                    if (add) {
                        row_t = ru;
                        f = fu;
                    }
                }
                if constexpr (NPAR > 1) {
                    const int in_row = __shfl_up_sync(full, row_t, LPN);
                    A in[VW];
#pragma unroll
                    for (int w = 0; w < VW; ++w) in[w] = shfl_up(full, acc[w], LPN);
                    if (broke) {
                        A h[VW];
#pragma unroll
                        for (int w = 0; w < VW; ++w) {
                            h[w] = sm_head[threadIdx.x][w];
                            if (sub > 0) h[w] = acc_add(in[w], h[w]);
                        }
                        finish(sub > 0 ? in_row : open_row, h);
                    }
                    const int next_joined = __shfl_down_sync(full, (int)joined, LPN);
                    if (sub < NPAR - 1 && !next_joined && row_t > 0) finish(row_t, acc);
                    // the open row's partial moves to the first sub-group
#pragma unroll
                    for (int w = 0; w < VW; ++w) acc[w] = shfl_idx(full, acc[w], (32 - LPN) + lig, 32);
                } else if (broke) {
                    A h[VW];
#pragma unroll
                    for (int w = 0; w < VW; ++w) h[w] = sm_head[threadIdx.x][w];
                    finish(open_row, h);
                }
                if (sub == 0) {
#pragma unroll
                    for (int w = 0; w < VW; ++w) sm_open[threadIdx.x][w] = acc[w];
                }
                open_row = __shfl_sync(full, row_t, 31);
                __syncwarp();  // the next chunk overwrites the staged one
            }
            if (last) break;
        }
        bool open = false;
        if (nk > 0) {
            if (n_rel > n_ends) {
                const int s1 = start_of(n_ends);
                open = nk > (s1 > 0 ? s1 : 0);
            }
            if (sub == 0 && col_ok) {
                if (open) put_partial(carry_val, unit, acc);
                else finish(open_row, acc);
            }
        }
        const int64_t r1 = r0 + n_ends;
        if (runs) {
            const int64_t ldc = (int64_t)(ldc_bytes / (uint32_t)sizeof(O));
            if (ptr64)
                walk_unit_tickets<A, O, I, int64_t, VW, STRIDED ? LPN : 1>(
                    unit, r0, r1, continued && n_ends > 0, open, lane, sub == 0 && col_ok, c0, runs,
                    tickets + (int64_t)blockIdx.y * n_units, carry_val, head_val, n_dense,
                    static_cast<const int64_t*>(ptr), (const I*)nullptr, C, ldc);
            else
                walk_unit_tickets<A, O, I, int32_t, VW, STRIDED ? LPN : 1>(
                    unit, r0, r1, continued && n_ends > 0, open, lane, sub == 0 && col_ok, c0, runs,
                    tickets + (int64_t)blockIdx.y * n_units, carry_val, head_val, n_dense,
                    static_cast<const int32_t*>(ptr), (const I*)nullptr, C, ldc);
        } else if (blockIdx.y == 0 && lane == 0) {
            carry_row[unit] = open ? r1 : -1;
        }
    }
}

template <class V, class A, class O, class I, int VW, bool STRIDED, int LPN_LOG2>
void launch_walk_one(dim3 g, cudaStream_t st, const V* val, const I* col, const void* ptr, int ptr64, const V* B,
                     uint32_t ldb_bytes, O* C, uint32_t ldc_bytes, int64_t n_rows, int64_t n_dense,
                     const int64_t* coords, int64_t n_units, int64_t* carry_row, A* cv, A* hv, const int64_t* runs,
                     int* tickets) {
    k_spmm_walk<V, A, O, I, VW, LPN_LOG2, STRIDED><<<g, kSpmmThreads, 0, st>>>(
        val, col, ptr, ptr64, B, ldb_bytes, C, ldc_bytes, n_rows, n_dense, coords, n_units, carry_row, cv, hv, runs,
        tickets);
}

// Lane shape of a column tile: contiguous 16-byte lane vectors where B and C
// allow, else `vw` columns LPN apart.
struct WalkTile {
    int vw, lpn_log2;
    bool strided;
    int width() const { return vw << lpn_log2; }
};

// Unaligned rows: the compiled (columns per lane, lanes) pairs covering
// `target` columns (at most 128 per tile) in the fewest lane loads, 1 column
// per lane before 3 (an odd width of 33 takes 3 x 16: 1.5 loads per nonzero
// where 32 + 32 single columns took two passes).
inline WalkTile walk_strided_tile(int64_t target) {
    if (target > 96) return {4, 5, true};
    if (target > 64) return {3, 5, true};
    if (target > 48) return {2, 5, true};
    for (int l = 0; l <= 5; ++l) {
        if (target <= (1 << l)) return {1, l, true};
        if (l >= 1 && target <= 3 << (l - 1)) return {3, l - 1, true};
    }
    return {3, 4, true};
}

// Compiled accumulator / value pairs of this form: all but the compensated
// ones (walk_takes keeps those calls in k_spmm_seq).
template <class V, class A, class O, class I>
int launch_walk(const fsb_csr* Am, const V* val, const I* col, const V* B, int64_t ldb, int64_t n_dense,
                O* C, int64_t ldc, const fsb_plan* plan, void* workspace, int64_t workspace_bytes,
                cudaStream_t st) {
    const int64_t n_units = plan->n_units;
    if (plan->items_per_unit < 1 || plan->items_per_unit > kMaxItemsPerUnit ||
        n_units != ceil_div(Am->n_rows + Am->nnz, plan->items_per_unit) || !plan->unit_coords || plan->row_cap > 0) {
        fsb_host::set_error("fsb_spmm_csr: seq plan does not match the matrix");
        return FSB_ERR_INVALID;
    }
    constexpr int kMaxVW = seq_max_vw<V, O>();
    constexpr size_t kCAlign = kMaxVW * sizeof(O) < 16 ? kMaxVW * sizeof(O) : 16;
    const bool wide_ok = kMaxVW > 1 && ((uintptr_t)B) % (kMaxVW * sizeof(V)) == 0 && ldb % kMaxVW == 0 &&
                         n_dense % kMaxVW == 0 && ((uintptr_t)C) % kCAlign == 0 && ldc % kMaxVW == 0;
    const int64_t target = plan->n_tile > 0 && plan->n_tile < n_dense ? plan->n_tile : n_dense;
    WalkTile t;
    if (wide_ok) {
        t = {kMaxVW, 0, false};
        while (t.width() < target && t.lpn_log2 < 5) ++t.lpn_log2;
    } else {
        t = walk_strided_tile(target);
    }
    const int64_t need = merge_scratch_bytes(n_units, n_dense, (int)sizeof(A));
    if (!workspace || workspace_bytes < need) {
        fsb_host::set_error("fsb_spmm_csr: workspace %lld bytes < %lld", (long long)workspace_bytes, (long long)need);
        return FSB_ERR_WORKSPACE;
    }
    const int64_t col_tiles = ceil_div(n_dense, (int64_t)t.width());
    const int64_t blocks = ceil_div(n_units, kSpmmThreads / 32);
    if (col_tiles > 65535 || blocks > 0x7fffffffLL) {
        fsb_host::set_error("fsb_spmm_csr: seq grid too large");
        return FSB_ERR_LIMIT;
    }
    MergeScratch ms = merge_scratch_carve(workspace, n_units, n_dense, (int)sizeof(A));
    A* cv = static_cast<A*>(ms.carry_val);
    A* hv = static_cast<A*>(ms.head_val);
    const int64_t grid = plan->grid_blocks > 0 && plan->grid_blocks < blocks ? plan->grid_blocks : blocks;
    const dim3 g((unsigned)grid, (unsigned)col_tiles);
    const bool in_kernel = plan->unit_runs && plan->tickets && plan->ticket_slots >= n_units * col_tiles;
    const int64_t* runs = in_kernel ? plan->unit_runs : nullptr;
    int* tickets = in_kernel ? reinterpret_cast<int*>(plan->tickets) : nullptr;
    const int ptr64 = Am->ptr_dtype == FSB_I64;
    const uint32_t ldb_bytes = (uint32_t)(ldb * (int64_t)sizeof(V)), ldc_bytes = (uint32_t)(ldc * (int64_t)sizeof(O));
    bool done = false;
#define FSB_WALK(W, L, S)                                                                                           \
    if (!done && t.vw == W && t.lpn_log2 == L && t.strided == S) {                                                   \
        launch_walk_one<V, A, O, I, W, S, L>(g, st, val, col, Am->row_ptr, ptr64, B, ldb_bytes, C, ldc_bytes,        \
                                             Am->n_rows, n_dense, plan->unit_coords, n_units, ms.carry_row, cv, hv, \
                                             runs, tickets);                                                         \
        done = true;                                                                                                 \
    }
#define FSB_WALK6(W, S)                                                                                          \
    FSB_WALK(W, 0, S) FSB_WALK(W, 1, S) FSB_WALK(W, 2, S) FSB_WALK(W, 3, S) FSB_WALK(W, 4, S) FSB_WALK(W, 5, S)
    if constexpr (kMaxVW > 1) {
        FSB_WALK6(kMaxVW, false)
    }
    FSB_WALK6(1, true)
    FSB_WALK(2, 5, true)
    FSB_WALK6(3, true)
    FSB_WALK(4, 5, true)
#undef FSB_WALK6
#undef FSB_WALK
    if (!done) {
        fsb_host::set_error("fsb_spmm_csr: no walk tile of %d x %d lanes", t.vw, 1 << t.lpn_log2);
        return FSB_ERR_INVALID;
    }
    int rc = fsb_host::check_launch("k_spmm_walk");
    if (rc || in_kernel) return rc;
    if (ptr64)
        k_spmm_merge_fixup<A, O, I, int64_t><<<fixup_grid(n_units, n_dense), kSpmmThreads, 0, st>>>(
            ms.carry_row, static_cast<const A*>(ms.carry_val), static_cast<const A*>(ms.head_val), n_units, n_dense,
            static_cast<const int64_t*>(Am->row_ptr), (const I*)nullptr, C, ldc);
    else
        k_spmm_merge_fixup<A, O, I, int32_t><<<fixup_grid(n_units, n_dense), kSpmmThreads, 0, st>>>(
            ms.carry_row, static_cast<const A*>(ms.carry_val), static_cast<const A*>(ms.head_val), n_units, n_dense,
            static_cast<const int32_t*>(Am->row_ptr), (const I*)nullptr, C, ldc);
    return fsb_host::check_launch("k_spmm_merge_fixup");
}

// Whether this form takes the call: 32-bit column numbers and row strides
// (rows of B are addressed as column x stride in 32 x 32 -> 64 bits), no
// compensated accumulator; the others run in k_spmm_seq.
inline bool walk_takes(const fsb_csr* A, int64_t ldb, int64_t ldc, int out_dtype, int acc_mode) {
    return acc_mode != FSB_ACC_COMP && !A->row_map && A->n_cols <= 0xffffffffLL &&
           ldb * (int64_t)elem_size(A->value_dtype) <= 0xffffffffLL &&
           ldc * (int64_t)elem_size(out_dtype) <= 0xffffffffLL;
}

template <class VSel>
int walk_dispatch_for(const fsb_csr* A, const void* B, int64_t ldb, int64_t n_dense, void* C, int64_t ldc,
                      int out_dtype, int acc_mode, const fsb_plan* plan, void* workspace, int64_t workspace_bytes,
                      cudaStream_t st) {
    return dispatch_vao(A->value_dtype, acc_mode, out_dtype, [&](auto tv, auto ta, auto to) -> int {
        using V = typename decltype(tv)::type;
        using Ac = typename decltype(ta)::type;
        using O = typename decltype(to)::type;
        if constexpr (!std::is_same<V, VSel>::value || is_comp_acc<Ac>::value) {
            return FSB_ERR_UNSUPPORTED;
        } else {
            return dispatch_idx(A->index_dtype, [&](auto ti) -> int {
                using I = typename decltype(ti)::type;
                if (A->ptr_dtype != FSB_I32 && A->ptr_dtype != FSB_I64) {
                    fsb_host::set_error("index dtype code %d is not int32/int64", A->ptr_dtype);
                    return FSB_ERR_UNSUPPORTED;
                }
                return launch_walk<V, Ac, O, I>(A, static_cast<const V*>(A->values), static_cast<const I*>(A->col_idx),
                                                static_cast<const V*>(B), ldb, n_dense, static_cast<O*>(C), ldc, plan,
                                                workspace, workspace_bytes, st);
            });
        }
    });
}

FSB_SEQ_DECL(walk_dispatch_f16);
FSB_SEQ_DECL(walk_dispatch_bf16);
FSB_SEQ_DECL(walk_dispatch_f32);
FSB_SEQ_DECL(walk_dispatch_f64);
FSB_SEQ_DECL(walk_dispatch_c32);
FSB_SEQ_DECL(walk_dispatch_c64);
FSB_SEQ_DECL(walk_dispatch_c128);

}  // namespace fsb
