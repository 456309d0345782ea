// ltp_device.cuh -- device helpers shared by the kernel translation units:
// bounded waits, look-back status words, table addressing, cache hints, op
// access and dependent launch.
#pragma once
#include <stdint.h>

#include "ltp_bounds.h"
#include "ltp_internal.cuh"

namespace ltp {

#define FULL_MASK 0xFFFFFFFFu

constexpr u64 kSpinLimitNs = 2000000000ull;  // 2 s per wait

// The dynamic shared memory of every kernel: the mark phase's tile hash and
// the insert phase's staging use it in turn.
extern __shared__ __align__(16) u32 ltp_dyn_smem[];

__device__ __forceinline__ u64 gtimer() {
    u64 t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ u64 ld_acquire(const u64 *p) {
    u64 v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(u64 *p, u64 v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ u32 ld_acquire32(const u32 *p) {
    u32 v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release32(u32 *p, u32 v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Look-back status words pack the flag and the value into one aligned word,
// so a reader that sees the flag sees the value: relaxed accesses suffice
// (no other data is published through them).
__device__ __forceinline__ u64 ld_status(const u64 *p) {
    u64 v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_status(u64 *p, u64 v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ u32 ld_status32(const u32 *p) {
    u32 v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_status32(u32 *p, u32 v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// The blocks among which a phase's work is spread: a launch's own, or those of
// them that take part.
struct Grid {
    u32 id, n;  // this block's number, their number
};
__device__ __forceinline__ Grid whole_grid() { return Grid{blockIdx.x, gridDim.x}; }

__device__ __forceinline__ u32 lanemask_lt() {
    u32 m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}
__device__ __forceinline__ void set_err(Counters *c, int e) { atomicCAS(&c->err, 0, e); }

// Debug builds (-DLTP_DEBUG_BOUNDS) check the index of every scatter into a
// scratch or table array, and of the conflict words, against the array's
// capacity: a violation records LTP_E_DEVICE_ASSERT and skips the access
// instead of trapping.  Release builds compile the checks away.
#ifdef LTP_DEBUG_BOUNDS
__device__ __forceinline__ bool in_bounds(Counters *ctr, u64 idx, u64 cap) {
    if (idx < cap) return true;
    set_err(ctr, LTP_E_DEVICE_ASSERT);
    return false;
}
#define LTP_IN_BOUNDS(ctr, idx, cap) in_bounds((ctr), (u64)(idx), (u64)(cap))
#else
#define LTP_IN_BOUNDS(ctr, idx, cap) true
#endif
__device__ __forceinline__ u64 mix64(u64 z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// One view of the device error word for the whole block: every thread takes
// the same early exit, so no barrier or full-warp collective is left short.
__device__ __forceinline__ bool block_err(Counters *ctr) {
    __shared__ int s_err;
    __syncthreads();
    if (threadIdx.x == 0) s_err = *(volatile int *)&ctr->err;
    __syncthreads();
    return s_err != 0;
}

// Claims the next tile for the whole block (tiles are handed out in order,
// which is what makes decoupled look-back safe without co-residency).
__device__ __forceinline__ u32 claim_tile(Counters *ctr, int slot) {
    __shared__ u32 s_tile;
    if (threadIdx.x == 0) s_tile = atomicAdd(&ctr->tile_ctr[slot], 1u);
    __syncthreads();
    u32 t = s_tile;
    __syncthreads();
    return t;
}

// ---- decoupled look-back, scalar sums (flag in bits 62-63) ---------------
constexpr u64 kAgg = 1ull << 62, kInc = 2ull << 62, kValMask = (1ull << 62) - 1;

// Publishes a tile's aggregate (tile 0: its inclusive prefix) early ...
__device__ __forceinline__ void lookback_publish(u64 *status, u32 tile, u64 agg) {
    st_status(&status[tile], (tile == 0 ? kInc : kAgg) | agg);
}
// ... and later walks back for the exclusive prefix, then publishes the
// inclusive one.  Bounded: gives up with LTP_E_TIMEOUT after 2 s.
__device__ __forceinline__ u64 lookback_wait(u64 *status, u32 tile, u64 agg, Counters *ctr) {
    constexpr int WIN = 4;  // predecessors read per round trip
    if (tile == 0) return 0;
    u64 excl = 0;
    long long t = (long long)tile - 1;
    const u64 t0 = gtimer();
    for (;;) {
        u64 st[WIN];
#pragma unroll
        for (int j = 0; j < WIN; j++) st[j] = t - j >= 0 ? ld_status(&status[t - j]) : kInc;
        int j = 0;
        bool done = false;
        for (; j < WIN; j++) {
            const u64 f = st[j] >> 62;
            if (f == 0) break;
            excl += st[j] & kValMask;
            if (f == 2) {
                done = true;
                break;
            }
        }
        if (done) break;
        t -= j;
        if (gtimer() - t0 > kSpinLimitNs) {
            set_err(ctr, LTP_E_TIMEOUT);
            return 0;
        }
    }
    st_status(&status[tile], kInc | (excl + agg));
    return excl;
}

// ---- table addressing ------------------------------------------------------
struct OpRef {
    u64 cell;
    char *ptr;
    bool valid;
    bool wide;
};

__device__ __forceinline__ OpRef decode_op(const TablesDev &T, u64 key, u32 w) {
    OpRef r;
    u32 tb = opw_table(w), col = opw_col(w), kind = opw_kind(w);
    r.valid = tb < T.n && kind <= 1u;
    const TableDev &t = T.t[r.valid ? tb : 0];
    r.valid = r.valid && key < T.rows_now[r.valid ? tb : 0] && col < t.n_cols;  // advanced by finish
    r.wide = r.valid && col_wide(t, col);
    r.cell = r.valid ? t.cell_base + key * t.n_cols + col : ~0ull;
    r.ptr = r.valid ? t.data + col_off(t, col) + key * (r.wide ? 8ull : 4ull) : nullptr;
    return r;
}

// Cell values are handled as 64-bit; int32 cells are sign-extended on load and
// truncated on store, which is exactly 32-bit two's-complement arithmetic.
// ---- L2 eviction-priority hints ---------------------------------------------
// Conflict words (the mark kernel's atomics) and their compact view (read
// by classify) are touched by every batch: keep them in L2.  Uncontended
// table cells are touched once: let them leave L2 first.
__device__ __forceinline__ u64 pol_evict_last() {
    u64 p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ u64 pol_evict_first() {
    u64 p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint4 ld_word_relaxed(const void *ptr) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(ptr)
                 : "memory");
    return v;
}
// Loads of scratch state with an L2 eviction-priority hint.  Coherent (not
// .nc): the persistent kernel writes this state and reads it again within one
// launch, where only the grid barrier's acquire orders the two, and the
// non-coherent path is defined only for data read-only for a whole kernel.
__device__ __forceinline__ uint4 ld_word_hint(const void *ptr, u64 pol) {
    uint4 v;
    asm volatile("ld.global.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(ptr), "l"(pol)
                 : "memory");
    return v;
}
// OR into a conflict word with an L2 eviction-priority hint: with the old
// value (atom) or without (red)
__device__ __forceinline__ u32 atom_or_hint(u32 *p, u32 v, u64 pol) {
    u32 old;
    asm volatile("atom.global.or.L2::cache_hint.b32 %0, [%1], %2, %3;" : "=r"(old) : "l"(p), "r"(v), "l"(pol) : "memory");
    return old;
}
__device__ __forceinline__ u64 atom_or_hint(u64 *p, u64 v, u64 pol) {
    u64 old;
    asm volatile("atom.global.or.L2::cache_hint.b64 %0, [%1], %2, %3;" : "=l"(old) : "l"(p), "l"(v), "l"(pol) : "memory");
    return old;
}
__device__ __forceinline__ void red_or_hint(u32 *p, u32 v, u64 pol) {
    asm volatile("red.global.or.L2::cache_hint.b32 [%0], %1, %2;" ::"l"(p), "r"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ void red_or_hint(u64 *p, u64 v, u64 pol) {
    asm volatile("red.global.or.L2::cache_hint.b64 [%0], %1, %2;" ::"l"(p), "l"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ void st_word_hint(void *ptr, uint4 v, u64 pol) {
    asm volatile("st.global.L2::cache_hint.v4.u32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(ptr), "r"(v.x), "r"(v.y), "r"(v.z),
                 "r"(v.w), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ uint2 ld_view_hint(const void *ptr, u64 pol) {
    uint2 v;
    asm volatile("ld.global.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;"
                 : "=r"(v.x), "=r"(v.y)
                 : "l"(ptr), "l"(pol)
                 : "memory");
    return v;
}
// ---- programmatic dependent launch -------------------------------------------
// The batch kernels are launched with programmatic stream serialization, so a
// kernel may be launched while its predecessor drains.  Each one first waits
// for the predecessor grid's completion and memory (griddepcontrol.wait; a
// no-op for a launch without the attribute), then lets its own successor be
// launched: the successor's launch and block placement overlap this kernel's
// run, and its blocks wait in turn before their first access.
__device__ __forceinline__ void pdl_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ long long load_cell_hint(const char *p, bool wide, u64 pol) {
    if (wide) {
        long long v;
        asm volatile("ld.global.L2::cache_hint.b64 %0, [%1], %2;" : "=l"(v) : "l"(p), "l"(pol) : "memory");
        return v;
    }
    int v;
    asm volatile("ld.global.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol) : "memory");
    return (long long)v;
}
__device__ __forceinline__ void store_cell_hint(char *p, bool wide, long long v, u64 pol) {
    if (wide) asm volatile("st.global.L2::cache_hint.b64 [%0], %1, %2;" ::"l"(p), "l"(v), "l"(pol) : "memory");
    else asm volatile("st.global.L2::cache_hint.b32 [%0], %1, %2;" ::"l"(p), "r"((int)v), "l"(pol) : "memory");
}

__device__ __forceinline__ long long load_cell(const char *p, bool wide) {
    return wide ? *reinterpret_cast<const long long *>(p) : (long long)*reinterpret_cast<const int32_t *>(p);
}
__device__ __forceinline__ void store_cell(char *p, bool wide, long long v) {
    if (wide) *reinterpret_cast<long long *>(p) = v;
    else *reinterpret_cast<int32_t *>(p) = (int32_t)v;
}
__device__ __forceinline__ void store_out(const BatchDev &b, u64 i, long long v) {
    b.out[i] = (int32_t)v;
    if (b.out64) b.out64[i] = v;
}

// Output of op i (a valid read or RMW) at full width: ops on int64 cells
// keep it in out64, ops on int32 cells only in out.
__device__ __forceinline__ long long op_value(const BatchDev &b, const TablesDev &T, u64 i) {
    const u32 w = b.opw[i], tb = opw_table(w);
    const bool wide = b.out64 && tb < T.n && col_wide(T.t[tb], opw_col(w));
    return wide ? b.out64[i] : (long long)b.out[i];
}

__device__ __forceinline__ char *cell_ptr(const TablesDev &T, u64 cell, bool *wide) {
    u32 k = 0;
    for (u32 i = 1; i < T.n; i++)
        if (cell >= T.t[i].cell_base) k = i;
    const TableDev &t = T.t[k];
    const u64 local = cell - t.cell_base;
    // 32-bit division whenever the table's cell numbers fit (the usual case)
    const u64 row = local < (1ull << 32) ? (u64)((u32)local / t.n_cols) : local / t.n_cols;
    const u32 col = (u32)(local - row * t.n_cols);
    *wide = col_wide(t, col);
    return t.data + col_off(t, col) + row * (*wide ? 8ull : 4ull);
}

__device__ __forceinline__ u32 op_tid(const BatchDev &b, u64 i);

// An insert's payload row holds one int32 slot per int32 column and two
// (low word first) per int64 column.
__device__ __forceinline__ u64 insert_slots(const TableDev &t) { return (u64)t.n_cols + (u64)__popcll(t.wide); }

// A linked insert (link distance d = low 10 bits of the immediate, d > 0)
// takes column `col` of its new row from the output of op i - d, which must
// be a read or read-modify-write of the same transaction.
__device__ __forceinline__ u32 insert_link(u32 w) { return (u32)opw_imm(w) & 0x3FFu; }
__device__ __forceinline__ bool insert_link_ok(const BatchDev &b, const TableDev &t, u64 i, u32 w) {
    const u32 d = insert_link(w);
    if (!d) return true;
    if (opw_col(w) >= t.n_cols || d > i) return false;
    const u32 tid = op_tid(b, i);
    // fixed-length batches carry ops_per_txn (their txn_first buffer is not loaded)
    const u64 first = b.ops_per_txn ? (u64)tid * b.ops_per_txn : (u64)b.txn_first[tid];
    return i - d >= first && opw_kind(b.opw[i - d]) <= LTP_OP_ADD;
}

// Key of op i (the batch carries 64-bit or 32-bit keys; the choice is
// uniform over the batch).
__device__ __forceinline__ u64 op_key(const BatchDev &b, u64 i) { return b.keys32 ? (u64)b.keys32[i] : b.keys[i]; }
__device__ __forceinline__ u64 op_key_stream(const BatchDev &b, u64 i) {  // read once: evict first
    return b.keys32 ? (u64)__ldcs(&b.keys32[i]) : __ldcs(&b.keys[i]);
}

__device__ __forceinline__ u32 op_tid(const BatchDev &b, u64 i) {
    return b.ops_per_txn ? (u32)(i / b.ops_per_txn) : b.op_txn[i];
}

// Launches a batch kernel, with programmatic stream serialization when `pdl`
// (see pdl_begin): it may start while its predecessor on the stream drains.
// The caller chooses: stream launches use it always; inside captured graphs
// the split and bucket kernels and the fallback do, the others in batches of
// fewer than 2^18 ops (see launch_execute and go_part).
template <typename... KP, typename... A>
static cudaError_t launch_k(bool pdl, void (*kernel)(KP...), unsigned grid, unsigned block, size_t smem,
                            cudaStream_t st, A... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, static_cast<KP>(args)...);
}

}  // namespace ltp
