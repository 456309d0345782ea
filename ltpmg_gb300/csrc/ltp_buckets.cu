// ltp_buckets.cu -- ordered-rule execution by buckets of cells.
//
// A batch under the ordered rule needs, per cell, the ops on it in (TID, op)
// order and nothing else, so the ops are split by a hash of their cell and
// every bucket is executed by one block in shared memory:
//
//   part    each block takes one tile of the batch: decodes and checks its
//           ops, ranks them by bucket in op order (per-warp counters in shared
//           memory) and writes the tile's records grouped by bucket into the
//           tile's own place, with the tile's bucket offsets -- no global
//           histogram, no look-back, no atomics per op
//   bucket  one block per bucket reads the bucket's run from every tile (so
//           its records arrive in op order), finds the distinct cells in a
//           shared-memory hash, reads each cell once, executes what is not
//           contended, resolves what is (compared by classes of hash slots,
//           or sorted and scanned) and writes each written cell once.  A
//           bucket longer than a chunk is executed chunk by chunk, the cells'
//           values carried in shared memory; a bucket with more distinct cells
//           than the hash holds is split into classes of cells.
//   solo    a batch of at most kSoloOps ops: the bucket kernel on the whole
//           batch, straight from its arrays, as one launch
//
// Against the conflict-word path (ltp_kernels.cu) there is no state per cell
// of the table to mark, scan and clear, each op's key and opword are read
// once, and a batch takes two launches (with the skew fallback's gate three)
// instead of eleven.  Measured on one GB300, per batch: 640 ops (a synchronous
// call, copies included) 77 -> 27 us; 17,000 to 270,000 ops in a list 64 -> 17
// us; 655,360 uniform ops over 2^20 x 10 cells 92 -> 42 us; 1.4 M order-entry
// ops with inserts 269 -> 186 us; 32,768 x 55 read-only ops with inserts 99 ->
// 78 us.  What bounds it: random sectors between the SMs and L2 -- per op one
// read of its cell, one atomic for the touched-word count and one store of its
// value (655,360 ops: 2.8 + 4.9 + 3.3 us at the measured rates, of 13 us in
// part and 34 in bucket) -- and, with two blocks of 512 threads per SM, the
// chain of their latencies.
#include <stdint.h>
#include <string.h>

#include <atomic>

#include "ltp_device.cuh"
#include "ltp_smem.h"
#include "ltp_trace.h"

namespace ltp {

namespace {

constexpr int kPartBlock = 512;
constexpr u32 kMaxTiles = 1024;
// odd multipliers: the golden ratio, the square roots of 3 and 7 (fractional parts)
constexpr u32 kMixMul = 0x9E3779B1u, kSlotMul = 0xBB67AE85u, kClassMul = 0xA54FF53Bu;

constexpr u32 inverse32(u32 a) {  // multiplicative inverse mod 2^32 (Newton)
    u32 x = a;
    for (int i = 0; i < 5; i++) x *= 2u - a * x;
    return x;
}
constexpr u32 kMixInv = inverse32(kMixMul);
static_assert(kMixInv * kMixMul == 1u, "kMixMul is odd");

constexpr u32 kSample = 8, kEarly = 32;  // see frequent_run
constexpr u32 kOpBits = 11;  // an op's place in its tile

// How a batch is split (host-made, passed by value).
struct BucketPlan {
    u64 *recs;           // [tiles * tile] records, grouped by bucket inside each tile: mixed
                         // cell number << 32 | add << 31 | increment << 11 | op's place in the tile
    uint16_t *offs;      // [tiles][buckets + 1] first record of each bucket in its tile
    PartCounters *ctr;   // [2], see PartState
    Counters *snap;      // where the batch's counters go
    PartState *state;
    u32 *epoch;          // [conflict words] stamp of the last batch that touched each word
    u32 *ins_pre;        // [insert tiles * LTP_MAX_TABLES]
    u32 cell_bits;       // cell numbers lie in [0, 2^cell_bits)
    u32 n_buckets, n_tiles, tile;
    u32 width;           // mixed cell numbers per bucket
    u64 width_inv;       // ceil(2^64 / width)
    u32 word_shift;      // cells per conflict word (statistics only)
    u32 limit;           // a batch with a bucket longer than this is left to the conflict-word path (0: none)
    u32 hot;             // a tile's run of one bucket longer than this counts towards the limit
    u32 often;           // a sampled tile's run longer than this speaks for a frequent cell
};

// Bijection on the cell numbers [0, 2^bits); equal parts of its range are the buckets.
__device__ __forceinline__ u32 low_mask(u32 bits) { return 0xFFFFFFFFu >> (32 - bits); }
__device__ __forceinline__ u32 mix_cell(u32 cell, u32 bits) { return (cell * kMixMul) & low_mask(bits); }
__device__ __forceinline__ u32 unmix_cell(u32 h, u32 bits) { return (h * kMixInv) & low_mask(bits); }

__device__ __forceinline__ int imm20(u32 x) { return (int)(x << 12) >> 12; }

// The tables as a block keeps them in shared memory: looking a cell's table
// up in the kernel's parameters costs a chain of indexed constant loads.
struct Tabs {
    char *data[LTP_MAX_TABLES];
    u64 rows_cap[LTP_MAX_TABLES], inv[LTP_MAX_TABLES], wide[LTP_MAX_TABLES];
    u32 base[LTP_MAX_TABLES], n_cols[LTP_MAX_TABLES];
    u32 n, top;  // top: first step of the search over base
};
__device__ __forceinline__ void load_tabs(const TablesDev &T, Tabs *s) {
    const u32 i = threadIdx.x;
    if (i < T.n) {
        const TableDev &t = T.t[i];
        s->data[i] = t.data;
        s->rows_cap[i] = t.rows_cap;
        s->inv[i] = t.inv;
        s->wide[i] = t.wide;
        s->base[i] = (u32)t.cell_base;
        s->n_cols[i] = t.n_cols;
    }
    if (i == 0) {
        s->n = T.n;
        s->top = T.n > 1 ? 1u << (31 - __clz((int)(T.n - 1))) : 0u;
    }
}

// A cell's address from its number (all cell numbers fit 32 bits here).
__device__ __forceinline__ char *cell_addr(const Tabs &T, u32 cell, bool *wide) {
    u32 k = 0;  // the last table with base <= cell
    for (u32 step = T.top; step; step >>= 1)
        if (k + step < T.n && T.base[k + step] <= cell) k += step;
    const u32 local = cell - T.base[k], nc = T.n_cols[k];
    // local / n_cols; inv = ceil(2^64 / n_cols) is exact for 32-bit numbers and up to 64 columns
    const u32 row = nc == 1u ? local : (u32)__umul64hi((u64)local, T.inv[k]), col = local - row * nc;
    const u64 wd = T.wide[k];
    *wide = (wd >> col) & 1ull;
    const u32 below = wd ? (u32)__popcll(wd & ((1ull << col) - 1ull)) : 0u;
    return T.data[k] + (T.rows_cap[k] * (col + below) + (*wide ? 2ull * row : (u64)row)) * 4;
}

// A read's or read-modify-write's cell, for a table of `rows` rows.
__device__ __forceinline__ bool op_cell(const TablesDev &T, const u64 *s_rows, u64 key, u32 w, u32 *cell) {
    const u32 tb = opw_table(w), col = opw_col(w);
    if (tb >= T.n || opw_kind(w) > LTP_OP_ADD) return false;
    const TableDev &t = T.t[tb];
    *cell = (u32)t.cell_base + (u32)key * t.n_cols + col;
    return key < s_rows[tb] && col < t.n_cols;
}

// An insert op's checks (it has no cell).
__device__ __forceinline__ bool insert_valid(const BatchDev &b, const TablesDev &T, u64 key, u64 i, u32 w) {
    const u32 tb = opw_table(w);
    return tb < T.n && payload_row_fits(key, insert_slots(T.t[tb]), b.payload_len) && insert_link_ok(b, T.t[tb], i, w);
}

__device__ __forceinline__ void set_bad(Counters *ctr, u64 i) {
    atomicMax(&ctr->bad_op, ~i);
    set_err(ctr, LTP_E_BADARG);
}

// Every transaction commits under the ordered rule: this block's share of
// the commit vector (parts = number of blocks that share the work).
__device__ __forceinline__ void commit_all(const BatchDev &b, u32 part, u32 parts) {
    const u64 nw = b.n_txns / 4, gsz = (u64)parts * blockDim.x;
    u32 *c = reinterpret_cast<u32 *>(b.commit);  // the batch's own allocation: aligned
    for (u64 j = (u64)part * blockDim.x + threadIdx.x; j < nw; j += gsz) c[j] = 0x01010101u;
    if (part == 0 && threadIdx.x < b.n_txns % 4) b.commit[nw * 4 + threadIdx.x] = 1;
}

template <typename X>
__device__ __forceinline__ void zero_words(X *x) {  // one block
    u32 *w = reinterpret_cast<u32 *>(x);
    for (u32 i = threadIdx.x; i < sizeof(X) / 4; i += blockDim.x) w[i] = 0u;
}

// Block-wide exclusive sum of one value per thread; *total is the sum over
// the block.  s_w: one word per warp; a barrier must separate two uses.
template <int NW>
__device__ __forceinline__ u32 block_excl(u32 v, u32 *s_w, u32 *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u32 incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const u32 y = __shfl_up_sync(FULL_MASK, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    u32 off = incl - v, all = 0;
#pragma unroll
    for (int w = 0; w < NW; w++) {
        const u32 x = s_w[w];
        if (w < warp) off += x;
        all += x;
    }
    *total = all;
    return off;
}

// ============================================================================
// part
// ============================================================================
size_t part_smem(u32 tile, u32 buckets) {
    // records, then per-warp bucket counters (two to a word)
    return (size_t)tile * 8 + (size_t)(kPartBlock / 32) * ((buckets + 1) / 2) * 4;
}

// A tile's run of more than hot records of one bucket.  Only these are added
// up: a bucket has at most tiles * hot <= limit / 2 records in its other runs,
// so it is within the limit while its long runs stay within limit / 2.
__device__ __forceinline__ void long_run(const BucketPlan &p, PartCounters *pc, u32 bucket, u32 len) {
    if (atomicAdd(&pc->total[bucket], len) + len > p.limit / 2) pc->skew = 1u;
}

// Every kSample'th tile's runs that are long against the mean: buckets with
// many of them are listed, to be executed first.  (All tiles' would be
// kSample times the atomics: 2% of 1.8 M reads with many frequent cells.)
__device__ __forceinline__ void frequent_run(PartCounters *pc, u32 bucket, u32 len) {
    const u32 old = atomicAdd(&pc->sample[bucket], len);
    if (old < kEarly && old + len >= kEarly) {
        const u32 at = atomicAdd(&pc->n_first, 1u);
        if (at < kMaxFirst) pc->first[at] = bucket;
    }
}

// Two blocks per SM, not three: a tile's ops are held in registers from their
// loads to the records, and at the 40 registers that three blocks leave they
// spill (order entry 468 -> 461 us, 32,768 x 55 read-only ops 164 -> 161 us,
// 65,536 x 10 with snapshots 173 -> 170 us).
template <int IPT>
__global__ void __launch_bounds__(kPartBlock, 2) k_part(BatchDev b, TablesDev T, BucketPlan p) {
    pdl_begin();
    constexpr int NW = kPartBlock / 32;
    constexpr u32 TILE = kPartBlock * IPT;
    static_assert(TILE <= 1u << kOpBits, "an op's place fits its field");
    static_assert(kInsTile % TILE == 0, "a tile lies inside one insert tile");
    const u32 B = p.n_buckets, BW = (B + 1) / 2, tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    u64 *stage = reinterpret_cast<u64 *>(ltp_dyn_smem);
    u32 *cnt = reinterpret_cast<u32 *>(stage + TILE);  // [NW][BW]
    __shared__ u32 s_ins[LTP_MAX_TABLES], s_wsum[NW], s_any;
    __shared__ u64 s_rows[LTP_MAX_TABLES];
    if (tid < T.n) s_rows[tid] = T.rows_now[tid];
    const u64 n = b.n_ops, base = (u64)blockIdx.x * TILE, wbase = base + (u64)warp * 32 * IPT;
    u64 key[IPT];
    u32 w[IPT];
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        const u64 i = wbase + (u64)k * 32 + lane;
        key[k] = i < n ? op_key_stream(b, i) : 0;
        w[k] = i < n ? __ldcs(&b.opw[i]) : 0xFFFFFFFFu;
    }
    const u32 stamp = p.state->stamp1, par = p.state->par1;
    PartCounters *pc = p.ctr + par;
    for (u32 i = tid; i < NW * BW; i += kPartBlock) cnt[i] = 0u;
    if (tid < LTP_MAX_TABLES) s_ins[tid] = 0u;
    if (tid == 0) s_any = 0u;
    if (blockIdx.x == 0) {  // the next batch's counters, this one's snapshot
        zero_words(p.ctr + (par ^ 1u));
        zero_words(p.snap);
        if (tid == 0) {
            p.state->stamp2 = stamp + 1u;
            p.state->par2 = par;
            p.state->skew = 0u;  // (set still after a fallback that gave up)
            p.state->joined = p.state->members = p.state->left = 0u;
            p.state->bar[0] = 0u;
        }
    }
    commit_all(b, blockIdx.x, gridDim.x);
    __syncthreads();
    u32 ins = 0;
#pragma unroll
    for (int k = 0; k < IPT; k++)
        if (wbase + (u64)k * 32 + lane < n && opw_kind(w[k]) == LTP_OP_INSERT) ins |= 1u << k;
    if (__any_sync(FULL_MASK, ins != 0u)) {
        // inserts: a link must name a read or read-modify-write before it in
        // its transaction.  Each of the three loads that takes is requested
        // for all rows at once (one row after another, they took a third of
        // the kernel on order entry), and before the cells are looked up, whose
        // registers they would need (order entry 375 -> 373 us, read-only ops
        // with inserts 163 -> 161, 65,536 x 10 with snapshots 169 -> 167).
        u32 tid_[IPT], linked[IPT], first[IPT];
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            const u64 i = wbase + (u64)k * 32 + lane;
            const u32 d = ins >> k & 1u ? insert_link(w[k]) : 0u;
            tid_[k] = d ? op_tid(b, i) : 0u;
            linked[k] = d && d <= i ? b.opw[i - d] : 0u;
        }
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            const bool on = (ins >> k & 1u) && insert_link(w[k]);
            first[k] = !on ? 0u : b.ops_per_txn ? tid_[k] * b.ops_per_txn : b.txn_first[tid_[k]];
        }
#pragma unroll
        for (int k = 0; k < IPT; k++)
            if (ins >> k & 1u) {
                const u64 i = wbase + (u64)k * 32 + lane;
                const u32 tb = opw_table(w[k]), d = insert_link(w[k]);
                bool ok = tb < T.n && payload_row_fits(key[k], insert_slots(T.t[tb]), b.payload_len);
                if (ok && d) ok = opw_col(w[k]) < T.t[tb].n_cols && d <= i && i - d >= first[k] && opw_kind(linked[k]) <= LTP_OP_ADD;
                if (ok) atomicAdd(&s_ins[tb], 1u);
                else set_bad(&pc->c, i);
            }
    }
    u64 rec[IPT];
    u32 bk[IPT];  // bucket, then bucket | rank << 16; ~0: no record
    bool any = false;
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        const u64 i = wbase + (u64)k * 32 + lane;
        bk[k] = 0xFFFFFFFFu;
        if (i >= n || (ins >> k & 1u)) continue;
        u32 cell;
        if (!op_cell(T, s_rows, key[k], w[k], &cell)) {
            set_bad(&pc->c, i);
            continue;
        }
        const u32 h = mix_cell(cell, p.cell_bits);
        const u32 add = opw_kind(w[k]) == LTP_OP_ADD;
        any |= add != 0u;
        bk[k] = (u32)__umul64hi((u64)h, p.width_inv);
        rec[k] = ((u64)h << 32) | (u64)(add << 31 | (add ? (w[k] >> 12) << kOpBits : 0u) | (u32)(i - base));
    }
    if (__any_sync(FULL_MASK, any) && lane == 0) s_any = 1u;
    // rank inside (warp, bucket), in op order: rows of 32 ops one after
    // another; a lane whose bucket gained one op has its rank at once, lanes
    // that share a bucket are ranked group by group (match.any over 32
    // different buckets takes about a thousand cycles a row)
    u32 *mine = cnt + (u32)warp * BW;
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        const bool v = bk[k] != 0xFFFFFFFFu;
        u32 *c = mine + (bk[k] >> 1);
        const u32 sh = (bk[k] & 1u) * 16u;
        u32 rank = v ? (*c >> sh) & 0xFFFFu : 0u;
        __syncwarp();
        if (v) atomicAdd(c, 1u << sh);
        __syncwarp();
        u32 shared = __ballot_sync(FULL_MASK, v && ((*c >> sh) & 0xFFFFu) - rank > 1u);
        while (shared) {
            const u32 lead = __shfl_sync(FULL_MASK, bk[k], __ffs(shared) - 1);
            const u32 peers = __ballot_sync(FULL_MASK, bk[k] == lead);
            if (bk[k] == lead) rank += (u32)__popc(peers & lanemask_lt());
            shared &= ~peers;
        }
        if (v) bk[k] |= rank << 16;
    }
    __syncthreads();
    // exclusive offsets: buckets in order, warps in order inside a bucket;
    // a thread owns pairs of buckets
    const u32 per = (BW + kPartBlock - 1) / kPartBlock, q0 = tid * per;
    u32 tot = 0;
    for (u32 q = q0; q < min(q0 + per, BW); q++) {
        u32 two = 0;  // both buckets' counts at once: neither reaches 2^16
#pragma unroll
        for (int wi = 0; wi < NW; wi++) two += cnt[wi * BW + q];
        tot += (two & 0xFFFFu) + (two >> 16);
    }
    u32 all;
    u32 run = block_excl<NW>(tot, s_wsum, &all);
    uint16_t *row = p.offs + (u64)blockIdx.x * (B + 1);
    const u32 often = blockIdx.x % kSample ? TILE : p.often;
    for (u32 q = q0; q < min(q0 + per, BW); q++) {
        u32 two = 0;
#pragma unroll
        for (int wi = 0; wi < NW; wi++) two += cnt[wi * BW + q];
        const u32 c0 = two & 0xFFFFu, c1 = two >> 16;
        u32 at = run | (run + c0) << 16;  // where the warp's records of the two buckets start
#pragma unroll
        for (int wi = 0; wi < NW; wi++) {
            const u32 x = cnt[wi * BW + q];
            cnt[wi * BW + q] = at;
            at += x;
        }
        row[2 * q] = (uint16_t)run;
        if (2 * q + 1 < B) row[2 * q + 1] = (uint16_t)(run + c0);
        if (c0 > p.hot) long_run(p, pc, 2 * q, c0);
        if (c1 > p.hot) long_run(p, pc, 2 * q + 1, c1);
        if (c0 > often) frequent_run(pc, 2 * q, c0);
        if (c1 > often) frequent_run(pc, 2 * q + 1, c1);
        run += c0 + c1;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IPT; k++)
        if (bk[k] != 0xFFFFFFFFu) {
            const u32 bb = bk[k] & 0xFFFFu;
            stage[((mine[bb >> 1] >> ((bb & 1u) * 16u)) & 0xFFFFu) + (bk[k] >> 16)] = rec[k];
        }
    if (tid < LTP_MAX_TABLES && s_ins[tid]) {
        atomicAdd(&pc->c.ins_total[tid], s_ins[tid]);
        atomicAdd(&p.ins_pre[(base / kInsTile) * LTP_MAX_TABLES + tid], s_ins[tid]);
    }
    if (tid == 0) {
        row[B] = (uint16_t)all;
        if (s_any) pc->writes = 1u;
    }
    __syncthreads();
    u64 *out = p.recs + base;
    for (u32 i = tid; i < all; i += kPartBlock) out[i] = stage[i];
}

// ============================================================================
// bucket
// ============================================================================
// A staged record: cell inside the bucket << 32 | add << 31 | increment << 11.
struct Rec {
    u32 lc;
    int imm;
    bool add;
};
constexpr u64 kNoRec = ~0ull;
__device__ __forceinline__ Rec unpack(u64 x) {
    const u32 lo = (u32)x;
    return Rec{(u32)(x >> 32), (int)(lo << 1) >> 12, (lo >> 31) != 0u};
}
// A contended op: slot << 52 | increment << 32 | op.
__device__ __forceinline__ u64 entry(u32 slot, int imm, u32 op) {
    return ((u64)(slot << 20 | ((u32)imm & 0xFFFFFu)) << 32) | op;
}

constexpr u32 kClassSlots = 8;  // neighbouring slots whose contended ops are compared with one another

template <int BLOCK_, int RPT_, int HB_, bool WIDE_>
struct Cfg {
    static constexpr int BLOCK = BLOCK_, RPT = RPT_, HB = HB_, NW = BLOCK / 32;
    static constexpr bool WIDE = WIDE_;
    static constexpr u32 HS = 1u << HB, CHUNK = (u32)BLOCK * RPT;
    static constexpr int DB = HB / 2;  // two radix passes over the slot number
    static constexpr u32 ND = 1u << DB;
    // insertions stop here: each thread may add one more before it sees the
    // count, and the probe loops need an empty slot to end on
    static constexpr u32 DISTINCT = HS - HS / 4;
    static constexpr u32 NC = HS / kClassSlots;  // classes of contended ops
    static_assert(NC <= (u32)BLOCK && NC < NW * ND, "a thread looks after a class");
    static_assert(DISTINCT + BLOCK <= HS && CHUNK < HS && ND <= (u32)BLOCK && NW <= 32 && RPT * NW <= 64 && HB == 12,
                  "layout");
    static constexpr u32 VB = WIDE ? 8 : 4;
    static constexpr u32 O_VAL = 0, O_CL = O_VAL + HS * VB, O_TAB = O_CL + 2 * CHUNK * 8, O_CNT = O_TAB + HS * 4,
                         O_OP = O_CNT + NW * ND * 4, BYTES_SOLO = O_OP, O_PRE = O_OP + CHUNK * 4,
                         BYTES = O_PRE + 2 * kMaxTiles * 4;
};
template <bool W>
struct ValT {
    typedef int V;
    typedef u32 S;
};
template <>
struct ValT<true> {
    typedef long long V;
    typedef u64 S;
};

constexpr u32 kEmpty = 0xFFFFFFFFu;
constexpr u32 kFew = 256;       // as many at most: the comparisons grow with the square
constexpr u32 kTiny = 64;       // so few in all are compared without classes
constexpr int kHotTries = 4;    // frequent cells of a long bucket's chunk that are scanned for themselves
// slot word: cell number << 3 | these
constexpr u32 kWritten = 1u, kMulti = 2u, kWideCell = 4u;

// An op's output from its cell's value, and the wrap of int32 cells.
template <class C, typename V>
__device__ __forceinline__ void put_out(const BatchDev &b, Counters *ctr, u32 op, V x, bool wide) {
    if (!LTP_IN_BOUNDS(ctr, op, b.n_ops)) return;
    b.out[op] = (int)x;
    if (C::WIDE && wide && b.out64) b.out64[op] = (long long)x;
}
template <class C, typename V>
__device__ __forceinline__ V narrow(V x, bool wide) {
    return C::WIDE && !wide ? (V)(int)x : x;
}

// Finds a cell's slot in the block's hash or takes one; *win: this op took it.
template <class C>
__device__ __forceinline__ u32 enter_cell(u32 *tab, u32 lc, bool add, bool *win) {
    const u32 want = add ? kWritten : 0u;
    u32 sl = (lc * kSlotMul) >> (32 - C::HB);
    for (;;) {
        u32 cur = tab[sl];  // (a hot cell's ops find it here: no atomic on one address)
        if (cur == kEmpty) {
            cur = atomicCAS(&tab[sl], kEmpty, (lc << 3) | want);
            if (cur == kEmpty) {
                *win = true;
                return sl;
            }
        }
        if ((cur >> 3) == lc) {
            if ((cur & (kMulti | want)) != (kMulti | want)) atomicOr(&tab[sl], kMulti | want);
            return sl;
        }
        sl = (sl + 1) & (C::HS - 1);
    }
}
__device__ __forceinline__ bool is_contended(u32 t) { return (t & (kWritten | kMulti)) == (kWritten | kMulti); }

template <class C>
struct Smem {
    typedef typename ValT<C::WIDE>::V V;
    unsigned char *sm;
    __device__ __forceinline__ Smem() : sm(reinterpret_cast<unsigned char *>(ltp_dyn_smem)) {}
    __device__ __forceinline__ V *val() const { return reinterpret_cast<V *>(sm + C::O_VAL); }
    __device__ __forceinline__ u64 *cl() const { return reinterpret_cast<u64 *>(sm + C::O_CL); }
    __device__ __forceinline__ u64 *stage() const { return cl() + C::CHUNK; }
    __device__ __forceinline__ u32 *tab() const { return reinterpret_cast<u32 *>(sm + C::O_TAB); }
    __device__ __forceinline__ u32 *cnt() const { return reinterpret_cast<u32 *>(sm + C::O_CNT); }
    __device__ __forceinline__ u32 *op() const { return reinterpret_cast<u32 *>(sm + C::O_OP); }    // ops of the staged records
    __device__ __forceinline__ u32 *pre() const { return reinterpret_cast<u32 *>(sm + C::O_PRE); }  // long buckets: [tiles],
    __device__ __forceinline__ u32 *adj() const { return pre() + kMaxTiles; }                       // [tiles], see TileSrc
};

// Exclusive sums of a per-row, per-warp value (row-major: the order of the
// staged records): s_row[k * NW + warp] in, offsets out; returns the total.
template <class C, typename X>
__device__ __forceinline__ X scan_rows(X *s_row, X *s_total) {
    const int lane = threadIdx.x & 31;
    __syncthreads();
    if (threadIdx.x < 32) {
        constexpr int N = C::RPT * C::NW, E = (N + 31) / 32;
        X x[E], sum = 0;
#pragma unroll
        for (int j = 0; j < E; j++) {
            const int i = lane * E + j;
            x[j] = i < N ? s_row[i] : (X)0;
            sum += x[j];
        }
        X incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const X y = __shfl_up_sync(FULL_MASK, incl, d);
            if (lane >= d) incl += y;
        }
        X run = incl - sum;
#pragma unroll
        for (int j = 0; j < E; j++) {
            const int i = lane * E + j;
            if (i < N) s_row[i] = run;
            run += x[j];
        }
        if (lane == 31) *s_total = incl;
    }
    __syncthreads();
    return *s_total;
}

// Executes rc contended ops that cl holds in op order: stable sort by slot
// (two passes, per-warp digit counters), segmented scan of the increments
// from val[slot]; done(slot, value) is called for the last op of every cell,
// after every value has been read.  Uses the stage.
template <class C, class Done>
__device__ __forceinline__ void run_sorted(const Smem<C> &m, const u32 rc, const BatchDev &b, Counters *ctr, Done done) {
    typedef typename ValT<C::WIDE>::V V;
    typedef typename ValT<C::WIDE>::S S;
    __shared__ u32 s_wsum[C::NW], s_dig[C::ND], s_wf[C::NW];
    __shared__ S s_ws[C::NW];
    const u32 tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    u64 *cl = m.cl();
    u32 *cnt = m.cnt(), *mine = cnt + (u32)warp * C::ND;
    const V *val = m.val();
    const u32 rows = (rc + C::BLOCK - 1) / C::BLOCK;
    const u32 w0 = (u32)warp * 32 * rows + lane;
    u64 e[C::RPT];
#pragma unroll
    for (int P = 0; P < 2; P++) {
        const u64 *from = cl + P * C::CHUNK;
        u64 *to = cl + (P ^ 1) * C::CHUNK;
        for (u32 i = tid; i < C::NW * C::ND; i += C::BLOCK) cnt[i] = 0u;
        __syncthreads();
        u32 rk[C::RPT];
#pragma unroll
        for (int k = 0; k < C::RPT; k++) {
            if ((u32)k >= rows) break;
            const u32 q = w0 + (u32)k * 32;
            const bool in = q < rc;
            e[k] = in ? from[q] : 0ull;
            const u32 d = (u32)(e[k] >> (52 + P * C::DB)) & (C::ND - 1);
            u32 peers = __ballot_sync(FULL_MASK, in);
#pragma unroll
            for (int bit = 0; bit < C::DB; bit++) {
                const u32 bm = __ballot_sync(FULL_MASK, d >> bit & 1u);
                peers &= d >> bit & 1u ? bm : ~bm;
            }
            const int ld = __ffs(peers) - 1;
            u32 old = 0;
            if (in && lane == ld) {
                old = mine[d];
                mine[d] = old + (u32)__popc(peers);
            }
            __syncwarp();
            rk[k] = __shfl_sync(FULL_MASK, old, ld & 31) + (u32)__popc(peers & lanemask_lt());
        }
        __syncthreads();
        u32 tot = 0, all;
        if (tid < C::ND) {
#pragma unroll
            for (int w = 0; w < C::NW; w++) {
                const u32 x = cnt[w * C::ND + tid];
                cnt[w * C::ND + tid] = tot;
                tot += x;
            }
        }
        const u32 off = block_excl<C::NW>(tot, s_wsum, &all);
        if (tid < C::ND) s_dig[tid] = off;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < C::RPT; k++) {
            if ((u32)k >= rows) break;
            if (w0 + (u32)k * 32 < rc) {
                const u32 d = (u32)(e[k] >> (52 + P * C::DB)) & (C::ND - 1);
                to[s_dig[d] + mine[d] + rk[k]] = e[k];
            }
        }
        __syncthreads();
    }
    S sv[C::RPT], cs = 0;
    u32 cf = 0, fl = 0, tails = 0;
#pragma unroll
    for (int k = 0; k < C::RPT; k++) {
        if ((u32)k >= rows) break;
        const u32 q = w0 + (u32)k * 32;
        const bool in = q < rc;
        e[k] = in ? cl[q] : 0ull;
        const u32 sl = (u32)(e[k] >> 52);
        const bool head = in && (q == 0 || (u32)(cl[q - 1] >> 52) != sl);
        if (in && (q + 1 == rc || (u32)(cl[q + 1] >> 52) != sl)) tails |= 1u << k;
        S sum = in ? (S)(V)imm20((u32)(e[k] >> 32)) : (S)0;
        u32 f = head;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const S us = __shfl_up_sync(FULL_MASK, sum, d);
            const u32 uf = __shfl_up_sync(FULL_MASK, f, d);
            if (lane >= d) {
                if (!f) sum += us;
                f |= uf;
            }
        }
        if (!f) sum += cs;
        f |= cf;
        sv[k] = sum;
        fl |= f << k;
        cs = __shfl_sync(FULL_MASK, sum, 31);
        cf = __shfl_sync(FULL_MASK, f, 31);
    }
    if (lane == 0) {
        s_wf[warp] = cf;
        s_ws[warp] = cs;
    }
    __syncthreads();
    S carry = 0;  // of the warps before: the sum since the last head
    for (int w = warp - 1; w >= 0; w--) {
        carry += s_ws[w];
        if (s_wf[w]) break;
    }
    V nv[C::RPT];
#pragma unroll
    for (int k = 0; k < C::RPT; k++) {
        if ((u32)k >= rows) break;
        if (w0 + (u32)k * 32 < rc) {
            const u32 sl = (u32)(e[k] >> 52);
            const bool wide = C::WIDE && (m.tab()[sl] & kWideCell);
            nv[k] = narrow<C>((V)((S)val[sl] + (fl >> k & 1u ? sv[k] : sv[k] + carry)), wide);
            put_out<C>(b, ctr, (u32)e[k], nv[k], wide);
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < C::RPT; k++) {
        if ((u32)k >= rows) break;
        if (tails >> k & 1u) done((u32)(e[k] >> 52), nv[k]);
    }
}

// The classes' counts (cnt, each op counted by its slot) become their first
// places; false if some class has more than kFew.
template <class C>
__device__ __forceinline__ bool class_starts(const Smem<C> &m) {
    __shared__ u32 s_wc[C::NW], s_big;
    const u32 tid = threadIdx.x;
    u32 *cnt = m.cnt(), rc;
    const u32 c = tid < C::NC ? cnt[tid] : 0u;
    if (tid == 0) s_big = 0u;
    const u32 off = block_excl<C::NW>(c, s_wc, &rc);
    if (c > kFew) s_big = 1u;
    if (tid < C::NC) cnt[tid] = off;
    if (tid == 0) cnt[C::NC] = rc;
    __syncthreads();
    return s_big == 0u;
}

// Executes the rc contended ops that cl holds class by class, in any order
// inside a class (WHOLE: in any order): each looks at its class, its cell's value is the sum over
// the ops on it up to its own.  done(slot, value) for the last op of every
// cell, AFTER: once every value has been read.
//
// Bound by instruction issue: all of a chunk's ops against all took a third of
// a block's time on order entry (250 ops: 13,000 cycles), by classes of eight
// slots an op meets a handful of others (order entry 461 -> 444 us, six
// batches of 327,680 ops in the pipeline 307 -> 276, 1.5 M uniform ops 92 ->
// 74; classes of sixteen the same).  The classes' scan costs two barriers: up
// to kTiny ops do without (3,000 ops 9.7 -> 9.2 us, uneven batches 207 -> 201
// us; 16 and 32: 207 and 204).
template <class C, bool AFTER, bool WHOLE, class Done>
__device__ __forceinline__ void compare(const Smem<C> &m, const u32 rc, const BatchDev &b, Counters *ctr, Done done) {
    typedef typename ValT<C::WIDE>::V V;
    typedef typename ValT<C::WIDE>::S S;
    const u64 *cl = m.cl();
    const u32 *cnt = m.cnt();
    V x[C::RPT];
    u32 last[C::RPT];
#pragma unroll
    for (int k = 0; k < C::RPT; k++) {
        const u32 q = (u32)k * C::BLOCK + threadIdx.x;
        last[k] = kEmpty;
        if (q >= rc) continue;
        const u64 me = cl[q];
        const u32 hi = (u32)(me >> 32) & 0xFFF00000u, sl = (u32)(me >> 52), op = (u32)me;
        const u32 to = WHOLE ? rc : cnt[sl / kClassSlots + 1];  // (of the last class: rc)
        bool later = false;
        int sum = 0;  // (256 increments of 20 bits)
#pragma unroll 4
        for (u32 j = WHOLE ? 0u : cnt[sl / kClassSlots]; j < to; j++) {
            const u64 o = cl[j];
            const u32 d = (u32)(o >> 32) - hi;  // same slot: the increment
            const bool same = d < 1u << 20, upto = (u32)o <= op;
            sum += same && upto ? imm20(d) : 0;
            later = later || (same && !upto);
        }
        const bool wd = C::WIDE && (m.tab()[sl] & kWideCell);
        x[k] = narrow<C>((V)((S)m.val()[sl] + (S)(V)sum), wd);
        put_out<C>(b, ctr, op, x[k], wd);
        if (later) continue;
        if (AFTER) last[k] = sl;
        else done(sl, x[k]);
    }
    if (AFTER) {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < C::RPT; k++)
            if (last[k] != kEmpty) done(last[k], x[k]);
    }
}

// Executes the R <= CHUNK records that are staged (op order; kNoRec: none).
// Adds this thread's share of the statistics.
template <class C, class Src>
__device__ __forceinline__ void exec_chunk(const Src &src, const u32 R, const BatchDev &b, const Tabs &T,
                                           const BucketPlan &p, Counters *ctr, const u32 stamp, u32 &n_tw, u32 &n_con,
                                           u32 &n_m) {
    typedef typename ValT<C::WIDE>::V V;
    typedef typename ValT<C::WIDE>::S S;
    const Smem<C> m;
    u32 *tab = m.tab();
    V *val = m.val();
    u64 *cl = m.cl();
    const u64 *stage = m.stage();
    u32 *cnt = m.cnt();
    __shared__ u32 s_con, s_at, s_row[C::RPT * C::NW], s_total;
    const u32 tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    if (tid < C::NC) cnt[tid] = 0u;
    if (tid == 0) s_con = s_at = 0u;
    for (u32 i = tid; i < C::HS / 4; i += C::BLOCK) reinterpret_cast<uint4 *>(tab)[i] = make_uint4(kEmpty, kEmpty, kEmpty, kEmpty);
    __syncthreads();
    // every op reads its cell while the hash is built: the value before the
    // batch, which is what all but the contended ops need
    u32 slot[C::RPT], old[C::RPT], won = 0, has = 0, wide = 0;
    V v[C::RPT];
    char *ptr[C::RPT];
#pragma unroll
    for (int k = 0; k < C::RPT; k++) {
        if ((u32)k * C::BLOCK >= R) break;
        const u32 q = (u32)k * C::BLOCK + tid;
        const u64 x = q < R ? stage[q] : kNoRec;
        if (x != kNoRec) {
            const Rec r = unpack(x);
            bool wd;
            const u32 cell = src.cell(r.lc);
            ptr[k] = cell_addr(T, cell, &wd);
            v[k] = (V)load_cell(ptr[k], C::WIDE && wd);
            has |= 1u << k;
            if (C::WIDE && wd) wide |= 1u << k;
            bool win = false;
            slot[k] = enter_cell<C>(tab, r.lc, r.add, &win);
            if (win) {
                won |= 1u << k;
                old[k] = atomicExch(&p.epoch[cell >> p.word_shift], stamp);
            }
        }
    }
    __syncthreads();
    u32 con = 0;
#pragma unroll
    for (int k = 0; k < C::RPT; k++) {
        if ((u32)k * C::BLOCK >= R) break;
        const u32 q = (u32)k * C::BLOCK + tid;
        if (!(has >> k & 1u)) continue;
        const Rec r = unpack(stage[q]);
        const bool wd = C::WIDE && (wide >> k & 1u);
        if (!is_contended(tab[slot[k]])) {  // the cell's only op, or one of its reads
            V x = v[k];
            if (r.add) {
                x = narrow<C>((V)((S)x + (S)(V)r.imm), wd);
                store_cell(ptr[k], wd, (long long)x);
            }
            put_out<C>(b, ctr, src.op(q), x, wd);
        } else {
            con |= 1u << k;
            if (won >> k & 1u) {
                val[slot[k]] = v[k];
                if (C::WIDE && wd) atomicOr(&tab[slot[k]], kWideCell);
                n_m++;
            }
            slot[k] |= atomicAdd(&cnt[slot[k] / kClassSlots], 1u) << C::HB;  // its rank in its class
        }
    }
    n_con += (u32)__popc(con);
    const u32 some = __reduce_add_sync(FULL_MASK, (u32)__popc(con));
    if (lane == 0 && some) atomicAdd(&s_con, some);
    __syncthreads();
    const u32 rc = s_con;
    auto store = [&](u32 sl, V x) {  // a contended cell's last value
        bool wd;
        char *a = cell_addr(T, src.cell(tab[sl] >> 3), &wd);
        store_cell(a, wd, (long long)x);
    };
    auto ent = [&](int k) {
        const u32 q = (u32)k * C::BLOCK + tid;
        return entry(slot[k] & (C::HS - 1), unpack(stage[q]).imm, src.op(q));
    };
    if (rc == 0) {
    } else if (rc <= kTiny) {
#pragma unroll
        for (int k = 0; k < C::RPT; k++)
            if (con >> k & 1u) cl[atomicAdd(&s_at, 1u)] = ent(k);
        __syncthreads();
        compare<C, false, true>(m, rc, b, ctr, store);
    } else if (class_starts<C>(m)) {
#pragma unroll
        for (int k = 0; k < C::RPT; k++)
            if (con >> k & 1u) cl[cnt[(slot[k] & (C::HS - 1)) / kClassSlots] + (slot[k] >> C::HB)] = ent(k);
        __syncthreads();
        compare<C, false, false>(m, rc, b, ctr, store);
    } else {
#pragma unroll
        for (int k = 0; k < C::RPT; k++) {
            const u32 bal = __ballot_sync(FULL_MASK, con >> k & 1u);
            if (lane == 0) s_row[k * C::NW + warp] = (u32)__popc(bal);
        }
        scan_rows<C>(s_row, &s_total);
#pragma unroll
        for (int k = 0; k < C::RPT; k++) {
            const bool cn = con >> k & 1u;
            const u32 bal = __ballot_sync(FULL_MASK, cn);
            if (cn) cl[s_row[k * C::NW + warp] + __popc(bal & lanemask_lt())] = ent(k);
        }
        run_sorted<C>(m, rc, b, ctr, store);
    }
#pragma unroll
    for (int k = 0; k < C::RPT; k++)
        if (won >> k & 1u) n_tw += old[k] != stamp;
}

// A bucket of more than CHUNK records (a hot cell's), chunk by chunk, the
// cells' values carried in shared memory and written back at the end.  The
// next chunk's records are requested before a chunk is executed.  Of a
// chunk's contended ops those on up to four cells that are frequent inside a
// warp are scanned by the whole block, cell by cell; what is left is compared
// by classes or sorted.  More
// distinct cells than the hash holds: class by class of cells, from the
// start (nothing but outputs, which come out the same, has been written).
// (Out of line, so that its registers don't spill those of the common case;
// by value, so that the kernel's parameters need no address.)
template <class C, class Src>
__device__ __noinline__ void exec_long(const Src src, const u32 R, const BatchDev b, const Tabs &T, const BucketPlan p,
                                       Counters *ctr, const u32 stamp, u32 *stats) {
    u32 n_tw = 0, n_con = 0, n_m = 0;
    typedef typename ValT<C::WIDE>::V V;
    typedef typename ValT<C::WIDE>::S S;
    static_assert(C::HS * 2 <= C::CHUNK * 4, "16-bit counts fit the ops' place");
    const Smem<C> m;
    u32 *tab = m.tab();
    V *val = m.val();
    u64 *cl = m.cl();
    // ops a cell had before it was contended, two 16-bit counts a word (a
    // longer bucket than 65535 is not executed here)
    u32 *count = m.op();
    u32 *cnt = m.cnt();
    __shared__ u32 s_distinct, s_con, s_cand[C::NW], s_row[C::RPT * C::NW], s_total;
    __shared__ S s_sum[C::RPT * C::NW], s_all;
    const u32 tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    u32 cbits = 0, cval = 0;  // the class of cells executed now: top cbits of their class hash == cval
    auto mine = [&](u32 lc) { return !cbits || ((lc * kClassMul) >> (32 - cbits)) == cval; };
    for (;;) {
        __syncthreads();
        for (u32 i = tid; i < C::HS; i += C::BLOCK) tab[i] = kEmpty;
        for (u32 i = tid; i < C::HS / 2; i += C::BLOCK) count[i] = 0u;
        if (tid == 0) s_distinct = 0u;
        u64 nx[C::RPT];
        u32 nt[C::RPT], contended = 0;  // contended: ops executed while their cell was known to be
        src.template request<C>(0, R, nx, nt);
        __syncthreads();
        bool over = false;
        for (u32 lo = 0; lo < R; lo += C::CHUNK) {
            Rec r[C::RPT];
            u32 op[C::RPT], slot[C::RPT], old[C::RPT], in = 0, won = 0, wide = 0;
            V v[C::RPT];
#pragma unroll
            for (int k = 0; k < C::RPT; k++)
                if (lo + (u32)k * C::BLOCK + tid < R) {
                    r[k] = unpack(nx[k] - ((u64)src.start << 32));
                    op[k] = nt[k] * src.tile + ((u32)nx[k] & ((1u << kOpBits) - 1u));
                    if (mine(r[k].lc)) in |= 1u << k;
                }
            src.template request<C>(lo + C::CHUNK, R, nx, nt);
            // ---- new cells, and their values before the batch ----
            if (tid == 0) s_con = 0u;
            if (tid < C::NC) cnt[tid] = 0u;
#pragma unroll
            for (int k = 0; k < C::RPT; k++) {
                bool win = false, add1 = false;
                slot[k] = 0;
                if ((in >> k & 1u) && *(volatile u32 *)&s_distinct < C::DISTINCT) {
                    slot[k] = enter_cell<C>(tab, r[k].lc, r[k].add, &win);
                    if (win) {
                        bool wd;
                        const u32 cell = src.cell(r[k].lc);
                        const char *a = cell_addr(T, cell, &wd);
                        v[k] = (V)load_cell(a, C::WIDE && wd);
                        old[k] = atomicExch(&p.epoch[cell >> p.word_shift], stamp);
                        won |= 1u << k;
                        if (C::WIDE && wd) wide |= 1u << k;
                    }
                    if (is_contended(tab[slot[k]])) contended++;
                    else add1 = true;
                }
                // an op on a cell not yet contended is counted there; the
                // first such op's cell for the whole warp
                const u32 some = __ballot_sync(FULL_MASK, add1);
                if (some) {
                    const int ld = __ffs(some) - 1;
                    const u32 first = __shfl_sync(FULL_MASK, slot[k], ld);
                    const u32 peers = __ballot_sync(FULL_MASK, add1 && slot[k] == first);
                    if (add1 && (lane == ld || !(peers >> lane & 1u)))
                        atomicAdd(&count[slot[k] >> 1], (lane == ld ? (u32)__popc(peers) : 1u) << (16 * (slot[k] & 1u)));
                }
                const u32 bal = __ballot_sync(FULL_MASK, win);
                if (lane == 0 && bal) atomicAdd(&s_distinct, (u32)__popc(bal));
            }
#pragma unroll
            for (int k = 0; k < C::RPT; k++)
                if (won >> k & 1u) {
                    val[slot[k]] = v[k];
                    if (C::WIDE && (wide >> k & 1u)) atomicOr(&tab[slot[k]], kWideCell);
                    n_tw += old[k] != stamp;
                }
            __syncthreads();
            if (s_distinct >= C::DISTINCT) {  // too many
                over = true;
                break;
            }
            // ---- ops on cells without a conflict so far; the others counted ----
            u32 con = 0, wd = 0, cand = kEmpty;
            V base[C::RPT];
#pragma unroll
            for (int k = 0; k < C::RPT; k++)
                if (in >> k & 1u) {
                    const u32 t = tab[slot[k]];
                    base[k] = val[slot[k]];
                    if (C::WIDE && (t & kWideCell)) wd |= 1u << k;
                    if (is_contended(t)) {
                        con |= 1u << k;
                        cand = slot[k];
                    } else {
                        V y = base[k];
                        if (r[k].add) {  // its first op
                            y = narrow<C>((V)((S)y + (S)(V)r[k].imm), t & kWideCell);
                            val[slot[k]] = y;
                        }
                        put_out<C>(b, ctr, op[k], y, t & kWideCell);
                    }
                }
            {
                const u32 c = __reduce_add_sync(FULL_MASK, (u32)__popc(con));
                const u32 some = __ballot_sync(FULL_MASK, con != 0u);
                cand = __shfl_sync(FULL_MASK, cand, some ? __ffs(some) - 1 : 0);
                u32 here = 0;
#pragma unroll
                for (int k = 0; k < C::RPT; k++) here += (con >> k & 1u) && slot[k] == cand;
                here = __reduce_add_sync(FULL_MASK, here);
                if (lane == 0) {
                    if (c) atomicAdd(&s_con, c);
                    s_cand[warp] = here >= kFew / C::NW ? cand : kEmpty;
                }
            }
            __syncthreads();
            u32 left = s_con;
            // ---- frequent cells: an ordered scan each ----
            int tries = 0;
#pragma unroll 1
            for (int h = 0; h < C::NW && tries < kHotTries && left > kFew; h++) {
                const u32 sl = s_cand[h];
                bool seen = sl == kEmpty;
                for (int j = 0; j < h; j++) seen = seen || s_cand[j] == sl;
                if (seen) continue;  // the same for the block
                tries++;
                S sum[C::RPT];
                u32 on = 0, rank[C::RPT];
#pragma unroll
                for (int k = 0; k < C::RPT; k++) {
                    const bool x = (con >> k & 1u) && slot[k] == sl;
                    if (x) on |= 1u << k;
                    sum[k] = x ? (S)(V)r[k].imm : (S)0;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const S y = __shfl_up_sync(FULL_MASK, sum[k], d);
                        if (lane >= d) sum[k] += y;
                    }
                    const u32 bal = __ballot_sync(FULL_MASK, x);
                    rank[k] = (u32)__popc(bal & lanemask_lt());
                    if (lane == 31) {
                        s_sum[k * C::NW + warp] = sum[k];
                        s_row[k * C::NW + warp] = (u32)__popc(bal);
                    }
                }
                scan_rows<C>(s_sum, &s_all);
                const u32 total = scan_rows<C>(s_row, &s_total);
#pragma unroll
                for (int k = 0; k < C::RPT; k++)
                    if (on >> k & 1u) {
                        const V y = narrow<C>((V)((S)base[k] + s_sum[k * C::NW + warp] + sum[k]), wd >> k & 1u);
                        put_out<C>(b, ctr, op[k], y, wd >> k & 1u);
                        if (s_row[k * C::NW + warp] + rank[k] + 1u == total) val[sl] = y;
                    }
                con &= ~on;
                left -= total;
                __syncthreads();
            }
            if (left) {
                u32 rank[C::RPT];
#pragma unroll
                for (int k = 0; k < C::RPT; k++)
                    if (con >> k & 1u) rank[k] = atomicAdd(&cnt[slot[k] / kClassSlots], 1u);
                __syncthreads();
                auto keep = [&](u32 sl, V y) { val[sl] = y; };
                if (class_starts<C>(m)) {
#pragma unroll
                    for (int k = 0; k < C::RPT; k++)
                        if (con >> k & 1u) cl[cnt[slot[k] / kClassSlots] + rank[k]] = entry(slot[k], r[k].imm, op[k]);
                    __syncthreads();
                    compare<C, true, false>(m, left, b, ctr, keep);
                } else {
#pragma unroll
                    for (int k = 0; k < C::RPT; k++) {
                        const u32 bal = __ballot_sync(FULL_MASK, con >> k & 1u);
                        if (lane == 0) s_row[k * C::NW + warp] = (u32)__popc(bal);
                    }
                    scan_rows<C>(s_row, &s_total);
#pragma unroll
                    for (int k = 0; k < C::RPT; k++) {
                        const bool cn = con >> k & 1u;
                        const u32 bal = __ballot_sync(FULL_MASK, cn);
                        if (cn) cl[s_row[k * C::NW + warp] + __popc(bal & lanemask_lt())] = entry(slot[k], r[k].imm, op[k]);
                    }
                    run_sorted<C>(m, left, b, ctr, keep);
                }
            }
            __syncthreads();
        }
        if (over) {  // half the class
            cbits++;
            cval <<= 1;
            continue;
        }
        n_con += contended;
        for (u32 i = tid; i < C::HS; i += C::BLOCK) {
            const u32 t = tab[i];
            if (t == kEmpty) continue;
            if (is_contended(t)) {
                n_m++;
                n_con += count[i >> 1] >> (16 * (i & 1u)) & 0xFFFFu;
            }
            if (t & kWritten) {
                bool wd;
                char *a = cell_addr(T, src.cell(t >> 3), &wd);
                store_cell(a, wd, (long long)val[i]);
            }
        }
        // the next class, if the cells were split: the sibling, else the parent's sibling
        cval++;
        while (cbits && !(cval & 1u)) {
            cval >>= 1;
            cbits--;
        }
        if (!cbits) break;
    }
    stats[0] = n_tw;
    stats[1] = n_con;
    stats[2] = n_m;
}

// Records of one bucket, tile by tile.
struct TileSrc {
    const u64 *recs;
    u32 *ops;              // ops of the staged records (shared memory)
    // long buckets (shared memory): records of the bucket before each tile,
    // and where its first one lies minus that
    const u32 *pre, *adj;
    u32 n_tiles, tile;
    u32 cell_bits, start;  // start: first mixed cell number of the bucket
    __device__ __forceinline__ u32 cell(u32 lc) const { return unmix_cell(start + lc, cell_bits); }
    __device__ __forceinline__ u32 op(u32 q) const { return ops[q]; }
    __device__ __forceinline__ void put(u64 *stage, u32 q, u64 x, u32 t) const {
        stage[q] = x - ((u64)start << 32);
        ops[q] = t * tile + ((u32)x & ((1u << kOpBits) - 1u));
    }
    // Requests record lo + q of a long bucket for q = k * BLOCK + thread
    // (below R in all); t: their tiles.  The warp finds its first record's
    // tile with two rounds of 32 comparisons, each lane walks on from there.
    template <class C>
    __device__ __forceinline__ void request(u32 lo, u32 R, u64 (&x)[C::RPT], u32 (&t)[C::RPT]) const {
        const u32 lane = threadIdx.x & 31;
#pragma unroll
        for (int k = 0; k < C::RPT; k++) {
            const u32 pos = lo + (u32)k * C::BLOCK + threadIdx.x, first = pos - lane;
            if (first >= R) break;  // the same for the warp
            const u32 g = (u32)__popc(__ballot_sync(FULL_MASK, lane * 32 < n_tiles && pre[lane * 32] <= first)) - 1u;
            const u32 i = g * 32 + lane;
            u32 at = g * 32 + (u32)__popc(__ballot_sync(FULL_MASK, i < n_tiles && pre[i] <= first)) - 1u;
            if (pos < R) {
                while (at + 1 < n_tiles && pre[at + 1] <= pos) at++;
                t[k] = at;
                x[k] = __ldcs(&recs[adj[at] + pos]);
            }
        }
    }
};

// Block-wide sums of the statistics into the batch's counters.
__device__ __forceinline__ void add_stats(Counters *ctr, u32 n_tw, u32 n_con, u32 n_m) {
    __shared__ u32 s_stat[3];
    if (threadIdx.x < 3) s_stat[threadIdx.x] = 0u;
    __syncthreads();
    n_tw = __reduce_add_sync(FULL_MASK, n_tw);
    n_con = __reduce_add_sync(FULL_MASK, n_con);
    n_m = __reduce_add_sync(FULL_MASK, n_m);
    if ((threadIdx.x & 31) == 0) {
        if (n_tw) atomicAdd(&s_stat[0], n_tw);
        if (n_con) atomicAdd(&s_stat[1], n_con);
        if (n_m) atomicAdd(&s_stat[2], n_m);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_stat[0]) atomicAdd(&ctr->n_tw, (u64)s_stat[0]);
        if (s_stat[1]) atomicAdd(&ctr->n_c, (u64)s_stat[1]);
        if (s_stat[2]) atomicAdd(&ctr->M, s_stat[2]);
    }
}

// Room for the batch's inserts?  (Every block comes to the same answer.)
__device__ __forceinline__ bool no_room(const TablesDev &T, const u32 *ins_total) {
    for (u32 t = 0; t < T.n; t++)
        if (ins_total[t] && T.rows_now[t] + ins_total[t] > T.t[t].row_limit) return true;
    return false;
}

// The insert tiles' counts become exclusive prefixes, table by table (one
// block; thread j scans a run of consecutive tiles).
template <int BLOCK>
__device__ __forceinline__ void ins_prefix(const BatchDev &b, const TablesDev &T, const BucketPlan &p, const Counters *ctr) {
    __shared__ u32 s_w[BLOCK / 32];
    const u64 tiles = (b.n_ops + kInsTile - 1) / kInsTile, per = (tiles + BLOCK - 1) / BLOCK;
    const u64 t0 = (u64)threadIdx.x * per, t1 = min(t0 + per, tiles);
    for (u32 tb = 0; tb < T.n; tb++) {
        if (!ctr->ins_total[tb]) continue;  // the same for every thread
        u32 sum = 0, all;
        for (u64 t = t0; t < t1; t++) sum += p.ins_pre[t * LTP_MAX_TABLES + tb];
        u32 run = block_excl<BLOCK / 32>(sum, s_w, &all);
        for (u64 t = t0; t < t1; t++) {
            const u32 c = p.ins_pre[t * LTP_MAX_TABLES + tb];
            p.ins_pre[t * LTP_MAX_TABLES + tb] = run;
            run += c;
        }
        __syncthreads();  // s_w is reused by the next table
    }
}

// A batch that writes no existing cell has nothing to order: every read
// takes its cell's value, in the batch's own order.
template <class C>
__device__ __forceinline__ void read_only(const BatchDev &b, const TablesDev &T, const BucketPlan &p, u32 stamp, u32 &n_tw) {
    constexpr int U = 4;
    const u64 n = b.n_ops, span = (u64)C::BLOCK * U;
    // words this block has stamped: a hot word is stamped once a block, not
    // once an op (the hash, direct-mapped)
    u32 *seen = Smem<C>().tab();
    for (u32 i = threadIdx.x; i < C::HS; i += C::BLOCK) seen[i] = kEmpty;
    __syncthreads();
    for (u64 base = (u64)blockIdx.x * span; base < n; base += (u64)p.n_buckets * span) {
        u64 key[U];
        u32 w[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
            const u64 i = base + (u64)k * C::BLOCK + threadIdx.x;
            key[k] = i < n ? op_key_stream(b, i) : 0;
            w[k] = i < n ? __ldcs(&b.opw[i]) : 0xFFFFFFFFu;
        }
        long long v[U];
        u32 old[U], ok = 0, wide = 0;
#pragma unroll
        for (int k = 0; k < U; k++) {
            const OpRef r = decode_op(T, key[k], w[k]);
            old[k] = stamp;
            if (r.valid) {
                ok |= 1u << k;
                if (r.wide) wide |= 1u << k;
                v[k] = load_cell(r.ptr, r.wide);
                const u32 word = (u32)r.cell >> p.word_shift;
                if (atomicExch(&seen[(word * kSlotMul) >> (32 - C::HB)], word) != word) old[k] = atomicExch(&p.epoch[word], stamp);
            }
        }
#pragma unroll
        for (int k = 0; k < U; k++)
            if (ok >> k & 1u) {
                const u64 i = base + (u64)k * C::BLOCK + threadIdx.x;
                __stcs(&b.out[i], (int)v[k]);
                if (C::WIDE && (wide >> k & 1u) && b.out64) b.out64[i] = v[k];
                n_tw += old[k] != stamp;
            }
    }
}

// The bucket of a block when some are listed to be executed first: the first
// blocks take the listed ones, whose own blocks take the buckets that the
// first ones left, in order.  (Full warps.)
__device__ __forceinline__ u32 first_order(const PartCounters *pc, u32 block) {
    static_assert(kMaxFirst == 32, "a lane per listed bucket");
    const u32 lane = threadIdx.x & 31, m = min(pc->n_first, kMaxFirst);
    const u32 h = lane < m ? pc->first[lane] : 0xFFFFFFFFu;
    // of the first m buckets those that are not listed; of the listed ones those beyond
    u32 left = ~__reduce_or_sync(FULL_MASK, h < 32u ? 1u << h : 0u) & (m == 32u ? FULL_MASK : (1u << m) - 1u);
    const u32 beyond = __ballot_sync(FULL_MASK, lane < m && h >= m), me = __ballot_sync(FULL_MASK, h == block);
    if (block < m) return __shfl_sync(FULL_MASK, h, (int)block);
    if (!me) return block;
    for (u32 k = (u32)__popc(beyond & (me - 1u)); k; k--) left &= left - 1u;
    return (u32)__ffs((int)left) - 1u;
}

// One block per bucket, two per SM: a block is a chain of latencies (offsets,
// records, cells, outputs) under which the other one executes.  A bucket with
// a frequent cell is several chunks long: started with the last wave, order
// entry's sixteen (5,000 records each) kept the kernel at 157 us for 1.4 M
// ops, started first 99 (the case 444 -> 372 us).
template <class C>
__global__ void __launch_bounds__(C::BLOCK, 2) k_bucket(BatchDev b, TablesDev T, BucketPlan p) {
    pdl_begin();
    const u32 tid = threadIdx.x;
    __shared__ u32 s_w[C::NW];
    __shared__ Tabs s_tabs;
    load_tabs(T, &s_tabs);
    // where the bucket's records lie: one column of the tiles' offsets.  A
    // thread looks at two tiles (of up to 1024); their first records are
    // requested before anything waits.
    constexpr int TPT = (int)kMaxTiles / C::BLOCK, PRE = 4;
    const bool extra = blockIdx.x == p.n_buckets;  // with inserts: one block more
    TileSrc src;
    src.recs = p.recs;
    src.ops = Smem<C>().op();
    src.pre = Smem<C>().pre();
    src.adj = Smem<C>().adj();
    src.n_tiles = p.n_tiles;
    src.tile = p.tile;
    const u32 per = (p.n_tiles + C::BLOCK - 1) / C::BLOCK;
    u32 at[TPT], cnt[TPT], len = 0, R, bucket = blockIdx.x;
    u64 x[TPT][PRE];
    auto column = [&]() {
        len = 0;
#pragma unroll
        for (int j = 0; j < TPT; j++) {
            const u32 t = tid * per + (u32)j;
            at[j] = cnt[j] = 0;
            if (!extra && (u32)j < per && t < p.n_tiles) {
                const uint16_t *o = p.offs + (u64)t * (p.n_buckets + 1) + bucket;
                at[j] = o[0];
                cnt[j] = o[1] - at[j];
            }
            len += cnt[j];
        }
    };
    column();
    // (kernel-uniform: nobody writes these now; both counters' flags, so that
    // the loads don't wait for one another)
    const u32 stamp = p.state->stamp2, par = p.state->par2;
    const u32 w0 = p.ctr[0].writes, w1 = p.ctr[1].writes, k0 = p.ctr[0].skew, k1 = p.ctr[1].skew;
    const u32 f0 = p.ctr[0].n_first, f1 = p.ctr[1].n_first;
    const int e0 = p.ctr[0].c.err, e1 = p.ctr[1].c.err;
    PartCounters *pc = p.ctr + par;
    const u32 writes = par ? w1 : w0, skew = writes && (par ? k1 : k0);
    const int err = par ? e1 : e0;
    if (par ? f1 : f0) {
        bucket = first_order(pc, bucket);
        if (bucket != blockIdx.x) column();
    }
#pragma unroll
    for (int j = 0; j < TPT; j++)
#pragma unroll
        for (int i = 0; i < PRE; i++)
            if (writes && (u32)i < cnt[j]) x[j][i] = __ldcs(&p.recs[(u64)(tid * per + (u32)j) * p.tile + at[j] + (u32)i]);
    const bool room = !b.payload_len || !no_room(T, pc->c.ins_total);
    if (blockIdx.x == 0 && tid == 0) {
        p.state->stamp1 = stamp;
        p.state->par1 = par ^ 1u;
        if (err) {
            p.snap->err = err;
            p.snap->bad_op = pc->c.bad_op;
        } else if (!room) {
            p.snap->err = LTP_E_CAPACITY;
            p.state->full = 1u;
        } else if (skew) {
            p.state->skew = 1u;  // left to the conflict-word path
        }
    }
    if (err || !room || skew) return;
    if (extra) {
        ins_prefix<C::BLOCK>(b, T, p, &pc->c);
        return;
    }
    u32 n_tw = 0, n_con = 0, n_m = 0;
    if (!writes) {
        read_only<C>(b, T, p, stamp, n_tw);
    } else {
        u32 pos = block_excl<C::NW>(len, s_w, &R);
        src.cell_bits = p.cell_bits;
        src.start = bucket * p.width;
        if (R > C::CHUNK) {
            u32 *pre = Smem<C>().pre(), *adj = Smem<C>().adj();
#pragma unroll
            for (int j = 0; j < TPT; j++) {
                const u32 t = tid * per + (u32)j;
                if ((u32)j < per && t < p.n_tiles) {
                    pre[t] = pos;
                    adj[t] = t * p.tile + at[j] - pos;
                    pos += cnt[j];
                }
            }
            u32 stats[3];
            exec_long<C>(src, R, b, s_tabs, p, p.snap, stamp, stats);
            n_tw = stats[0];
            n_con = stats[1];
            n_m = stats[2];
        } else if (R) {
            u64 *stage = Smem<C>().stage();
#pragma unroll
            for (int j = 0; j < TPT; j++) {
                const u32 t = tid * per + (u32)j;
#pragma unroll
                for (int i = 0; i < PRE; i++)
                    if ((u32)i < cnt[j]) src.put(stage, pos + (u32)i, x[j][i], t);
                const u64 *from = p.recs + (u64)t * p.tile + at[j];
                for (u32 i = PRE; i < cnt[j]; i += PRE) {
                    u64 y[PRE];
#pragma unroll
                    for (int q = 0; q < PRE; q++)
                        if (i + (u32)q < cnt[j]) y[q] = __ldcs(&from[i + (u32)q]);
#pragma unroll
                    for (int q = 0; q < PRE; q++)
                        if (i + (u32)q < cnt[j]) src.put(stage, pos + i + (u32)q, y[q], t);
                }
                pos += cnt[j];
            }
            exec_chunk<C>(src, R, b, s_tabs, p, p.snap, stamp, n_tw, n_con, n_m);
        }
    }
    add_stats(p.snap, n_tw, n_con, n_m);
}

struct BatchSrc {
    __device__ __forceinline__ u32 cell(u32 lc) const { return lc; }
    __device__ __forceinline__ u32 op(u32 q) const { return q; }
};

// The whole batch in one block, straight from its arrays.
template <class C>
__global__ void __launch_bounds__(C::BLOCK, 1) k_solo(BatchDev b, TablesDev T, BucketPlan p) {
    pdl_begin();
    __shared__ u32 s_ins[LTP_MAX_TABLES], s_fail[2], s_stat[3];
    __shared__ u64 s_rows[LTP_MAX_TABLES];
    __shared__ Tabs s_tabs;
    load_tabs(T, &s_tabs);
    const u32 tid = threadIdx.x, n = (u32)b.n_ops;
    u64 key[C::RPT];
    u32 w[C::RPT];
#pragma unroll
    for (int k = 0; k < C::RPT; k++) {
        const u32 i = (u32)k * C::BLOCK + tid;
        key[k] = i < n ? op_key(b, i) : 0;
        w[k] = i < n ? b.opw[i] : 0u;
    }
    if (tid < T.n) s_rows[tid] = T.rows_now[tid];
    if (tid < LTP_MAX_TABLES) s_ins[tid] = 0u;
    if (tid < 2) s_fail[tid] = 0u;
    if (tid < 3) s_stat[tid] = 0u;
    const u32 stamp = p.state->stamp1 + 1u, par = p.state->par1;
    commit_all(b, 0, 1);
    zero_words(p.snap);
    if (b.payload_len) zero_words(p.ctr + (par ^ 1u));
    __syncthreads();
    u64 *stage = Smem<C>().stage();
#pragma unroll
    for (int k = 0; k < C::RPT; k++) {
        const u32 i = (u32)k * C::BLOCK + tid;
        if (i >= n) break;
        u64 rec = kNoRec;
        u32 cell;
        if (opw_kind(w[k]) == LTP_OP_INSERT && insert_valid(b, T, key[k], i, w[k])) {
            atomicAdd(&s_ins[opw_table(w[k])], 1u);
        } else if (op_cell(T, s_rows, key[k], w[k], &cell)) {
            const u32 add = opw_kind(w[k]) == LTP_OP_ADD;
            rec = ((u64)cell << 32) | (u64)(add << 31 | (add ? (w[k] >> 12) << kOpBits : 0u));
        } else {
            s_fail[0] = 1u;
            atomicMax(&s_fail[1], ~i);
        }
        stage[i] = rec;
    }
    __syncthreads();
    u32 n_tw = 0, n_con = 0, n_m = 0;
    const bool full = b.payload_len && !s_fail[0] && no_room(T, s_ins);
    if (!s_fail[0] && !full) exec_chunk<C>(BatchSrc(), n, b, s_tabs, p, p.snap, stamp, n_tw, n_con, n_m);
    n_tw = __reduce_add_sync(FULL_MASK, n_tw);
    n_con = __reduce_add_sync(FULL_MASK, n_con);
    n_m = __reduce_add_sync(FULL_MASK, n_m);
    if ((tid & 31) == 0) {
        atomicAdd(&s_stat[0], n_tw);
        atomicAdd(&s_stat[1], n_con);
        atomicAdd(&s_stat[2], n_m);
    }
    __syncthreads();
    if (tid == 0) {
        p.snap->n_tw = s_stat[0];
        p.snap->n_c = s_stat[1];
        p.snap->M = s_stat[2];
        Counters *c = &p.ctr[par].c;
        if (s_fail[0]) {
            p.snap->err = LTP_E_BADARG;
            p.snap->bad_op = ~(u64)(u32)~s_fail[1];
            if (b.payload_len) c->err = LTP_E_BADARG;
        } else if (full) {
            p.snap->err = c->err = LTP_E_CAPACITY;
        }
        p.state->stamp1 = p.state->stamp2 = stamp;
        p.state->par2 = par;
        if (b.payload_len) p.state->par1 = par ^ 1u;
    }
    // (one insert tile: its prefix is zero already)
    if (b.payload_len && tid < LTP_MAX_TABLES) p.ctr[par].c.ins_total[tid] = s_ins[tid];
}

// After the inserts: the tables' row counts, clean insert counts.
__global__ void __launch_bounds__(1024) k_end(BatchDev b, TablesDev T, BucketPlan p) {
    pdl_begin();
    if (p.state->skew) return;  // the conflict-word path ends this batch
    const Counters *c = &p.ctr[p.state->par2].c;
    const u32 tid = threadIdx.x;
    if (tid < T.n && !c->err && !p.state->full) T.rows_now[tid] += c->ins_committed[tid];
    const u64 n = (b.n_ops + kInsTile - 1) / kInsTile * LTP_MAX_TABLES;
    for (u64 j = tid; j < n; j += blockDim.x) p.ins_pre[j] = 0u;
    __syncthreads();
    if (tid == 0) {
        p.state->full = 0u;
        // noted since the snapshot was taken (a bounds check of the row kernel)
        if (c->err && !p.snap->err) p.snap->err = c->err;
    }
}

// ============================================================================
// host side
// ============================================================================
u32 bits_for(u64 count) {  // bits that number `count` things, at least 1
    u32 b = 1;
    while (b < 64 && (1ull << b) < count) b++;
    return b;
}

template <class C>
cudaError_t go_solo(const Launch &L, const BatchDev &b, const TablesDev &T, const BucketPlan &p) {
    static std::atomic<uint64_t> done{0};
    cudaError_t e = allow_smem(k_solo<C>, C::BYTES_SOLO, done);
    if (e == cudaSuccess) e = launch_k(L.pdl, k_solo<C>, 1, C::BLOCK, C::BYTES_SOLO, L.stream, b, T, p);
    return e;
}

template <class C>
cudaError_t go_bucket(const Launch &L, const BatchDev &b, const TablesDev &T, const BucketPlan &p) {
    static std::atomic<uint64_t> done{0};
    cudaError_t e = allow_smem(k_bucket<C>, C::BYTES, done);
    const u32 grid = p.n_buckets + (b.payload_len ? 1u : 0u);
    if (e == cudaSuccess) e = launch_k(true, k_bucket<C>, grid, C::BLOCK, C::BYTES, L.stream, b, T, p);
    return e;
}

// (the two kernels of the split follow each other by dependent launch inside
// captured graphs too: +1.5% on 655,360-op batches; the insert kernel, whose
// blocks would take shared memory while the bucket kernel runs, does not)
template <int IPT>
cudaError_t go_part(const Launch &L, const BatchDev &b, const TablesDev &T, const BucketPlan &p) {
    static std::atomic<uint64_t> done{0};
    cudaError_t e = allow_smem(k_part<IPT>, part_smem(kPartBlock * IPT, kMaxBuckets), done);
    if (e == cudaSuccess)
        e = launch_k(true, k_part<IPT>, p.n_tiles, kPartBlock, part_smem(p.tile, p.n_buckets), L.stream, b, T, p);
    return e;
}

constexpr u64 kSoloSmall = 1024, kSoloOps = 2048;  // batches that one block executes
constexpr u64 kPartOps = 2ull << 20;               // largest batch that is split
constexpr u32 kBucketLimit = 32767;                // a longer bucket would keep one block busy for too long
constexpr u32 kMaxLcBits = 28;                     // the slot word holds a cell number and three flags

// Can the batch go this way, and how is it split?
bool plan_buckets(const Launch &L, const BatchDev &b, const TablesDev &T, const Scratch &s, Counters *snap, BucketPlan *p,
                  bool *solo) {
    if (L.rule == LTP_RULE_PRIORITY || L.stall || !s.pctr || T.n == 0 || b.n_ops == 0 || b.n_ops > kPartOps) return false;
    if (L.tune.flags & LTP_TUNE_CONFLICT_WORDS) return false;
    const TableDev &lt = T.t[T.n - 1];
    const u64 cells = lt.cell_base + lt.row_limit * lt.n_cols;
    const u32 cb = bits_for(cells), n = (u32)b.n_ops;
    if (cb > 32) return false;
    memset(p, 0, sizeof(*p));
    p->recs = s.list[0];
    p->offs = reinterpret_cast<uint16_t *>(s.list[1]);
    p->ctr = s.pctr;
    p->snap = snap;
    p->state = s.pstate;
    p->epoch = s.word_epoch;
    p->ins_pre = s.ins_pre;
    p->cell_bits = cb;
    p->word_shift = L.tune.word_bits == 64 && tiling_supported((int)L.tune.block, (int)L.tune.ipt, 64) ? 6 : 5;
    *solo = n <= kSoloOps && cb <= kMaxLcBits;
    if (*solo) return true;
    // Whole waves of two blocks per SM, their buckets well inside a chunk: a
    // small batch is spread over all of them too (65,536 Zipf ops a batch,
    // the request log: 304 buckets 550 us a pass, 128 buckets 575; 12 uneven
    // batches of 17,000 to 270,000 ops: 226 and 246 us)
    const u32 wave = 2u * (u32)L.num_sms;
    u32 nb = wave * ((n + wave * 1700 - 1) / (wave * 1700));
    if (cb > kMaxLcBits && nb < 1u << (cb - kMaxLcBits)) nb = 1u << (cb - kMaxLcBits);
    if (nb > 1u << (cb - 1)) nb = 1u << (cb - 1);
    p->width = (u32)(((1ull << cb) + nb - 1) / nb);
    if (p->width < 2) p->width = 2;
    nb = (u32)(((1ull << cb) + p->width - 1) / p->width);
    p->width_inv = ~0ull / p->width + 1ull;
    if (nb > kMaxBuckets || p->width > 1u << kMaxLcBits) return false;
    u32 tile = kPartBlock;
    while (tile < kPartBlock * 4 && (n + tile - 1) / tile > 160) tile <<= 1;
    p->n_buckets = nb;
    p->tile = tile;
    p->n_tiles = (n + tile - 1) / tile;
    p->limit = n > kBucketLimit ? kBucketLimit : 0;
    p->hot = p->limit ? kBucketLimit / 2 / p->n_tiles : tile;
    // Runs of more than twice the mean and five ops are rare by chance; within
    // one wave every bucket starts at once and none need be known.
    p->often = nb > wave ? 2 * tile / nb + 5 : tile;
    // the fallback counts touched words of 32 cells
    if (p->limit && p->word_shift != 5) return false;
    return p->n_tiles <= kMaxTiles && (u64)p->n_tiles * (nb + 1) * 2 <= s.cap_ops * 8 && (u64)p->n_tiles * tile <= s.cap_ops;
}

}  // namespace

bool launch_buckets(const Launch &L_in, const BatchDev &b_in, const TablesDev &T, const Scratch &s, Counters *snap,
                    cudaError_t *status) {
    BucketPlan p;
    bool solo = false;
    Launch L = L_in;
    BatchDev b = b_in;
    b.flags = L.tune.flags;
    if (!plan_buckets(L, b, T, s, snap, &p, &solo)) return false;
    TraceRange tr("launch bucket kernels");
    (void)cudaGetLastError();
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(L.stream, &cap);
    L.pdl = cap != cudaStreamCaptureStatusActive || b.n_ops < (1ull << 18);
    const unsigned ev_flags = cap == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : cudaEventRecordDefault;
    auto mark_ev = [&](int i) {
        if (L.timing) cudaEventRecordWithFlags(L.ev[i], L.stream, ev_flags);
        if (L.progress && i == L.progress_stage) cudaEventRecordWithFlags(L.progress, L.stream, ev_flags);
    };
    cudaError_t le = cudaSuccess;  // the first failed launch
    auto chk = [&](cudaError_t e) {
        if (le == cudaSuccess) le = e;
    };
    // stages: part counts as mark, bucket (or solo) as apply
    mark_ev(0);
    if (!solo) {
        switch (p.tile / kPartBlock) {
        case 1: chk(go_part<1>(L, b, T, p)); break;
        case 2: chk(go_part<2>(L, b, T, p)); break;
        default: chk(go_part<4>(L, b, T, p)); break;
        }
    }
    for (int i = 1; i <= 7; i++) mark_ev(i);
    if (solo) {
        if (b.n_ops <= kSoloSmall)
            chk(T.any_wide ? go_solo<Cfg<1024, 1, 12, true>>(L, b, T, p) : go_solo<Cfg<1024, 1, 12, false>>(L, b, T, p));
        else
            chk(T.any_wide ? go_solo<Cfg<1024, 2, 12, true>>(L, b, T, p) : go_solo<Cfg<1024, 2, 12, false>>(L, b, T, p));
    } else {
        chk(T.any_wide ? go_bucket<Cfg<512, 4, 12, true>>(L, b, T, p) : go_bucket<Cfg<512, 4, 12, false>>(L, b, T, p));
    }
    mark_ev(8);
    if (b.payload_len) {
        chk(launch_insert(L, b, T, s, &s.pctr->c, 1, s.pstate));
        mark_ev(9);
        chk(launch_k(L.pdl, k_end, 1, 1024, 0, L.stream, b, T, p));
    } else {
        mark_ev(9);
    }
    if (!solo && p.limit) chk(launch_fallback(L, b, T, s, snap));
    mark_ev(10);
    const cudaError_t e = cudaGetLastError();
    *status = le != cudaSuccess ? le : e;
    return true;
}

}  // namespace ltp
