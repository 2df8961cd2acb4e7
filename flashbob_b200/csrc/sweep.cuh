// One tiled "sweep" kernel for every stage of second-order attention on sm_100a.
//
// A CTA owns 128 rows of one side of the score matrix (query rows in the row-owned stages, key
// columns in the column-owned stages) and sweeps tiles of TN positions of the other side.  For
// each tile pair it
//   1. forms score-shaped products  own[128, D] x other[TN, D]^T  with tcgen05.mma into tensor
//      memory (fp32),
//   2. reads them back (one thread per own row and per 16-column slice), applies the mask and the
//      softmax recomputation from the saved log-sum-exp, builds the derived 16-bit operands and
//      writes them back into tensor memory (tcgen05.st),
//   3. accumulates output-shaped products  operand[128, TN] x other[TN, D]  (operand read from
//      tensor memory, swept tile MN-major from shared memory) into tensor memory accumulators
//      that live for the whole sweep.
// Column-owned stages compute the transposed scores (own = K-side), so the thread that owns key j
// holds column j of the score matrix and the operands come out already transposed; the per-query
// statistics then vary along the tensor-memory columns and are staged in shared memory.
//
// Warp roles: NG groups of 128*NSPLIT pointwise threads, and four role warps - a TMA warp, two that issue products (one
// the scores, as far ahead as accumulators are free, one the outputs, as operands arrive; a single elected thread
// runs the loop of each) and one that moves results.  Tiles of the other side sit in a ring of 2 to 8 tiles.  Work
// items (own tile x head x batch) are handed out longest first, either from a global counter (persistent launches) or
// one per CTA.
//
// The algebra follows the reference's second backward (reference: src/bob/kernels/common.py:15-30
// for the formulas, :463-654 for the row-owned tile body and epilogue, :661-786 for the
// column-owned tile body) and the usual flash-attention forward / first backward.
#pragma once

#include "ptx.cuh"

namespace bob {

#if defined(BOB_TRACE)
// Event trace (development builds only): the CTA with blockIdx.x == BOB_TRACE records (event id, SM
// clock) pairs of one pointwise thread (buffer 0) and the two MMA warps (buffers 1, 2);
// SweepParams::trace points to 4 x 8192 words.
#define BOB_TR_DECL(r) const int tr_role = (r); int tr_n = 0;
#define BOB_TR(i) { if (tr_role >= 0 && (lane == 0 || tr_role > 0) && MODE == BOB_TRACE_MODE && (int)blockIdx.x == BOB_TRACE && p.trace && tr_n < 8190) { p.trace[tr_role * 8192 + 1 + tr_n] = ((long long)(i) << 48) | (clock64() & 0xFFFFFFFFFFFFLL); ++tr_n; } }
#define BOB_TR_FLUSH if (tr_role >= 0 && (lane == 0 || tr_role > 0) && MODE == BOB_TRACE_MODE && (int)blockIdx.x == BOB_TRACE && p.trace) p.trace[tr_role * 8192] = tr_n;
#else
#define BOB_TR_DECL(r)
#define BOB_TR(i)
#define BOB_TR_FLUSH
#endif

enum Mode : int { kFwd = 0, kBwd1Row = 1, kBwd1Col = 2, kBwd2Row = 3, kBwd2Col = 4 };
enum TensorId : int { kTQ = 0, kTK, kTV, kTDO, kTUQ, kTUK, kTUV, kTOUT, kNumTensors };

// Status codes written to the status word by a CTA that gave up on a wait.
enum : int { kStatusOk = 0, kStatusTimeoutLoad = 11, kStatusTimeoutMma = 12, kStatusTimeoutPw = 13, kStatusMisaligned = 14 };

struct SweepParams {
    CUtensorMap map[kNumTensors];
    CUtensorMap res_map[3];       // results that leave through shared memory (SweepConfig::STAGED_OUT): res0, res1, pk
    // geometry
    int B, Hq, Hkv, G, Nq, Nk, D;
    int is_causal, window;
    int delta_off;                // q_offset - k_offset, clamped to +-2^29
    float scale;
    int has_uq, has_uk, has_uv;   // 0 = that tangent is undefined (treated as zero, products skipped)
    // global tensors read with plain loads (element strides: batch, head, row; unit head-dim stride)
    const void* out;  long long out_sb, out_sh, out_sn;    // first backward: only where a tile cannot be addressed (zero strides)
    const void* dQ;   long long dQ_sb, dQ_sh, dQ_sn;
    // fp32 row statistics, contiguous [B, Hq, Nq]
    float* lse;       // natural log
    float* delta;
    float* alpha;
    float* ecirc;
    // fp32 [B, Hq, Nq, D]: PK = P K, written by the first backward (may be null there: not needed
    // unless a second backward follows), read by the second backward's row-owned kernel
    float* pk;
    // results, contiguous [B, H, N, D] in the input dtype
    void* res0;
    void* res1;
    int* status;
    int* sticky;                  // optional second word that a CTA giving up also writes (host-visible memory)
    int* work_counter;            // persistent launches: next work item (zeroed by the host); null: one item per CTA
    long long* trace;             // development builds with BOB_TRACE
};

template <int MODE> struct ModeTraits;
template <> struct ModeTraits<kFwd>     { static constexpr int NOWN = 1, NOTH = 2, NSC = 1, NOUT = 1, NOPER = 1; static constexpr bool COL = false; };
template <> struct ModeTraits<kBwd1Row> { static constexpr int NOWN = 2, NOTH = 2, NSC = 2, NOUT = 2, NOPER = 2; static constexpr bool COL = false; };
template <> struct ModeTraits<kBwd1Col> { static constexpr int NOWN = 2, NOTH = 2, NSC = 2, NOUT = 2, NOPER = 2; static constexpr bool COL = true; };
template <> struct ModeTraits<kBwd2Row> { static constexpr int NOWN = 3, NOTH = 4, NSC = 4, NOUT = 2, NOPER = 4; static constexpr bool COL = false; };
template <> struct ModeTraits<kBwd2Col> { static constexpr int NOWN = 4, NOTH = 3, NSC = 4, NOUT = 2, NOPER = 3; static constexpr bool COL = true; };

// Which global tensor fills own slot / other slot `i` of a mode.
template <int MODE> __host__ __device__ constexpr int own_tensor(int i) {
    if (MODE == kFwd) return kTQ;
    if (MODE == kBwd1Row) return i == 0 ? kTQ : kTDO;
    if (MODE == kBwd1Col) return i == 0 ? kTK : kTV;
    if (MODE == kBwd2Row) return i == 0 ? kTQ : (i == 1 ? kTDO : kTUQ);
    return i == 0 ? kTK : (i == 1 ? kTV : (i == 2 ? kTUK : kTUV));
}
template <int MODE> __host__ __device__ constexpr int other_tensor(int i) {
    if (MODE == kFwd || MODE == kBwd1Row) return i == 0 ? kTK : kTV;
    if (MODE == kBwd1Col) return i == 0 ? kTQ : kTDO;
    if (MODE == kBwd2Row) return i == 0 ? kTK : (i == 1 ? kTUK : (i == 2 ? kTV : kTUV));   // K, uK adjacent; V, uV adjacent
    return i == 0 ? kTQ : (i == 1 ? kTUQ : kTDO);                                          // Q, uQ adjacent
}

// NG pointwise groups take the swept tiles in turn (group g: tiles g, g + NG, ... of an item), each with
// its own score accumulators and operand columns, so that one group's latencies (barriers, tensor-memory
// accesses) hide behind the other's arithmetic and the tensor pipe always has a tile to work on.  (In the
// forward each group also has its own output accumulator and online softmax.)
// CW: score columns per pointwise thread; TN / CW threads share a row.
// ALIAS: the derived operands overwrite the group's own score columns, 16 columns at a time (each thread
// only those it has read itself).  A group's next scores then wait for its output products; with two groups
// in turn the other one's products fill that time, and the tensor memory saved buys the second group.
template <int MODE, int DPAD, int TN, int NG, int CW, bool ALIAS>
struct SweepConfig {
    using MT = ModeTraits<MODE>;
    static constexpr bool BWD2 = MODE == kBwd2Row || MODE == kBwd2Col;
    static constexpr int NSPLIT = TN / CW;
    static constexpr int GP = 128 * NSPLIT;                // pointwise threads per group
    static constexpr int NPW = GP * NG;                    // pointwise threads
    static_assert(NPW == 256 || NPW == 512, "two or four pointwise warpgroups");
    static_assert(NG == 1 || NG == 2, "one or two pointwise groups");
    static_assert(MODE != kFwd || (NG == 2 && CW == TN), "forward: two groups, one thread per row");
    // One more warpgroup holds the role warps: score products, TMA producer, output products, results.
    // Two warps issue products because the queue in front of the tensor pipe is short (a few
    // instructions): while one warp is between two bursts - barriers, commits, loop - the other's
    // instructions keep the pipe busy.
    static constexpr int NTHREADS = NPW + 128;
    // Registers follow the work (setmaxnreg): the role warpgroup gives some up, the pointwise warpgroups
    // take them.  256 pointwise threads: 208 / 88 of 168 at launch (224 / 56 starves the role warps' issue
    // loops, measured 4 % slower); 512: 104 / 64 of 96.
    static constexpr int REGS_LAUNCH = NPW == 256 ? 168 : 96;
    static constexpr int REGS_POINTWISE = NPW == 256 ? 208 : 104;
    static constexpr int REGS_ROLE = NPW == 256 ? 88 : 64;
    static_assert(NPW * REGS_POINTWISE + 128 * REGS_ROLE <= NTHREADS * REGS_LAUNCH, "register trade must fit the launch's registers");
    // Row-owned second backward whose threads load all of a tile's columns at once: the score products are
    // ordered so that S, dP and C are complete before the last product (the second term of F) is issued,
    // and a barrier of its own tells the pointwise threads, whose loads of those three accumulators then run
    // under that last product (row-owned kernel 1.6-1.8 % faster; in the column-owned kernel it did not pay).
    static constexpr bool SPLIT_SC = MODE == kBwd2Row && NG == 1 && CW == 32;
    static constexpr int KSUB = DPAD / 64;                 // 64-element sub-tiles along the head dim
    static constexpr int OWN_TILE_BYTES = 128 * 128 * KSUB;
    // First backward, row-owned: the item's `out` rows come with its own tiles, for delta = rowsum(dO * out).
    static constexpr bool OWN_OUT = MODE == kBwd1Row;
    static constexpr int OWN_TILES = MT::NOWN + (OWN_OUT ? 1 : 0);
    // Swept tiles sit in a ring of slots.  A slot holds all tensors of a tile; in the forward, K and V tiles
    // take slots in turn (K is free again after the scores, V after the output product).
    static constexpr bool SPLIT_KV = MODE == kFwd;
    static constexpr int SLOT_TENSORS = SPLIT_KV ? 1 : MT::NOTH;
    static constexpr int SLOTS_PER_TILE = SPLIT_KV ? 2 : 1;
    static constexpr int OTH_SUB_BYTES = TN * 128;         // one 64-element-wide sub-tile of a swept tensor
    static constexpr int SLOT_BYTES = KSUB * SLOT_TENSORS * OTH_SUB_BYTES;    // laid out [sub][tensor]
    // tensor memory map: [score accumulators | derived 16-bit operands | output accumulators | own tile 0]
    static constexpr int SC_COLS = MT::NSC * TN;
    static constexpr int OPER_COLS_EACH = TN / 2;          // 128 x TN 16-bit values, two per 32-bit column
    static constexpr int OPER_COLS = ALIAS ? 0 : MT::NOPER * OPER_COLS_EACH;
    static constexpr int NACC = (MODE == kFwd) ? NG : MT::NOUT;
    static constexpr int OUT_COLS = NACC * DPAD;
    static constexpr int TMEM_BASE_NEED = NG * (SC_COLS + OPER_COLS) + OUT_COLS;
    // Second backward: where tensor memory has DPAD / 2 columns to spare, the first own tile (Q, or K
    // in the column-owned kernel) is also kept there, 16-bit packed like the derived operands, and its
    // score product reads it from tensor memory (measured at N = 64: 32 cycles per instruction against 48 with
    // both operands in shared memory).
    static constexpr bool OWN_TM = BWD2 && NG == 1 && DPAD == 128 && TMEM_BASE_NEED + DPAD / 2 <= 512;
    static constexpr int OWN_TM_COLS = OWN_TM ? DPAD / 2 : 0;
    static constexpr int TMEM_NEED = TMEM_BASE_NEED + OWN_TM_COLS;
    static constexpr int TMEM_COLS = TMEM_NEED <= 128 ? 128 : (TMEM_NEED <= 256 ? 256 : 512);
    static_assert(TMEM_NEED <= 512, "tensor memory budget exceeded");
    // Row-owned second backward at head dim <= 64: the epilogue's 16-bit global operands (out, dQ:
    // 16 KB each) are copied into shared memory with coalesced asynchronous copies while the item
    // runs, and the results leave through the same buffers with coalesced stores, both by the fourth role
    // warp.  The fp32 pk rows are read straight from global memory into registers when the sweep ends.
    static constexpr bool STAGED_IO = MODE == kBwd2Row && DPAD == 64;
    // Elsewhere the results are put into shared memory (128-byte swizzle, conflict-free) and leave by TMA
    // while the next item runs.  A thread owns one row of the result: storing it straight to global memory
    // touches 32 lines per instruction and kept the pointwise threads busy for 2000 (16-bit) to 4500 (with
    // fp32 pk) cycles per item.
    static constexpr bool STAGED_OUT = MODE <= kBwd1Col || (MODE == kBwd2Col && DPAD == 64);
    static constexpr bool STAGED_PK = MODE == kBwd1Row && DPAD == 64;          // (no room at head dim 128)
    static constexpr int N_STAGED = STAGED_OUT ? (MODE == kBwd1Col || MODE == kBwd2Col ? 2 : 1) : 0;
    static constexpr int IO_BYTES = STAGED_IO ? 32 * 1024 : N_STAGED * OWN_TILE_BYTES + (STAGED_PK ? DPAD * 512 : 0);
    // Where shared memory has no room for that (head dim 128: both results of the second backward, the epilogue
    // operands of its row-owned kernel, and pk of the first backward), eight lanes turn their eight rows' 128 bytes
    // around in registers, so that a warp-wide access touches 4 lines.  With a row per lane it touches 32, and the
    // row-owned second backward spent 19600 cycles between an item's last tile and the end of its epilogue (a tile
    // takes 1900), the column-owned one 7100, the first backward 9400; with the rows turned around 13900, 5000 and 6900
    // (kernels at H=32 S=2048: 184 to 174, 167 to 165 and 88 to 83 us).  The price is paid where an item has half a tile of
    // rows or less and so had few lines to touch: the second backward's two kernels over one such item per CTA take 14.4
    // and 12.2 us, against 12.4 and 10.4 with a row per lane (a full tile: 16.5 and 14.4 against 20.7 and 16.4).  Leaving out the
    // turns of warps without rows did not help (14.4), and slowed full tiles (18.4).
    static constexpr bool TURN_IO = BWD2 && DPAD == 128;
    static constexpr bool TURN_PK = MODE == kBwd1Row && !STAGED_PK;
    static_assert(!TURN_IO || DPAD / (NSPLIT * NG) == 64, "128 bytes of a 16-bit row per thread");
    static_assert(!TURN_PK || DPAD / (NSPLIT * NG) == 32, "128 bytes of an fp32 row per thread");
    // shared memory map (offsets from the 1024-byte aligned base)
    static constexpr int RED_COPIES = MODE == kBwd2Row && DPAD == 64 ? 2 : 1;
    static constexpr int RED_FLOATS = MODE == kFwd ? 8 * 128 : (MODE == kBwd1Row ? NG * NSPLIT * 128 : (MODE == kBwd2Row ? RED_COPIES * 2 * NG * NSPLIT * 128 : 0));
    static constexpr int NSTAT = MT::COL ? (BWD2 ? 4 : 2) : 0;                  // per-query statistics of a swept tile
    static constexpr int RING = 4;                                              // work items announced ahead
    static constexpr int MAX_SLOTS = 8;
    static constexpr int NBARS = 3 * MAX_SLOTS + 9 + 4 * NG + 2 * RING + (MODE == kFwd ? 8 : 0);
    static constexpr int MISC_BYTES = NBARS * 8 + 16 + 8 * RING;
    static constexpr int SMEM_LIMIT = 232448;
    static constexpr int SLOT_ROOM = (SMEM_LIMIT - OWN_TILES * OWN_TILE_BYTES - IO_BYTES - RED_FLOATS * 4 - MISC_BYTES) / (SLOT_BYTES + NSTAT * TN * 4);
    static constexpr int NSLOT = SLOT_ROOM >= MAX_SLOTS ? MAX_SLOTS : SLOT_ROOM;
    static_assert(SPLIT_KV ? NSLOT >= 2 * NG : NSLOT > NG, "score products run up to NG tiles ahead");
    static_assert(NG * SLOTS_PER_TILE <= NSLOT, "a group's step through the ring wraps at most once");
    static_assert(!ALIAS || 2 * SLOTS_PER_TILE <= NSLOT, "two tiles on, a tile's slot is at the earliest in use again");
    static constexpr int OFF_OWN = 0;
    static constexpr int OFF_OTH = OFF_OWN + OWN_TILES * OWN_TILE_BYTES;
    static constexpr int OFF_IO = OFF_OTH + NSLOT * SLOT_BYTES;                 // staged results / epilogue operands
    static constexpr int OFF_STAT = OFF_IO + IO_BYTES;                          // [NSLOT][NSTAT][TN] floats
    static constexpr int OFF_RED = OFF_STAT + NSLOT * NSTAT * TN * 4;
    static constexpr int OFF_BAR = OFF_RED + RED_FLOATS * 4;
    static constexpr int OFF_MISC = OFF_BAR + NBARS * 8;                        // tmem slot, item ring
    static constexpr int SMEM_BYTES = OFF_MISC + 16 + 8 * RING;
    static_assert(SMEM_BYTES <= SMEM_LIMIT, "shared memory budget exceeded");
    static_assert(OFF_OTH % 1024 == 0 && OFF_IO % 1024 == 0 && SLOT_BYTES % 1024 == 0, "swizzled tiles start on 1024-byte boundaries");
};

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <bool BF16>
__device__ __forceinline__ void unpack8_as_float(const uint4 a, float* v) {
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        if constexpr (BF16) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
            v[2 * i] = f.x; v[2 * i + 1] = f.y;
        } else {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
            v[2 * i] = f.x; v[2 * i + 1] = f.y;
        }
    }
}

// Transposes an 8 x 8 block of 16-byte chunks held by eight consecutive lanes (lane l: row l, chunks 0..7): afterwards
// lane l holds chunk l of rows 0..7, with which one warp-wide access touches four 128-byte lines instead of 32.
__device__ __forceinline__ void transpose_chunks(uint4 (&c)[8], int lane) {
    #pragma unroll
    for (int k = 1; k < 8; k <<= 1) {
        const bool up = (lane & k) != 0;
        #pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (i & k) continue;
            uint4 t = up ? c[i] : c[i | k];
            t.x = __shfl_xor_sync(0xffffffffu, t.x, k);
            t.y = __shfl_xor_sync(0xffffffffu, t.y, k);
            t.z = __shfl_xor_sync(0xffffffffu, t.z, k);
            t.w = __shfl_xor_sync(0xffffffffu, t.w, k);
            if (up) c[i] = t; else c[i | k] = t;
        }
    }
}

template <int V> struct IntTag { static constexpr int value = V; };

template <int MODE, int DPAD, int TN, bool BF16, int NG, int CW, bool ALIAS, bool ALLT = false>
__global__ void __launch_bounds__(SweepConfig<MODE, DPAD, TN, NG, CW, ALIAS>::NTHREADS, 1)
sweep_kernel(const __grid_constant__ SweepParams p) {
    static_assert(!ALLT || MODE == kBwd2Row || MODE == kBwd2Col, "only the second backward has tangents");
    using CFG = SweepConfig<MODE, DPAD, TN, NG, CW, ALIAS>;
    static_assert(CW == 16 || CW == 32 || CW == 48 || ((CW == 64 || CW == 128) && MODE == kFwd), "score columns per pointwise thread");
    using MT = ModeTraits<MODE>;
    constexpr int NSPLIT = CFG::NSPLIT, NPW = CFG::NPW, GP = CFG::GP, NSLOT = CFG::NSLOT, KSUB = CFG::KSUB;
    constexpr int SPT = CFG::SLOTS_PER_TILE;
    constexpr bool COL = MT::COL;
    constexpr bool BWD2 = CFG::BWD2;
    constexpr float kLog2e = 1.4426950408889634f;
    constexpr float kLn2 = 0.6931471805599453f;

    extern __shared__ __align__(1024) uint8_t sptr[];
    const uint32_t sbase = smem_u32(sptr);
    float* stat_buf = reinterpret_cast<float*>(sptr + CFG::OFF_STAT);
    float* red_buf = reinterpret_cast<float*>(sptr + CFG::OFF_RED);
    volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(sptr + CFG::OFF_MISC);  // [0] = tensor memory base
    const uint32_t bar0 = sbase + CFG::OFF_BAR;
    auto bar_full = [&](int s) { return bar0 + 8u * s; };                        // slot s: swept tile landed
    auto bar_empty = [&](int s) { return bar0 + 8u * (NSLOT + s); };             // slot s: its products have finished
    auto bar_stat = [&](int s) { return bar0 + 8u * (2 * NSLOT + s); };          // slot s: row statistics staged
    const uint32_t bar_misc0 = bar0 + 8u * 3 * NSLOT;
    const uint32_t bar_own = bar_misc0;                                          // own tiles landed
    const uint32_t bar_own_free = bar_misc0 + 8;                                 // own tiles no longer needed
    const uint32_t bar_done = bar_misc0 + 16;                                    // all products of the item have finished
    const uint32_t bar_pw_all = bar_misc0 + 24;                                  // all pointwise threads
    const uint32_t bar_out_free = bar_misc0 + 32;                                // output accumulators read out
    const uint32_t bar_own_tm = bar_misc0 + 40;                                  // own tile 0 copied into tensor memory
    const uint32_t bar_io_full = bar_misc0 + 48;                                 // STAGED_IO: out / dQ rows staged
    const uint32_t bar_io_ready = bar_misc0 + 56;                                // the item's results are in shared memory
    const uint32_t bar_io_free = bar_misc0 + 64;                                 // STAGED_OUT: ... and have been read from there
    const uint32_t bar_grp0 = bar_misc0 + 72;                                    // per group:
    auto bar_sc_full = [&](int g) { return bar_grp0 + 32u * g; };               //   scores ready
    auto bar_sc_empty = [&](int g) { return bar_grp0 + 32u * g + 8; };          //   scores read (not ALIAS)
    auto bar_op_full = [&](int g) { return bar_grp0 + 32u * g + 16; };          //   operands written
    auto bar_sc_part = [&](int g) { return bar_grp0 + 32u * g + 24; };          //   S, dP, C ready (SPLIT_SC)
    const uint32_t bar_ring0 = bar_grp0 + 32u * NG;
    auto bar_item_full = [&](int s) { return bar_ring0 + 8u * s; };             // ring slot announced
    auto bar_item_empty = [&](int s) { return bar_ring0 + 8u * (CFG::RING + s); };   // ring slot read by every follower
    auto bar_exp = [&](int g) { return bar_ring0 + 8u * (2 * CFG::RING + 4 * g + ((threadIdx.x >> 5) & 3)); };   // forward: see tile_body
    // Parity: a wait for the phase before a barrier's first one returns at once, so the "free" barriers that
    // are passed once per use need no special case for the first.

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;

    // ---- work items ----------------------------------------------------------------------------
    // One item = one own tile of one head of one batch element, swept over the other side.  Items
    // are numbered longest-sweep-first (all heads' heaviest tile, then all heads' second heaviest,
    // ...).  Persistent launches (more items than SMs) take them from a counter; a CTA keeps its tensor
    // memory and barriers across items, and every role runs ahead of the next one into the next item.
    const int n_own = COL ? p.Nk : p.Nq;
    const int n_oth = COL ? p.Nq : p.Nk;
    const int n_own_tiles = (n_own + 127) / 128;
    const int grid_heads = COL ? p.Hkv : p.Hq;
    const int per_rank = grid_heads * p.B;
    const int n_items = n_own_tiles * per_rank;
    const int n_outer = COL ? p.G : 1;
    const int doff = p.delta_off;                // q_offset - k_offset, within +-2^29 (see the host's fill_mask)
    // kernel parameters that the per-tile code needs, read once
    const bool causal = p.is_causal != 0;
    const int window = p.window;
    // ALLT (second backward): all three tangents are defined, the usual case.  Their flags are then
    // compile-time constants, so the loads and arithmetic of F and C are unconditional instead of
    // predicated on values only known at run time.
    const bool has_uq = ALLT || p.has_uq != 0, has_uk = ALLT || p.has_uk != 0, has_uv = ALLT || p.has_uv != 0;
    struct Item { int own0, head, batch, kv_head, t_lo, t_hi, T, total; };
    auto decode = [&](int item) {
        Item w;
        const int tile_rank = item / per_rank;
        const int rem = item % per_rank;
        w.head = rem % grid_heads;               // query head (row-owned) or KV head (column-owned)
        w.batch = rem / grid_heads;
        // causal: row-owned sweeps grow with the row index, column-owned ones shrink with the column
        const int own_tile = (!COL && causal) ? (n_own_tiles - 1 - tile_rank) : tile_rank;
        w.own0 = own_tile * 128;
        w.kv_head = COL ? w.head : w.head / p.G;
        int lo = 0, hi = n_oth;                  // other-side positions [lo, hi) that can be unmasked
        const int own_last = min(w.own0 + 127, n_own - 1);
        // (lengths are at most 2^28, |doff| 2^29 and the window 2^30: 32-bit sums cannot overflow)
        if (causal) {
            if (!COL) {
                hi = min(n_oth, own_last + doff + 1);
                if (window > 0) lo = max(0, w.own0 + doff - window + 1);
            } else {
                lo = max(0, w.own0 - doff);
                if (window > 0) hi = min(n_oth, own_last - doff + window);
            }
        }
        w.t_lo = (hi > lo) ? lo / TN : 0;
        w.t_hi = (hi > lo) ? (hi + TN - 1) / TN : 0;
        w.T = w.t_hi - w.t_lo;
        w.total = w.T * n_outer;
        return w;
    };
    constexpr int RING = CFG::RING;
    volatile int* item_ring = reinterpret_cast<volatile int*>(sptr + CFG::OFF_MISC + 16);
#define BOB_ITEM_LOCALS(w)                                                                         \
    const int own0 = (w).own0, head = (w).head, batch = (w).batch, kv_head = (w).kv_head;         \
    const int t_lo = (w).t_lo, t_hi = (w).t_hi, total = (w).total;                                 \
    (void)own0; (void)head; (void)batch; (void)kv_head; (void)t_lo; (void)t_hi; (void)total;

    auto give_up = [&](int code) {
        atomicCAS(p.status, 0, code);
        if (p.sticky) { *reinterpret_cast<volatile int*>(p.sticky) = code; __threadfence_system(); }
    };
    if (sbase & 1023u) {                         // every swizzled tile relies on it
        if (tid == 0) give_up(kStatusMisaligned);
        return;
    }

    auto has_tensor = [&](int t) {
        if (CFG::OWN_OUT && t == kTOUT) return p.out == nullptr;     // otherwise read with plain loads
        return t == kTUQ ? has_uq : (t == kTUK ? has_uk : (t == kTUV ? has_uv : true));
    };

    // -lse in log2 units.  A row without keys has lse = -inf: kept finite, so that its scores, all masked to -inf, still
    // give probability zero.
    auto neg_log2 = [](float lse) { return lse == -INFINITY ? 3.0e38f : -lse * kLog2e; };

    // ---- set-up ------------------------------------------------------------------------------
    if (tid == 0) {
        for (int s = 0; s < NSLOT; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); mbar_init(bar_stat(s), 32); }
        for (int g = 0; g < NG; ++g) {
            mbar_init(bar_sc_full(g), 1);
            mbar_init(bar_sc_part(g), 1);
            mbar_init(bar_sc_empty(g), GP / 32);
            mbar_init(bar_op_full(g), GP / 32);
        }
        mbar_init(bar_own, 1);
        // the last score products and, where they read the own tiles too, the pointwise threads
        mbar_init(bar_own_free, 1 + (CFG::OWN_OUT || CFG::OWN_TM ? NPW / 32 : 0));
        mbar_init(bar_done, 1);
        mbar_init(bar_pw_all, NPW / 32);
        mbar_init(bar_out_free, NPW / 32);
        for (int s = 0; s < RING; ++s) { mbar_init(bar_item_full(s), 1); mbar_init(bar_item_empty(s), 2 + (CFG::STAGED_IO || CFG::STAGED_OUT ? 1 : 0) + NPW / 32); }
        mbar_init(bar_own_tm, NPW / 32);
        mbar_init(bar_io_full, 1);
        mbar_init(bar_io_ready, NPW / 32);
        mbar_init(bar_io_free, 1);
        if constexpr (MODE == kFwd) { for (int i = 0; i < 8; ++i) mbar_init(bar_ring0 + 8u * (2 * RING + i), 1); }
        mbar_fence_init();
    }
    if (warp == NPW / 32) {
        tmem_alloc(sbase + CFG::OFF_MISC, CFG::TMEM_COLS);
        tmem_relinquish();
    }
    if (warp == NPW / 32 + 1) {                  // the tensor maps, while the others set up
        bool used = false;
        #pragma unroll
        for (int i = 0; i < CFG::OWN_TILES; ++i) used = used || lane == (i < MT::NOWN ? own_tensor<MODE>(i) : (int)kTOUT);
        #pragma unroll
        for (int i = 0; i < MT::NOTH; ++i) used = used || lane == other_tensor<MODE>(i);
        if (used && has_tensor(lane)) tma_prefetch_desc(&p.map[lane]);
        if (lane >= 16 && lane < 16 + CFG::N_STAGED) tma_prefetch_desc(&p.res_map[lane - 16]);
        if (CFG::STAGED_PK && lane == 20 && p.pk) tma_prefetch_desc(&p.res_map[2]);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, misc[0], 0);      // warp-uniform, and known to be
    const uint32_t tmem_oper = tmem + NG * CFG::SC_COLS;
    const uint32_t tmem_out = tmem_oper + NG * CFG::OPER_COLS;
    const uint32_t tmem_own = tmem_out + CFG::OUT_COLS;                          // own tile 0, packed (OWN_TM only)
    (void)tmem_own;

    // Bounded wait of the per-tile loops.  The control flow after it does not depend on the outcome: a wait
    // that runs out is recorded, and from then on this thread's waits return at once, so its loops end on
    // their own (the results of the call are undefined).
    bool dead = false;
    auto wait = [&](uint32_t bar, uint32_t parity, int code) {
        if (!mbar_try_wait(bar, parity)) {
            if (!dead && !mbar_wait(bar, parity)) { dead = true; give_up(code); }
        }
        __syncwarp();
    };
    auto wait_alone = [&](uint32_t bar, uint32_t parity, int code) {             // the same for a single thread
        if (!mbar_try_wait(bar, parity)) {
            if (!dead && !mbar_wait(bar, parity)) { dead = true; give_up(code); }
        }
    };
    auto follow_ring_alone = [&](int k) -> int {
        const int slot = k % RING;
        if (dead || !mbar_wait(bar_item_full(slot), (k / RING) & 1)) return -2;
        const int item = item_ring[2 * slot];
        mbar_arrive(bar_item_empty(slot));
        return item;
    };
    // Followers of the item ring: the k-th announced item (-1: none left; -2: the wait ran out).
    auto follow_ring = [&](int k) -> int {
        const int slot = k % RING;
        if (!__all_sync(0xffffffffu, !dead && mbar_wait(bar_item_full(slot), (k / RING) & 1))) return -2;
        // every lane reads the same word; the broadcast tells the compiler that the value (and all
        // the loop bounds and addresses derived from it) is uniform across the warp
        const int item = __shfl_sync(0xffffffffu, item_ring[2 * slot], 0);
        if (lane == 0) mbar_arrive(bar_item_empty(slot));
        return item;
    };

    // shared-memory address of sub-tile `sub` of tensor `i` in slot `s`
    auto oth_addr = [&](int s, int sub, int i) {
        return sbase + CFG::OFF_OTH + s * CFG::SLOT_BYTES + (sub * CFG::SLOT_TENSORS + i) * CFG::OTH_SUB_BYTES;
    };

    if (warp >= NPW / 32) {
    setmaxnreg_dec<CFG::REGS_ROLE>();
    if (warp == NPW / 32 + 1) {
        // =========================== TMA producer =============================================
        // Lane 0 issues the TMA copies.  In column-owned modes all 32 lanes also stage the swept
        // tile's per-query statistics, negated, into the slot's statistics buffer:
        // [-lse*log2e | -delta | -alpha | -ecirc], TN floats each.  They are read from global memory one
        // tile ahead, into registers: with the loads' latency inside the loop the producer could not keep
        // up with the tensor pipe (its next copies waited for this tile's statistics).
        int cnt = 0;                             // slots filled so far, over all items
        int s = 0, round = 0;                    // slot of the next copy, and how often the ring has turned
        int n_live = 0;                          // items with at least one tile started so far
        bool alive = true;
        constexpr int RPL = COL ? (TN + 31) / 32 : 1;                            // rows per lane
        float st_l2[RPL], st_d[RPL], st_al[RPL], st_ec[RPL];
        auto load_stats = [&](int tile, int oth_head, int batch) {
            #pragma unroll
            for (int k = 0; k < RPL; ++k) {
                const int r = lane + 32 * k, i = tile * TN + r;
                st_l2[k] = st_d[k] = st_al[k] = st_ec[k] = 0.f;
                if (r < TN && i < p.Nq) {
                    const long long off = ((long long)batch * p.Hq + oth_head) * p.Nq + i;
                    st_l2[k] = p.lse[off];
                    st_d[k] = p.delta[off];
                    if constexpr (BWD2) { st_al[k] = p.alpha[off]; st_ec[k] = p.ecirc[off]; }
                }
            }
        };
        for (int k_item = 0; alive; ++k_item) {
            const int slot = k_item % RING;
            if (!__all_sync(0xffffffffu, mbar_wait(bar_item_empty(slot), ((k_item / RING) & 1) ^ 1))) {
                if (lane == 0) give_up(kStatusTimeoutLoad);
                break;
            }
            int item = -1;
            if (p.work_counter) { if (lane == 0) item = atomicAdd(p.work_counter, 1); item = __shfl_sync(0xffffffffu, item, 0); }
            else if (k_item == 0) item = (int)blockIdx.x;
            if (item >= n_items) item = -1;
            if (lane == 0) {
                item_ring[2 * slot] = item;
                mbar_arrive(bar_item_full(slot));
            }
            if (item < 0) break;
            const Item w = decode(item);
            BOB_ITEM_LOCALS(w)
            if constexpr (!COL && MODE != kFwd) {
                // The pointwise threads start the item by reading their rows' statistics with plain loads:
                // ask for those lines now, a few tiles before they get there.
                const long long rs0 = ((long long)batch * p.Hq + head) * p.Nq + own0;
                const int r4 = (lane & 3) * 32;                      // 32 floats per line
                if (lane < 4 && own0 + r4 < n_own) prefetch_l2(p.lse + rs0 + r4);
                if (MODE == kBwd2Row && lane >= 4 && lane < 8 && own0 + r4 < n_own) prefetch_l2(p.delta + rs0 + r4);
            }
            if (total == 0) continue;
            if constexpr (COL) load_stats(t_lo, head * p.G, batch);
            if (!__all_sync(0xffffffffu, mbar_wait(bar_own_free, (n_live & 1) ^ 1))) {
                if (lane == 0) give_up(kStatusTimeoutLoad);
                break;
            }
            if (lane == 0) {
                uint32_t own_bytes = CFG::OWN_OUT && has_tensor(kTOUT) ? CFG::OWN_TILE_BYTES : 0;
                #pragma unroll
                for (int i = 0; i < MT::NOWN; ++i)
                    if (has_tensor(own_tensor<MODE>(i))) own_bytes += CFG::OWN_TILE_BYTES;
                mbar_arrive_expect_tx(bar_own, own_bytes);
                #pragma unroll
                for (int i = 0; i < CFG::OWN_TILES; ++i) {
                    const int t = i < MT::NOWN ? own_tensor<MODE>(i) : (int)kTOUT;
                    if (!has_tensor(t)) continue;
                    #pragma unroll
                    for (int ks = 0; ks < KSUB; ++ks)
                        tma_load_4d(sbase + CFG::OFF_OWN + i * CFG::OWN_TILE_BYTES + ks * (128 * 128),
                                    &p.map[t], bar_own, ks * 64, own0, head, batch);
                }
            }
            ++n_live;
            int tile = t_lo, outer = 0;          // swept tile, and its head in the group
            for (int it = 0; alive && it < total; ++it) {
                const int oth_head = COL ? (head * p.G + outer) : kv_head;
                #pragma unroll
                for (int part = 0; part < SPT; ++part) {
                    if (!alive || !__all_sync(0xffffffffu, mbar_wait(bar_empty(s), (round & 1) ^ 1))) {
                        if (alive && lane == 0) give_up(kStatusTimeoutLoad);
                        alive = false;
                        continue;
                    }
                    if (lane == 0) {
                        uint32_t bytes = 0;
                        #pragma unroll
                        for (int i = 0; i < CFG::SLOT_TENSORS; ++i)
                            if (has_tensor(other_tensor<MODE>(part + i))) bytes += KSUB * CFG::OTH_SUB_BYTES;
                        mbar_arrive_expect_tx(bar_full(s), bytes);
                        #pragma unroll
                        for (int i = 0; i < CFG::SLOT_TENSORS; ++i) {
                            const int t = other_tensor<MODE>(part + i);
                            if (!has_tensor(t)) continue;
                            #pragma unroll
                            for (int ks = 0; ks < KSUB; ++ks)
                                tma_load_4d(oth_addr(s, ks, i), &p.map[t], bar_full(s), ks * 64, tile * TN, oth_head, batch);
                        }
                    }
                    if constexpr (COL) {
                        float* sb = stat_buf + s * CFG::NSTAT * TN;
                        #pragma unroll
                        for (int k = 0; k < RPL; ++k) {
                            const int r = lane + 32 * k;
                            if (r < TN) {
                                sb[r] = neg_log2(st_l2[k]); sb[TN + r] = -st_d[k];
                                if constexpr (BWD2) { sb[2 * TN + r] = -st_al[k]; sb[3 * TN + r] = -st_ec[k]; }
                            }
                        }
                        mbar_arrive(bar_stat(s));
                    }
                    ++cnt;
                    if (++s == NSLOT) { s = 0; ++round; }
                }
                if (++tile == t_hi) { tile = t_lo; ++outer; }
                if constexpr (COL) { if (it + 1 < total) load_stats(tile, head * p.G + outer, batch); }
            }
        }
        // Do not leave while copies into this CTA's shared memory may still be in flight.
        if (lane == 0) {
            for (int k = max(0, cnt - NSLOT); k < cnt; ++k)
                mbar_wait(bar_full(k % NSLOT), (k / NSLOT) & 1);
            if (n_live > 0) mbar_wait(bar_own, (n_live - 1) & 1);
        }
    } else if (CFG::STAGED_OUT && warp == NPW / 32 + 3) {
        // =========================== results ==================================================
        // Once the pointwise threads have put an item's results into shared memory, lane 0 sends them off
        // by TMA (rows and columns outside the tensor are clipped) and hands the buffer back when it has
        // been read.
        const uint32_t io = sbase + CFG::OFF_IO;
        for (int k_item = 0;; ++k_item) {
            const int item = follow_ring(k_item);
            if (item == -2) give_up(kStatusTimeoutLoad);
            if (item < 0) break;
            const Item w = decode(item);
            BOB_ITEM_LOCALS(w)
            if (!__all_sync(0xffffffffu, mbar_wait(bar_io_ready, k_item & 1))) { give_up(kStatusTimeoutLoad); break; }
            if (lane == 0) {
                #pragma unroll
                for (int i = 0; i < CFG::N_STAGED; ++i) {
                    #pragma unroll
                    for (int ks = 0; ks < KSUB; ++ks)
                        if (ks * 64 < p.D) tma_store_4d(&p.res_map[i], io + i * CFG::OWN_TILE_BYTES + ks * (128 * 128), ks * 64, own0, head, batch);
                }
                if constexpr (CFG::STAGED_PK) {
                    #pragma unroll
                    for (int ks = 0; ks < DPAD / 32; ++ks)
                        if (p.pk && ks * 32 < p.D)
                            tma_store_4d(&p.res_map[2], io + CFG::N_STAGED * CFG::OWN_TILE_BYTES + ks * (128 * 128), ks * 32, own0, head, batch);
                }
                bulk_commit();
                bulk_wait_read();
                mbar_arrive(bar_io_free);
            }
            __syncwarp();
        }
    } else if (CFG::STAGED_IO && warp == NPW / 32 + 3) {
        // =========================== IO warp ==================================================
        // Per item: copy the tile's `out` and `dQ` rows into the two staging buffers (16-byte chunk c of
        // row r at chunk position c ^ (r & 7) of its 128-byte line), tell the pointwise threads, wait
        // until they have replaced them by the results (Qbar over dQ, dObar over out) and write those
        // out, whole 128-byte lines per quarter warp.
        const uint32_t io_out = sbase + CFG::OFF_IO, io_dq = io_out + 16384;
        for (int k_item = 0;; ++k_item) {
            const int item = follow_ring(k_item);
            if (item == -2) give_up(kStatusTimeoutLoad);
            if (item < 0) break;
            const Item w = decode(item);
            BOB_ITEM_LOCALS(w)
            const uint16_t* g_out = static_cast<const uint16_t*>(p.out) + (long long)batch * p.out_sb + (long long)head * p.out_sh + (long long)own0 * p.out_sn;
            const uint16_t* g_dq = static_cast<const uint16_t*>(p.dQ) + (long long)batch * p.dQ_sb + (long long)head * p.dQ_sh + (long long)own0 * p.dQ_sn;
            #pragma unroll 4
            for (int k = 0; k < 1024 / 32; ++k) {
                const int id = lane + 32 * k, r = id >> 3, c = id & 7;
                if (own0 + r < n_own && c * 8 < p.D) {
                    const uint32_t off = r * 128 + ((c ^ (r & 7)) << 4);
                    cp_async16(io_out + off, g_out + (long long)r * p.out_sn + c * 8);
                    cp_async16(io_dq + off, g_dq + (long long)r * p.dQ_sn + c * 8);
                }
            }
            cp_async_commit();
            cp_async_wait_all();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_io_full);
            if (!__all_sync(0xffffffffu, mbar_wait(bar_io_ready, k_item & 1))) { give_up(kStatusTimeoutLoad); break; }
            const long long tile_row0 = ((long long)batch * p.Hq + head) * p.Nq + own0;     // results are contiguous
            uint16_t* g_q = static_cast<uint16_t*>(p.res0) + tile_row0 * p.D;
            uint16_t* g_do = static_cast<uint16_t*>(p.res1) + tile_row0 * p.D;
            #pragma unroll 4
            for (int k = 0; k < 1024 / 32; ++k) {
                const int id = lane + 32 * k, r = id >> 3, c = id & 7;
                if (own0 + r < n_own && c * 8 < p.D) {
                    const uint32_t off = r * 128 + ((c ^ (r & 7)) << 4);
                    *reinterpret_cast<uint4*>(g_q + (long long)r * p.D + c * 8) = ld_shared_v4(io_dq + off);
                    *reinterpret_cast<uint4*>(g_do + (long long)r * p.D + c * 8) = ld_shared_v4(io_out + off);
                }
            }
            __syncwarp();
        }
    } else if (warp == NPW / 32 || warp == NPW / 32 + 2) {
        // =========================== MMA issuers ==============================================
        // Warp NPW/32 issues the score-shaped products (as far ahead as accumulators are free), warp
        // NPW/32 + 2 the output-shaped ones (as operands arrive).  The tensor pipe takes whichever is ready.
        // One elected thread runs the whole loop of a role: its waits, addresses and loop overhead then cost 30-80
        // cycles per tile, against 250-300 when the warp waits together and elects a lane for every burst
        // (measured with eight 128x64x16 products per burst, 384 cycles of tensor time: 418 against 637 in all).
        constexpr uint32_t fmt = BF16 ? kFmtBF16 : kFmtF16;
        // Descriptor low words: (shared-memory address >> 4) | 0x10000 (leading byte offset 16).
        // Everything but the slot is a compile-time offset from these bases.
        const uint32_t own16 = ((sbase + CFG::OFF_OWN) >> 4) | 0x10000u;
        const uint32_t oth16 = ((sbase + CFG::OFF_OTH) >> 4) | 0x10000u;
        int s = 0, par = 0;                      // slot of the next tile, parity of its use
        int n_live = 0;                          // items with at least one tile handled so far
        if (!elect_one()) {
            // the other lanes meet this one at the teardown
        } else if (warp == NPW / 32) {
            BOB_TR_DECL(1)
            // score-shaped product: acc[128, NS*TN] (+)= own[slot_a] * other[slot_b .. slot_b+NS-1]^T.
            // NS = 2 takes two adjacent swept tiles as one 2*TN-row operand and fills two adjacent
            // accumulators with one instruction per K step (the own tile is read once, not twice).
            auto score_mma = [&](auto ns_tag, uint32_t sc_base, int acc, int slot_a, int slot_b, uint32_t stage16, bool accumulate) {
                constexpr int NS = decltype(ns_tag)::value;
                constexpr uint32_t idesc = umma_idesc(fmt, fmt, NS * TN, false);
                const uint32_t a = own16 + ((slot_a * CFG::OWN_TILE_BYTES) >> 4);
                const uint32_t b = stage16 + ((slot_b * CFG::OTH_SUB_BYTES) >> 4);
                const bool from_tm = CFG::OWN_TM && slot_a == 0;          // own tile 0 also sits in tensor memory
                #pragma unroll
                for (int ks = 0; ks < DPAD / 16; ++ks) {
                    const uint32_t ao = ((ks / 4) * (128 * 128) + (ks % 4) * 32) >> 4;
                    const uint32_t bo = ((ks / 4) * (CFG::SLOT_TENSORS * CFG::OTH_SUB_BYTES) + (ks % 4) * 32) >> 4;
                    if (from_tm) umma_ts_lo(sc_base + acc * TN, tmem_own + ks * 8, b + bo, idesc, (accumulate || ks > 0) ? 1u : 0u);
                    else umma_ss_lo(sc_base + acc * TN, a + ao, b + bo, idesc, (accumulate || ks > 0) ? 1u : 0u);
                }
            };
            using NS1 = IntTag<1>;
            using NS2 = IntTag<2>;
            uint32_t free_par = 0;               // !ALIAS: bit g = parity of group g's next "scores read" wait
            // ALIAS: each group's last tile - its slot, parity and number (-1: none yet) - and the newest tile whose
            // products are known to have finished.
            int last_s0 = 0, last_s1 = 0, last_p0 = 0, last_p1 = 0, last_n0 = -1, last_n1 = -1;
            int n_sc = 0, done_n = -1;
            for (int k_item = 0;; ++k_item) {
                const int item = follow_ring_alone(k_item);
                if (item == -2) give_up(kStatusTimeoutMma);
                if (item < 0) break;
                const Item w = decode(item);
                BOB_ITEM_LOCALS(w)
                if (total == 0) continue;
                wait_alone(bar_own, n_live & 1, kStatusTimeoutMma);
                if constexpr (CFG::OWN_TM) wait_alone(bar_own_tm, n_live & 1, kStatusTimeoutMma);
                ++n_live;
                // The group of tile `it` is it % NG: a function of the item alone, so that which group sums which
                // tiles, and with it the rounding of the result, does not depend on what the CTA did before.
                int g = 0;
                for (int it = 0; it < total; ++it) {
                    const uint32_t st16 = oth16 + ((s * CFG::SLOT_BYTES) >> 4);
                    const uint32_t sc = tmem + g * CFG::SC_COLS;
                    BOB_TR(0)
                    wait_alone(bar_full(s), par, kStatusTimeoutMma);
                    BOB_TR(1)
                    if constexpr (ALIAS) {
                        // The group's operands sit in its score columns until its output products have read them.
                        // Products finish in the order of the tiles, so a tile up to done_n needs no wait, and must have
                        // none: after an item with an odd number of tiles a group's last tile is three or more back, its
                        // slot may have been filled and emptied once more, and the parity would then mean a
                        // phase that only tiles yet to be issued can complete.  Where the wait is taken, the other group
                        // has had at most one tile since (with a second one, that one's wait raised done_n), so
                        // the slot's next tile is not issued yet.
                        const int ln = g ? last_n1 : last_n0;
                        if (ln > done_n) {
                            wait_alone(bar_empty(g ? last_s1 : last_s0), g ? last_p1 : last_p0, kStatusTimeoutMma);
                            done_n = ln;
                        }
                    } else {
                        wait_alone(bar_sc_empty(g), ((free_par >> g) & 1u) ^ 1u, kStatusTimeoutMma);
                        free_par ^= 1u << g;
                    }
                    BOB_TR(2)
                    tc_fence_after_sync();
                    if constexpr (MODE == kFwd) {
                        score_mma(NS1{}, sc, 0, 0, 0, st16, false);
                    } else if constexpr (MODE == kBwd1Row || MODE == kBwd1Col) {
                        score_mma(NS1{}, sc, 0, 0, 0, st16, false);     // S  = Q K^T      | S^T  = K Q^T
                        score_mma(NS1{}, sc, 1, 1, 1, st16, false);     // dP = dO V^T     | dP^T = V dO^T
                    } else if constexpr (MODE == kBwd2Row) {
                        // own: Q, dO, uQ;  swept: K, uK, V, uV;  accumulators: S, F, dP, C
                        if (has_uk) score_mma(NS2{}, sc, 0, 0, 0, st16, false);      // S | F  = Q [K; uK]^T
                        else          score_mma(NS1{}, sc, 0, 0, 0, st16, false);      // S      = Q K^T
                        if (!CFG::SPLIT_SC && has_uq) score_mma(NS1{}, sc, 1, 2, 0, st16, has_uk);   // F     += uQ K^T
                        if (has_uv) score_mma(NS2{}, sc, 2, 1, 2, st16, false);      // dP | C = dO [V; uV]^T
                        else          score_mma(NS1{}, sc, 2, 1, 2, st16, false);      // dP     = dO V^T
                        if constexpr (CFG::SPLIT_SC) {
                            umma_commit(bar_sc_part(g));                              // S, dP, C are complete
                            if (has_uq) score_mma(NS1{}, sc, 1, 2, 0, st16, has_uk);   // F     += uQ K^T
                        }
                    } else {
                        // own: K, V, uK, uV;  swept: Q, uQ, dO;  accumulators: S^T, F^T, dP^T, C^T
                        if (has_uq) score_mma(NS2{}, sc, 0, 0, 0, st16, false);      // S^T | F^T = K [Q; uQ]^T
                        else          score_mma(NS1{}, sc, 0, 0, 0, st16, false);      // S^T       = K Q^T
                        if (has_uk) score_mma(NS1{}, sc, 1, 2, 0, st16, has_uq);   // F^T      += uK Q^T
                        score_mma(NS1{}, sc, 2, 1, 2, st16, false);                    // dP^T      = V dO^T
                        if (has_uv) score_mma(NS1{}, sc, 3, 3, 2, st16, false);      // C^T       = uV dO^T
                    }
                    umma_commit(bar_sc_full(g));
                    if constexpr (CFG::SPLIT_KV) umma_commit(bar_empty(s));           // K is free again
                    if (it + 1 == total) umma_commit(bar_own_free);                   // the item's own tiles too
                    BOB_TR(3)
                    int vs = s + SPT - 1, vp = par;                   // the tile's last slot (forward: V's)
                    if (SPT == 2 && vs == NSLOT) { vs = 0; vp ^= 1; }
                    if (g) { last_s1 = vs; last_p1 = vp; last_n1 = n_sc; } else { last_s0 = vs; last_p0 = vp; last_n0 = n_sc; }
                    ++n_sc;
                    if constexpr (NG == 2) g ^= 1;
                    s += SPT;
                    if (s >= NSLOT) { s -= NSLOT; par ^= 1; }
                }
            }
            BOB_TR_FLUSH
        } else {
            BOB_TR_DECL(2)
            // output-shaped product: out[128, DPAD] (+)= operand[oper] * other[slot_b]; the operand is read from
            // tensor memory (8 columns per 16-element K step), the swept tile MN-major from shared memory,
            // all DPAD output columns in one instruction: at head dim 128 the second 64 columns come from the
            // swept tensor's second sub-tile, one `leading byte offset` further on
            auto out_mma = [&](int g, int out, int oper, int slot_b, uint32_t stage16, bool accumulate) {
                constexpr uint32_t idesc = umma_idesc(fmt, fmt, DPAD, true);
                constexpr uint32_t lbo16 = (KSUB > 1) ? ((CFG::SLOT_TENSORS * CFG::OTH_SUB_BYTES) >> 4) : 1u;
                const uint32_t a = ALIAS ? tmem + g * CFG::SC_COLS + (oper >> 1) * TN + (oper & 1) * 8
                                         : tmem_oper + g * CFG::OPER_COLS + oper * CFG::OPER_COLS_EACH;
                const uint32_t b = (stage16 - 0x10000u) + (lbo16 << 16) + ((slot_b * CFG::OTH_SUB_BYTES) >> 4);
                #pragma unroll
                for (int ks = 0; ks < TN / 16; ++ks)
                    umma_ts_lo(tmem_out + out * DPAD, a + ks * (ALIAS ? 16 : 8), b + ((ks * 2048) >> 4), idesc,
                               (accumulate || ks > 0) ? 1u : 0u);
            };
            uint32_t op_par = 0;                 // bit g = parity of group g's next "operands written" wait
            if constexpr (CFG::SPLIT_KV) s = 1;  // V sits in the slot after K
            for (int k_item = 0;; ++k_item) {
                const int item = follow_ring_alone(k_item);
                if (item == -2) give_up(kStatusTimeoutMma);
                if (item < 0) break;
                const Item w = decode(item);
                BOB_ITEM_LOCALS(w)
                if (total == 0) continue;
                int g = 0;
                for (int it = 0; it < total; ++it) {
                    const uint32_t st16 = oth16 + ((s * CFG::SLOT_BYTES) >> 4);
                    BOB_TR(0)
                    wait_alone(bar_op_full(g), (op_par >> g) & 1u, kStatusTimeoutMma);
                    op_par ^= 1u << g;
                    // the first products of an item overwrite the output accumulators: the pointwise
                    // threads must have read out the previous item's
                    if (it == 0) wait_alone(bar_out_free, (n_live & 1) ^ 1, kStatusTimeoutMma);
                    if constexpr (CFG::SPLIT_KV) wait_alone(bar_full(s), par, kStatusTimeoutMma);
                    BOB_TR(1)
                    tc_fence_after_sync();
                    const bool acc = it > 0;
                    if constexpr (MODE == kFwd) {
                        out_mma(g, g, 0, 0, st16, it >= NG);                 // O_g += P V (group g's own accumulator)
                    } else if constexpr (MODE == kBwd1Row) {
                        out_mma(g, 0, 0, 0, st16, acc);                      // dQ += dS K
                        if (p.pk) out_mma(g, 1, 1, 0, st16, acc);            // PK += P K
                    } else if constexpr (MODE == kBwd1Col) {
                        out_mma(g, 0, 1, 0, st16, acc);                      // dK += dS^T Q
                        out_mma(g, 1, 0, 1, st16, acc);                      // dV += P^T dO
                    } else if constexpr (MODE == kBwd2Row) {
                        // operands: P, P*F, P*T, dS;  swept: K, uK, V, uV;  outputs: dObar, Omega
                        if (has_uv) out_mma(g, 0, 0, 3, st16, acc);          // dObar += P uV
                        out_mma(g, 0, 1, 2, st16, acc || has_uv);            // dObar += (P*F) V
                        out_mma(g, 1, 2, 0, st16, acc);                      // Omega += (P*T) K
                        if (has_uk) out_mma(g, 1, 3, 1, st16, true);         // Omega += dS uK
                    } else {
                        // operands: Sbar^T, dS^T, (P*(F-alpha))^T;  outputs: Kbar, Vbar
                        out_mma(g, 0, 0, 0, st16, acc);                      // Kbar += Sbar^T Q
                        if (has_uq) out_mma(g, 0, 1, 1, st16, true);         // Kbar += dS^T uQ
                        out_mma(g, 1, 2, 2, st16, acc);                      // Vbar += (P*(F-alpha))^T dO
                    }
                    // operands consumed, and the slot is free again (the score products that read it
                    // finished before these operands could be formed)
                    umma_commit(bar_empty(s));
                    if (it + 1 == total) umma_commit(bar_done);              // the item's accumulators are complete
                    BOB_TR(2)
                    if constexpr (NG == 2) g ^= 1;
                    s += SPT;
                    if (s >= NSLOT) { s -= NSLOT; par ^= 1; }
                }
                ++n_live;
            }
            BOB_TR_FLUSH
        }
        __syncwarp();
    }
    } else {
        // =========================== pointwise threads =======================================
        setmaxnreg_inc<CFG::REGS_POINTWISE>();
        const int grp = tid / GP;                // pointwise group: takes iterations grp, grp + NG, ...
        const int gtid = tid % GP;
        const int row = gtid & 127;              // own row inside the tile == tensor-memory lane
        const int sp = gtid >> 7;                // which slice of every score tile
        const int col0 = sp * CW;                // my first column inside a swept tile
        const uint32_t tlane = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);   // my lane, column 0
        const uint32_t tsc = tlane + grp * CFG::SC_COLS;                                  // my group's scores
        const uint32_t tout = tlane + NG * (CFG::SC_COLS + CFG::OPER_COLS);               // output accumulators
        const float c_exp = p.scale * kLog2e;
        // 16 columns of a tile in one round (RW): eight packed words per operand
        constexpr int RW = 16, R = CW / RW;
        // where operand k of my columns' round r goes in tensor memory: next to the other operands, or (ALIAS)
        // over the 16 score columns of that round, two operands per accumulator
        auto op_addr = [&](int k, int r) -> uint32_t {
            if constexpr (ALIAS) return tsc + (k >> 1) * TN + col0 + RW * r + (k & 1) * 8;
            else return tlane + NG * CFG::SC_COLS + grp * CFG::OPER_COLS + k * CFG::OPER_COLS_EACH + (col0 >> 1) + 8 * r;
        };

        uint32_t pw_all_phase = 0;               // phase of the all-groups barrier
        auto all_sync = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_pw_all);
            wait(bar_pw_all, pw_all_phase, kStatusTimeoutPw);
            pw_all_phase ^= 1u;
        };
        int s = 0, par = 0;                      // slot of the item's next tile, parity of its use
        int last_s = -1, last_par = 0;           // !ALIAS: my group's last tile of this item, whose products must have read its operands
        uint32_t sc_par = 0;                     // parity of my group's next scores
        int n_live = 0;                          // items with at least one tile finished so far
        int n_done = 0;                          // items finished so far, with or without tiles
        int exp_base = 0;                        // forward: exponential phases of the other group before this item
        (void)exp_base;
        BOB_TR_DECL(warp == 0 ? 0 : -1)

        for (int k_item = 0;; ++k_item) {
            const int item = follow_ring(k_item);
            if (item == -2) give_up(kStatusTimeoutPw);
            if (item < 0) break;
        const Item w = decode(item);
        BOB_ITEM_LOCALS(w)
        const int own_idx = own0 + row;
        const bool own_ok = own_idx < n_own;
        const long long row_stat = ((long long)batch * p.Hq + head) * p.Nq + own_idx;   // row-owned only

        // per-row state (row-owned modes): -lse*log2e and -delta of my row
        float nL2 = 0.f, ndlt = 0.f;
        float2 acc_a = make_float2(0.f, 0.f), acc_b = make_float2(0.f, 0.f);   // row sums alpha, ecirc
        // forward: my group's online softmax over the tiles it takes.  m_ref is the exponent reference
        // (log2 units): it follows the running maximum only when that has grown by more than 8, so
        // that the output accumulator rarely needs rescaling; probabilities stay below 2^8.
        float m_ref = -1e30f, l_run = 0.f;
        bool first_tile = true;                  // forward: my group has no accumulator yet
        (void)m_ref; (void)l_run; (void)first_tile;

        if constexpr (MODE == kBwd1Row) {
            // delta = rowsum(dO * out), from the two tiles in shared memory: each of the threads that share a
            // row sums its part of it, the parts are added in a fixed order.
            float l_row = 0.f;
            if (own_ok) l_row = p.lse[row_stat];
            float dlt = 0.f;
            if (total > 0) {
                wait(bar_own, n_live & 1, kStatusTimeoutPw);
                constexpr int NPART = NG * NSPLIT, CH = DPAD / 8 / NPART;      // 16-byte chunks per thread
                const int part = grp * NSPLIT + sp;
                const uint32_t t_do = sbase + CFG::OFF_OWN + CFG::OWN_TILE_BYTES, t_out = t_do + CFG::OWN_TILE_BYTES;
                float sum = 0.f;
                #pragma unroll
                for (int c = 0; c < CH; ++c) {
                    const int ch = part * CH + c;
                    const uint32_t off = (ch / 8) * (128 * 128) + sw128_offset(row, ch % 8);
                    float a[8], b[8];
                    uint4 w = make_uint4(0, 0, 0, 0);
                    if (!p.out) w = ld_shared_v4(t_out + off);
                    else if (own_ok && ch * 8 < p.D)
                        w = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.out) + (long long)batch * p.out_sb +
                                                            (long long)head * p.out_sh + (long long)own_idx * p.out_sn + ch * 8);
                    unpack8_as_float<BF16>(w, a);
                    unpack8_as_float<BF16>(ld_shared_v4(t_do + off), b);
                    #pragma unroll
                    for (int i = 0; i < 8; ++i) sum = fmaf(a[i], b[i], sum);
                }
                red_buf[part * 128 + row] = sum;
                all_sync();
                #pragma unroll
                for (int k = 0; k < NPART; ++k) dlt += red_buf[k * 128 + row];
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_own_free);        // (the next item's sums come after its tiles, so after this)
            }
            if (grp == 0 && sp == 0 && own_ok) p.delta[row_stat] = dlt;
            ndlt = -dlt;
            nL2 = neg_log2(l_row);
        }
        if constexpr (MODE == kBwd2Row) {
            if (own_ok) { nL2 = neg_log2(p.lse[row_stat]); ndlt = -p.delta[row_stat]; }
        }
        // Own tile 0 into tensor memory (see SweepConfig::OWN_TM): once the item's own tiles have landed,
        // every thread copies its share of its own row, 16 elements (two 16-byte chunks of the swizzled
        // shared-memory tile = eight packed columns) at a time.  The previous item's products are all
        // finished by now (its epilogue waited for them), so nothing reads the old copy any more.
        if constexpr (CFG::OWN_TM) {
            if (total > 0) {
                wait(bar_own, n_live & 1, kStatusTimeoutPw);
                constexpr int PER = (DPAD / 8) / NSPLIT;             // 16-byte chunks of my row that I copy
                static_assert(PER % 2 == 0, "two chunks per tensor-memory store");
                #pragma unroll
                for (int c = sp * PER; c < (sp + 1) * PER; c += 2) {
                    const uint32_t src = sbase + CFG::OFF_OWN + (c / 8) * (128 * 128);
                    const uint4 lo = ld_shared_v4(src + sw128_offset(row, c % 8));
                    const uint4 hi = ld_shared_v4(src + sw128_offset(row, c % 8 + 1));
                    const uint32_t wds[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                    tmem_st8(tlane + (tmem_own - tmem) + 4 * c, wds);
                }
                tmem_wait_st();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) { mbar_arrive(bar_own_tm); mbar_arrive(bar_own_free); }
            }
        }
        if constexpr (MODE == kBwd2Row) {
            // my row's pk columns are read when the sweep ends: have them in L2 by then
            constexpr int DCP = DPAD / (NSPLIT * NG);            // fp32 columns per thread, 128 bytes per 32
            const int c0 = (grp * NSPLIT + sp) * DCP;
            #pragma unroll
            for (int c = 0; c < DCP; c += 32)
                if (own_ok && c0 + c < p.D) prefetch_l2(p.pk + (((long long)batch * p.Hq + head) * p.Nq + own_idx) * p.D + c0 + c);
        }
        // staged rows: 16-byte chunk c of row r sits at chunk position c ^ (r & 7) of its 128-byte line, so
        // that both the row-wise and the chunk-wise accesses are conflict-free
        const uint32_t io_out = sbase + CFG::OFF_IO, io_dq = io_out + 16384;
        const long long tile_row0 = ((long long)batch * p.Hq + head) * p.Nq + own0;   // first row of the contiguous results
        (void)io_out; (void)io_dq; (void)tile_row0;

        // One swept tile.  full: every (row, column) of the tile pair is unmasked and in range.  Elsewhere masked
        // scores become -inf, which makes their probabilities zero.  One body serves both: a second, unrolled copy
        // for masked tiles cost more in instruction fetches than it saved in selects (a masked tile of the forward took
        // 4800 cycles longer than a full one, and every causal item has one; with one body B=8 H=12 S=1024 D=64 training
        // went from 151.7 to 134.3 us, S=8192 with a window of 1024 from 274.3 to 254.8 us).
        auto tile_body = [&](const bool full, int it, int tile, int s, int par) {
            const int oth0 = tile * TN;

            BOB_TR(0)
            if constexpr (COL) wait(bar_stat(s), par, kStatusTimeoutPw);   // staged by the producer warp
            wait(CFG::SPLIT_SC ? bar_sc_part(grp) : bar_sc_full(grp), sc_par, kStatusTimeoutPw);
            BOB_TR(1)
            tc_fence_after_sync();

            // ---- which of my columns are unmasked --------------------------------------------
            // dist = query position - key position; unmasked iff in range and, when causal,
            // 0 <= dist (< window)
            uint32_t vmask[(CW + 31) / 32];          // bit c % 32 of word c / 32: column c of mine is unmasked
            if (!full) {
                int mlo = 0, mhi = min(CW - 1, n_oth - (oth0 + col0) - 1);
                if (causal) {
                    if constexpr (!COL) {
                        const int d0 = own_idx + doff - (oth0 + col0);       // dist falls with the column
                        mhi = min(mhi, d0);
                        if (window > 0) mlo = max(mlo, d0 - window + 1);
                    } else {
                        const int d0 = (oth0 + col0) + doff - own_idx;       // dist grows with the column
                        mlo = max(mlo, -d0);
                        if (window > 0) mhi = min(mhi, window - 1 - d0);
                    }
                }
                if (!own_ok) mhi = -1;
                #pragma unroll
                for (int k = 0; k < (CW + 31) / 32; ++k) {
                    const int lo = max(mlo - 32 * k, 0), hi = min(mhi - 32 * k, 31);
                    vmask[k] = hi >= lo ? (0xffffffffu >> (31 - hi)) & (0xffffffffu << lo) : 0u;
                }
            }
            // n scores from column c0 of mine on
            auto mask_scores = [&](float* v, int c0, int n) {
                #pragma unroll
                for (int c = 0; c < n; ++c) v[c] = (vmask[(c0 + c) / 32] >> ((c0 + c) % 32)) & 1u ? v[c] : -INFINITY;
            };
            // The previous products of my group must have read its operands before I write new ones (with ALIAS
            // they have: the scores just read were issued after them).
            auto operands_free = [&]() {
                if constexpr (!ALIAS) { if (last_s >= 0) wait(bar_empty(last_s), last_par, kStatusTimeoutPw); }
            };

            if constexpr (MODE == kFwd) {
                // One thread owns a whole row of the tile.
                float s_[CW];
                #pragma unroll
                for (int h = 0; h < CW / 16; ++h) tmem_ld16(tsc + 16 * h, s_ + 16 * h);
                tmem_wait_ld();
                if constexpr (!ALIAS) {
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_sc_empty(grp));
                }
                BOB_TR(2)
                if (!full) mask_scores(s_, 0, CW);
                // largest unmasked score of my row in this tile (the scale is positive)
                float mr4[4] = {-3.0e38f, -3.0e38f, -3.0e38f, -3.0e38f};     // four chains, for instruction-level parallelism
                #pragma unroll
                for (int c = 0; c < CW; c += 2)
                    mr4[(c >> 1) & 3] = fmaxf(fmaxf(mr4[(c >> 1) & 3], s_[c]), s_[c + 1]);
                const float mr = fmaxf(fmaxf(mr4[0], mr4[1]), fmaxf(mr4[2], mr4[3]));
                const float mt = fmaxf(mr * c_exp, -1e30f);
                // move the reference only when the maximum has outgrown it; the whole warp then
                // rescales its rows of the output accumulator (factor 1 where nothing changed)
                const bool grow = mt > m_ref + 8.f;
                const bool rescale = __any_sync(0xffffffffu, grow) && !first_tile;
                float factor = 1.f;
                if (grow) { factor = fast_exp2(m_ref - mt); m_ref = mt; }
                l_run *= factor;
                // My group's previous product must have consumed its operand and finished with the
                // accumulator before I touch either.
                operands_free();
                BOB_TR(3)
                if (rescale) {
                    tc_fence_after_sync();
                    const uint32_t tacc = tout + grp * DPAD;
                    #pragma unroll
                    for (int ch = 0; ch < DPAD / 16; ++ch) {
                        float t[16];
                        uint32_t u[16];
                        tmem_ld16(tacc + 16 * ch, t);
                        tmem_wait_ld();
                        #pragma unroll
                        for (int i = 0; i < 16; ++i) u[i] = __float_as_uint(t[i] * factor);
                        tmem_st8(tacc + 16 * ch, u);
                        tmem_st8(tacc + 16 * ch + 8, u + 8);
                    }
                }
                // The two groups take turns with the exponentials: a warp starts its tile's when the other group's warp
                // on the same scheduler has finished those of the tile before.  Left alone, the groups fall into step,
                // compete for the special-function unit at the same time and leave it idle at the same time
                // (128.0 against 134.8 us on B=1 GQA 32/8 S=4096 D=64, 100.2 against 112.5 us on B=2 S=2048 D=128).
                if (it > 0) wait(bar_exp(1 - grp), (exp_base + ((it - 1) >> 1)) & 1, kStatusTimeoutPw);
                // probabilities relative to the reference, 16 columns at a time straight into tensor memory
                const float nm = -m_ref;
                float2 sum4[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                const float2 cexp2 = make_float2(c_exp, c_exp), nm2 = make_float2(nm, nm);
                #pragma unroll
                for (int h = 0; h < CW / 16; ++h) {
                    uint32_t w0[8];
                    #pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int c = 16 * h + 2 * k;
                        const float2 x = __ffma2_rn(make_float2(s_[c], s_[c + 1]), cexp2, nm2);
                        const float2 pr = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                        sum4[k & 3] = __fadd2_rn(sum4[k & 3], pr);
                        w0[k] = pack2<BF16>(pr.x, pr.y);
                    }
                    tmem_st8(op_addr(0, h), w0);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_exp(grp));
                const float2 t = __fadd2_rn(__fadd2_rn(sum4[0], sum4[1]), __fadd2_rn(sum4[2], sum4[3]));
                l_run += t.x + t.y;
                first_tile = false;
            } else {
                // accumulator order: S, dP (first backward) or S, F, dP, C (second backward).
                // My CW columns are taken in rounds of 16.  Without ALIAS every round's loads are issued at once
                // and the score accumulators are handed back before any arithmetic, so that the next tile's
                // score products run under this tile's arithmetic.  With ALIAS the scores stay where they are
                // until their round, one round's loads ahead of its arithmetic.  Each round's packed operands go
                // to tensor memory as soon as they are formed.
                constexpr int NB = ALIAS ? (R > 1 ? 2 : 1) : R;
                const float2 cexp2 = make_float2(c_exp, c_exp);
                const float2 scale2 = make_float2(p.scale, p.scale);
                const bool has_f = BWD2 && (ALLT || has_uq || has_uk);
                const bool has_c = BWD2 && (ALLT || has_uv);
                float in_s[NB][RW], in_dp[NB][RW], in_f[NB][RW], in_c[NB][RW];
                // part: 0 = every accumulator, 1 = all but F, 2 = F alone
                auto issue_loads = [&](int r, int part = 0) {
                    const int b = r % NB, cb = col0 + RW * r;
                    if (part != 2) {
                        tmem_ld16(tsc + 0 * TN + cb, in_s[b]);
                        tmem_ld16(tsc + (BWD2 ? 2 : 1) * TN + cb, in_dp[b]);
                    }
                    if constexpr (BWD2) {
                        if (part != 1 && has_f) tmem_ld16(tsc + 1 * TN + cb, in_f[b]);
                        if (part != 2 && has_c) tmem_ld16(tsc + 3 * TN + cb, in_c[b]);
                    }
                };
                if constexpr (CFG::SPLIT_SC) {
                    // S, dP and C now; F once its second term has been added (the loads above are on
                    // their way while that product runs)
                    #pragma unroll
                    for (int r = 0; r < R; ++r) issue_loads(r, 1);
                    wait(bar_sc_full(grp), sc_par, kStatusTimeoutPw);
                    tc_fence_after_sync();
                    #pragma unroll
                    for (int r = 0; r < R; ++r) issue_loads(r, 2);
                } else {
                    #pragma unroll
                    for (int r = 0; r < (ALIAS ? 1 : R); ++r) issue_loads(r);
                }
                #pragma unroll
                for (int half = 0; half < R; ++half) {            // `half` = round of RW columns
                    const int cb = col0 + RW * half;
                    const int b = half % NB;
                    if (ALIAS || half == 0) tmem_wait_ld();
                    if constexpr (ALIAS) {
                        if (half + 1 < R) issue_loads(half + 1);
                    } else if (half == 0) {
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_sc_empty(grp));
                        BOB_TR(2)
                    }
                    float* s_ = in_s[b];
                    if (!full) mask_scores(s_, RW * half, RW);
                    float* dp_ = in_dp[b];
                    float* f_ = in_f[b];
                    float* cc_ = in_c[b];
                    if constexpr (BWD2) {
                        if (!has_f) {
                            #pragma unroll
                            for (int c = 0; c < RW; ++c) f_[c] = 0.f;
                        }
                        if (!has_c) {
                            #pragma unroll
                            for (int c = 0; c < RW; ++c) cc_[c] = 0.f;
                        }
                    }
                    uint32_t wbuf[4][RW / 2];
                    // negated statistics of these columns (column-owned modes), four columns per load
                    const float4* sb4 = reinterpret_cast<const float4*>(stat_buf + s * CFG::NSTAT * TN + cb);
                    #pragma unroll
                    for (int c4 = 0; c4 < RW / 4; ++c4) {
                        float4 q_l2, q_dl, q_al, q_ec;
                        if constexpr (COL) {
                            q_l2 = sb4[c4]; q_dl = sb4[TN / 4 + c4];
                            if constexpr (MODE == kBwd2Col) { q_al = sb4[2 * (TN / 4) + c4]; q_ec = sb4[3 * (TN / 4) + c4]; }
                        }
                        (void)q_al; (void)q_ec;
                        #pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int c = 4 * c4 + 2 * h;          // columns c, c + 1 of this round
                            const int wi = c >> 1;                 // packed word index inside this round
                            float2 nl2, ndl, nal, nec;
                            (void)nal; (void)nec;
                            if constexpr (COL) {
                                nl2 = h ? make_float2(q_l2.z, q_l2.w) : make_float2(q_l2.x, q_l2.y);
                                ndl = h ? make_float2(q_dl.z, q_dl.w) : make_float2(q_dl.x, q_dl.y);
                                if constexpr (MODE == kBwd2Col) {
                                    nal = h ? make_float2(q_al.z, q_al.w) : make_float2(q_al.x, q_al.y);
                                    nec = h ? make_float2(q_ec.z, q_ec.w) : make_float2(q_ec.x, q_ec.y);
                                }
                            } else {
                                nl2 = make_float2(nL2, nL2);
                                ndl = make_float2(ndlt, ndlt);
                            }
                            const float2 x = __ffma2_rn(make_float2(s_[c], s_[c + 1]), cexp2, nl2);
                            const float2 pr = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                            const float2 dps = __fadd2_rn(make_float2(dp_[c], dp_[c + 1]), ndl);
                            if constexpr (MODE == kBwd1Row) {
                                const float2 ds = __fmul2_rn(pr, dps);
                                wbuf[0][wi] = pack2<BF16>(ds.x, ds.y);                         // dS
                                wbuf[1][wi] = pack2<BF16>(pr.x, pr.y);                         // P
                            } else if constexpr (MODE == kBwd1Col) {
                                const float2 ds = __fmul2_rn(pr, dps);
                                wbuf[0][wi] = pack2<BF16>(pr.x, pr.y);                         // P^T
                                wbuf[1][wi] = pack2<BF16>(ds.x, ds.y);                         // dS^T
                            } else if constexpr (MODE == kBwd2Row) {
                                const float2 f = __fmul2_rn(make_float2(f_[c], f_[c + 1]), scale2);
                                const float2 t = __ffma2_rn(f, dps, make_float2(cc_[c], cc_[c + 1]));
                                const float2 pf = __fmul2_rn(pr, f);
                                const float2 pt = __fmul2_rn(pr, t);
                                const float2 ds = __fmul2_rn(pr, dps);
                                acc_a = __fadd2_rn(acc_a, pf);
                                acc_b = __fadd2_rn(acc_b, pt);
                                wbuf[0][wi] = pack2<BF16>(pr.x, pr.y);                         // P
                                wbuf[1][wi] = pack2<BF16>(pf.x, pf.y);                         // P*F
                                wbuf[2][wi] = pack2<BF16>(pt.x, pt.y);                         // P*T
                                wbuf[3][wi] = pack2<BF16>(ds.x, ds.y);                         // dS
                            } else {
                                // T - alpha (dP - delta) - ecirc = (F - alpha) (dP - delta) + (C - ecirc)
                                const float2 fa = __ffma2_rn(make_float2(f_[c], f_[c + 1]), scale2, nal);   // F - alpha
                                const float2 u = __ffma2_rn(fa, dps, __fadd2_rn(make_float2(cc_[c], cc_[c + 1]), nec));
                                const float2 sbar = __fmul2_rn(pr, u);
                                const float2 ds = __fmul2_rn(pr, dps);
                                const float2 ph = __fmul2_rn(pr, fa);
                                wbuf[0][wi] = pack2<BF16>(sbar.x, sbar.y);                     // Sbar^T
                                wbuf[1][wi] = pack2<BF16>(ds.x, ds.y);                         // dS^T
                                wbuf[2][wi] = pack2<BF16>(ph.x, ph.y);                         // (P*(F-alpha))^T
                            }
                        }
                    }
                    if (half == 0) { operands_free(); BOB_TR(3) }
                    #pragma unroll
                    for (int k = 0; k < MT::NOPER; ++k) tmem_st8(op_addr(k, half), wbuf[k]);
                }
            }
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_op_full(grp));
            sc_par ^= 1u;
            last_s = s + (SPT - 1); last_par = par;
            if (SPT == 2 && last_s == NSLOT) { last_s = 0; last_par ^= 1; }
            BOB_TR(4)
        };

        {
            // swept tiles [full_lo, full_hi) pair with my own tile entirely unmasked and in range
            int full_lo = 0, full_hi = 0;
            if (own0 + 127 < n_own) {
                int lo = 0, hi = n_oth / TN;                        // tiles that lie inside the tensor
                if (causal) {
                    // oldest and newest own position of the tile pair against the swept tile's extremes
                    if constexpr (!COL) {
                        hi = min(hi, (own0 + doff + 1) / TN);                           // dist >= 0 everywhere
                        if (window > 0) {
                            const int x = own0 + 127 + doff - window;                   // last swept position with dist >= window
                            lo = max(lo, x < 0 ? 0 : (x + TN) / TN);
                        }
                    } else {
                        const int a = own0 + 127 - doff;                                // first swept position with dist >= 0
                        lo = max(lo, a <= 0 ? 0 : (a + TN - 1) / TN);
                        if (window > 0) {
                            const int b = own0 - doff + window;                         // one past the last with dist < window
                            hi = min(hi, b <= 0 ? 0 : b / TN);
                        }
                    }
                }
                if (hi > lo) { full_lo = lo; full_hi = hi; }
            }
            // my group's tiles; from one to the next, NG tiles and their slots are passed
            int tile = t_lo + (NG == 2 ? grp : 0), ts = s + (NG == 2 ? grp : 0) * SPT, tp = par;
            const int n_sweep = t_hi - t_lo;
            if (ts >= NSLOT) { ts -= NSLOT; tp ^= 1; }
            if (COL && tile >= t_hi) tile -= n_sweep;
            for (int it = NG == 2 ? grp : 0; it < total; it += NG) {
                tile_body(tile >= full_lo && tile < full_hi, it, tile, ts, tp);
                tile += NG;
                if (COL && tile >= t_hi) {               // the next head of the group
                    tile -= n_sweep;
                    if (NG == 2 && tile >= t_hi) tile -= n_sweep;
                }
                ts += NG * SPT;
                if (ts >= NSLOT) { ts -= NSLOT; tp ^= 1; }
            }
            const int end = s + total * SPT;
            par ^= (end / NSLOT) & 1;
            s = end % NSLOT;
        }

        // ---- epilogue ------------------------------------------------------------------------
        BOB_TR(5)
        exp_base += grp == 0 ? total / 2 : (total + 1) / 2;
        float fwd_k0 = 0.f, fwd_k1 = 0.f;            // forward: weights of the two groups' accumulators
        if constexpr (MODE == kFwd) {
            // both groups' (reference, sum) of my row -> the row's normaliser and lse.  The
            // exchange buffer alternates between items: a thread may start the next item while
            // another still reads this one's values.
            float* xb = red_buf + (n_done & 1) * (2 * NG * 128);
            xb[grp * 128 + row] = m_ref;
            xb[(NG + grp) * 128 + row] = l_run;
            all_sync();
            const float m0 = xb[row], m1 = xb[128 + row];
            const float m = fmaxf(m0, m1);
            const float a0 = fast_exp2(m0 - m), a1 = fast_exp2(m1 - m);
            const float l = a0 * xb[2 * 128 + row] + a1 * xb[3 * 128 + row];
            const float inv = (l > 0.f) ? 1.f / l : 0.f;
            // a group that took no tile of this item has never written its accumulator
            fwd_k0 = (total >= 1) ? a0 * inv : 0.f;
            fwd_k1 = (total >= 2) ? a1 * inv : 0.f;
            if (grp == 0 && own_ok) p.lse[row_stat] = (l > 0.f) ? (m + log2f(l)) * kLn2 : -INFINITY;
        }
        // my row's pk columns, on their way while the row sums are combined and the last products finish
        constexpr int PKN = CFG::STAGED_IO ? DPAD / (NSPLIT * NG) : 1;
        float pk_pre[PKN];
        if constexpr (CFG::STAGED_IO) {
            const int col_pk = (grp * NSPLIT + sp) * PKN;
            const float4* src = reinterpret_cast<const float4*>(p.pk + (tile_row0 + row) * p.D + col_pk);
            #pragma unroll
            for (int i = 0; i < PKN / 4; ++i) {
                float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
                if (own_ok && col_pk + 4 * i < p.D) t = __ldg(src + i);
                pk_pre[4 * i] = t.x; pk_pre[4 * i + 1] = t.y; pk_pre[4 * i + 2] = t.z; pk_pre[4 * i + 3] = t.w;
            }
        }
        (void)pk_pre;
        // TURN_IO: the epilogue operands, chunk lane % 8 of rows turn_row0 ... + 7, on their way meanwhile
        const int turn_row0 = own0 + (warp & 3) * 32 + (lane & 24);
        const int turn_col0 = (grp * NSPLIT + sp) * (DPAD / (NSPLIT * NG));
        constexpr int TURN_N = CFG::TURN_IO ? 8 : 1, TURN_OPER = CFG::TURN_IO && MODE == kBwd2Row ? 8 : 1;
        uint4 turn0[TURN_N], turn1[TURN_N], turn_pk[2][TURN_OPER];       // dQ / first result, out / second result, pk
        (void)turn0; (void)turn1; (void)turn_pk; (void)turn_row0; (void)turn_col0;
        if constexpr (CFG::TURN_IO && MODE == kBwd2Row) {
            const int col = turn_col0 + (lane & 7) * 8, col_pk = turn_col0 + (lane & 7) * 4;
            const uint16_t* g_out = static_cast<const uint16_t*>(p.out) + (long long)batch * p.out_sb + (long long)head * p.out_sh + col;
            const uint16_t* g_dq = static_cast<const uint16_t*>(p.dQ) + (long long)batch * p.dQ_sb + (long long)head * p.dQ_sh + col;
            const float* g_pk = p.pk + ((long long)batch * p.Hq + head) * p.Nq * p.D + col_pk;
            #pragma unroll
            for (int i = 0; i < 8; ++i) {
                const long long r = turn_row0 + i;
                const bool ok = r < n_own;
                const uint4 zero = make_uint4(0, 0, 0, 0);
                turn0[i] = ok && col < p.D ? __ldg(reinterpret_cast<const uint4*>(g_dq + r * p.dQ_sn)) : zero;
                turn1[i] = ok && col < p.D ? __ldg(reinterpret_cast<const uint4*>(g_out + r * p.out_sn)) : zero;
                turn_pk[0][i] = ok && col_pk < p.D ? __ldg(reinterpret_cast<const uint4*>(g_pk + r * p.D)) : zero;
                turn_pk[1][i] = ok && col_pk + 32 < p.D ? __ldg(reinterpret_cast<const uint4*>(g_pk + r * p.D + 32)) : zero;
            }
        }
        float alpha = 0.f, ecirc = 0.f;
        if constexpr (MODE == kBwd2Row) {
            // Every pointwise thread of my row holds a partial sum.  The exchange buffer alternates between items with
            // tiles where there is room for two; elsewhere it is written only once the item's products have finished,
            // which they cannot before every warp has left the epilogue of the previous item with tiles.  An item
            // without tiles has no sums to exchange, and no products to wait for before it could write the buffer.
            constexpr int NPART = NG * NSPLIT;
            if (total > 0) {
                float* xb = red_buf + (CFG::RED_COPIES == 2 ? (n_live & 1) * (2 * NPART * 128) : 0);
                if (CFG::RED_COPIES == 1) wait(bar_done, n_live & 1, kStatusTimeoutPw);
                xb[(grp * NSPLIT + sp) * 128 + row] = acc_a.x + acc_a.y;
                xb[(NPART + grp * NSPLIT + sp) * 128 + row] = acc_b.x + acc_b.y;
                all_sync();
                #pragma unroll
                for (int k = 0; k < NPART; ++k) { alpha += xb[k * 128 + row]; ecirc += xb[(NPART + k) * 128 + row]; }
            }
            if constexpr (CFG::STAGED_IO) wait(bar_io_full, n_done & 1, kStatusTimeoutPw);   // the IO warp has staged out, dQ
            if (grp == 0 && sp == 0 && own_ok) { p.alpha[row_stat] = alpha; p.ecirc[row_stat] = ecirc; }
        }
        if (total > 0) wait(bar_done, n_live & 1, kStatusTimeoutPw);
        last_s = -1;                                 // all products have finished; by the group's next tile the slot may be in use again
        tc_fence_after_sync();
        // the previous item's results have left the staging buffer
        if constexpr (CFG::STAGED_OUT) wait(bar_io_free, (n_done & 1) ^ 1, kStatusTimeoutPw);
        BOB_TR(6)
        {
            constexpr int DC = DPAD / (NSPLIT * NG);    // output columns per pointwise thread
            constexpr int NCH = DC / 16;
            const int res_heads = COL ? p.Hkv : p.Hq;
            // All of my accumulator columns come out of tensor memory first (warp-wide loads), so that
            // the MMA warp may start overwriting them for the next item while I combine and store.
            // (With more than two 16-column chunks per thread that would cost too many registers: then
            // the chunks are taken one at a time and the accumulators are released after the last.)
            constexpr bool EARLY = NCH <= 2;
            float acc0[EARLY ? NCH : 1][16], acc1[EARLY ? NCH : 1][16];
            auto load_chunk = [&](int col, float* a0, float* a1) {
                if (total > 0 && col < p.D) {
                    tmem_ld16(tout + 0 * DPAD + col, a0);
                    if constexpr (CFG::NACC > 1) tmem_ld16(tout + 1 * DPAD + col, a1);
                } else {
                    #pragma unroll
                    for (int i = 0; i < 16; ++i) { a0[i] = 0.f; a1[i] = 0.f; }
                }
            };
            auto release_outputs = [&]() {
                tmem_wait_ld();
                tc_fence_before_sync();
                __syncwarp();
                if (total > 0 && lane == 0) mbar_arrive(bar_out_free);
            };
            if constexpr (EARLY) {
                #pragma unroll
                for (int ch = 0; ch < NCH; ++ch) load_chunk((grp * NSPLIT + sp) * DC + 16 * ch, acc0[ch], acc1[ch]);
                release_outputs();
            }
            // 16 columns of my row into a staged 16-bit tile (two 16-byte chunks)
            auto stage16 = [&](uint32_t tile_base, int col, const float* v) {
                #pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t off = (col / 64) * (128 * 128) + sw128_offset(row, (col % 64) / 8 + i);
                    st_shared_v4(tile_base + off, pack2<BF16>(v[8 * i], v[8 * i + 1]), pack2<BF16>(v[8 * i + 2], v[8 * i + 3]),
                                 pack2<BF16>(v[8 * i + 4], v[8 * i + 5]), pack2<BF16>(v[8 * i + 6], v[8 * i + 7]));
                }
            };
            (void)stage16; (void)res_heads;
            // 16 columns of my row, the c-th of this thread on, as two chunks
            auto pack_chunks = [&](uint4 (&dst)[TURN_N], int c, const float* v) {
                #pragma unroll
                for (int i = 0; i < 2; ++i)
                    dst[c / 8 + i] = make_uint4(pack2<BF16>(v[8 * i], v[8 * i + 1]), pack2<BF16>(v[8 * i + 2], v[8 * i + 3]),
                                                pack2<BF16>(v[8 * i + 4], v[8 * i + 5]), pack2<BF16>(v[8 * i + 6], v[8 * i + 7]));
            };
            (void)pack_chunks;
            // rows turned around by transpose_chunks, as 16-byte chunks at column offset `col` of my eight rows
            auto store_turned = [&](auto* base, const uint4 (&c)[8], int col) {
                auto* dst = base + (((long long)batch * res_heads + head) * n_own + turn_row0) * p.D + col;
                #pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (turn_row0 + i < n_own && col < p.D) *reinterpret_cast<uint4*>(dst + (long long)i * p.D) = c[i];
            };
            (void)store_turned;
            if constexpr (CFG::TURN_IO && MODE == kBwd2Row) {
                transpose_chunks(turn0, lane);           // now my own row's 64 columns
                transpose_chunks(turn1, lane);
                transpose_chunks(turn_pk[0], lane);
                transpose_chunks(turn_pk[1], lane);
            }
            #pragma unroll
            for (int c = 0; c < DC; c += 16) {
                const int col = (grp * NSPLIT + sp) * DC + c;
                float late0[16], late1[16];
                if constexpr (!EARLY) {
                    load_chunk(col, late0, late1);
                    if (c + 16 >= DC) release_outputs(); else tmem_wait_ld();
                }
                float* a0 = EARLY ? acc0[EARLY ? c / 16 : 0] : late0;
                float* a1 = EARLY ? acc1[EARLY ? c / 16 : 0] : late1;
                if (col >= p.D) continue;
                if constexpr (MODE == kFwd) {
                    // weighted sum of the two groups' accumulators (weight 0: never written, not read)
                    #pragma unroll
                    for (int i = 0; i < 16; ++i)
                        a0[i] = (fwd_k0 != 0.f ? fwd_k0 * a0[i] : 0.f) + (fwd_k1 != 0.f ? fwd_k1 * a1[i] : 0.f);
                    stage16(io_out, col, a0);
                } else if constexpr (MODE == kBwd1Row) {
                    #pragma unroll
                    for (int i = 0; i < 16; ++i) a0[i] *= p.scale;
                    stage16(io_out, col, a0);                                                     // dQ
                    if (p.pk) {                                                                   // PK
                        if constexpr (CFG::STAGED_PK) {
                            const uint32_t base = io_out + CFG::OWN_TILE_BYTES + (col / 32) * (128 * 128);
                            #pragma unroll
                            for (int i = 0; i < 4; ++i)
                                st_shared_v4(base + sw128_offset(row, (col % 32) / 4 + i), __float_as_uint(a1[4 * i]), __float_as_uint(a1[4 * i + 1]),
                                             __float_as_uint(a1[4 * i + 2]), __float_as_uint(a1[4 * i + 3]));
                        }
                    }
                } else if constexpr (COL) {
                    #pragma unroll
                    for (int i = 0; i < 16; ++i) a0[i] *= p.scale;
                    if constexpr (CFG::STAGED_OUT) {
                        stage16(io_out, col, a0);
                        stage16(io_out + CFG::OWN_TILE_BYTES, col, a1);
                    } else {
                        pack_chunks(turn0, c, a0);
                        pack_chunks(turn1, c, a1);
                    }
                } else {
                    if (CFG::STAGED_IO && !own_ok) continue;
                    // accumulators: a0 = P uV + (P*F) V, a1 = (P*T) K + dS uK;  PK comes from the first backward
                    float o[16], g[16], pkv[16];
                    if constexpr (CFG::STAGED_IO) {
                        const uint32_t sw = row & 7;
                        #pragma unroll
                        for (int i = 0; i < 16; ++i) pkv[i] = pk_pre[c + i];
                        #pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint32_t off = row * 128 + (((col / 8 + i) ^ sw) << 4);
                            unpack8_as_float<BF16>(ld_shared_v4(io_out + off), o + 8 * i);
                            unpack8_as_float<BF16>(ld_shared_v4(io_dq + off), g + 8 * i);
                        }
                    } else {
                        #pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint4 t = turn_pk[c / 32][(c % 32) / 4 + i];
                            pkv[4 * i] = __uint_as_float(t.x); pkv[4 * i + 1] = __uint_as_float(t.y);
                            pkv[4 * i + 2] = __uint_as_float(t.z); pkv[4 * i + 3] = __uint_as_float(t.w);
                        }
                        #pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            unpack8_as_float<BF16>(turn1[c / 8 + i], o + 8 * i);
                            unpack8_as_float<BF16>(turn0[c / 8 + i], g + 8 * i);
                        }
                    }
                    #pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float dob = a0[i] - alpha * o[i];                                   // dObar
                        const float qb = p.scale * (a1[i] - ecirc * pkv[i]) - alpha * g[i];       // Qbar
                        a0[i] = qb; a1[i] = dob;
                    }
                    if constexpr (CFG::STAGED_IO) {
                        // results replace my own chunks of the staged operands: Qbar over dQ, dObar over out
                        stage16(io_dq, col, a0);
                        stage16(io_out, col, a1);
                    } else {
                        pack_chunks(turn0, c, a0);
                        pack_chunks(turn1, c, a1);
                    }
                }
            }
            if constexpr (CFG::TURN_IO) {
                transpose_chunks(turn0, lane);
                transpose_chunks(turn1, lane);
                store_turned(static_cast<uint16_t*>(p.res0), turn0, turn_col0 + (lane & 7) * 8);
                store_turned(static_cast<uint16_t*>(p.res1), turn1, turn_col0 + (lane & 7) * 8);
            }
            if constexpr (CFG::TURN_PK) {
                if (p.pk) {
                    uint4 t[8];
                    #pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float* a1 = acc1[EARLY ? i / 4 : 0] + 4 * (i % 4);
                        t[i] = make_uint4(__float_as_uint(a1[0]), __float_as_uint(a1[1]), __float_as_uint(a1[2]), __float_as_uint(a1[3]));
                    }
                    transpose_chunks(t, lane);
                    store_turned(p.pk, t, turn_col0 + (lane & 7) * 4);
                }
            }
        }
        if constexpr (CFG::STAGED_IO || CFG::STAGED_OUT) {
            // my rows' results are in shared memory: the fourth role warp sends the tile off
            if constexpr (CFG::STAGED_OUT) fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_io_ready);
        }
        if (total > 0) ++n_live;
        ++n_done;
        BOB_TR(7)
        }   // items
        BOB_TR_FLUSH
    }
#undef BOB_ITEM_LOCALS

    // ---- teardown --------------------------------------------------------------------------------
    tc_fence_before_sync();
    __syncthreads();
    if (warp == NPW / 32) {
        __syncwarp();
        tmem_dealloc(tmem, CFG::TMEM_COLS);
    }
}

}  // namespace bob
