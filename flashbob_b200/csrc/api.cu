// Host side of the C ABI: argument checks, tensor-map construction and kernel dispatch.
#include "internal.h"
#include "decode.cuh"
#include "sweep.cuh"
#include "tmap.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace bob {

enum : int {
    kErrNull = -1, kErrGeom = -2, kErrDtype = -3, kErrHeadDim = -4, kErrStride = -5,
    kErrWorkspace = -6, kErrDevice = -7, kErrLaunch = -8, kErrAttr = -9, kErrAlign = -10, kErrRegs = -13,
    kErrNoDriver = -100,
};

// The first 256 bytes of every workspace: word 0 = status, words 8.. = work counters of the launches
// of one call.  The whole block is cleared by each call.
static constexpr size_t kStatusBlock = 256;
static constexpr int kCounterWord0 = 8;

static size_t round256(size_t x) { return (x + 255) / 256 * 256; }

static int check_geom(const bob_sm100_geom* g) {
    if (!g) return kErrNull;
    if (g->B <= 0 || g->Hq <= 0 || g->Hkv <= 0 || g->Nq <= 0 || g->Nk <= 0 || g->D <= 0) return kErrGeom;
    if (g->Hq % g->Hkv) return kErrGeom;
    if (g->Nq > (1 << 28) || g->Nk > (1 << 28)) return kErrGeom;
    if (g->dtype != BOB_SM100_FP16 && g->dtype != BOB_SM100_BF16) return kErrDtype;
    if (g->D % 16 || g->D > 128) return kErrHeadDim;
    if (g->window < 0 || (g->window > 0 && !g->is_causal)) return kErrGeom;
    if (g->q_offset < 0 || g->k_offset < 0) return kErrGeom;
    if (!(g->scale > 0.f) || !std::isfinite(g->scale)) return kErrGeom;
    return 0;
}

// Results are written with 16-byte stores, pk is read and written as float4.
static int check_aligned16(std::initializer_list<const void*> ptrs) {
    for (const void* p : ptrs)
        if (reinterpret_cast<uintptr_t>(p) % 16) return kErrAlign;
    return 0;
}
static int check_aligned4(std::initializer_list<const void*> ptrs) {
    for (const void* p : ptrs)
        if (reinterpret_cast<uintptr_t>(p) % 4) return kErrAlign;
    return 0;
}

static int check_strides(const int64_t* s, const void* ptr) {
    if (reinterpret_cast<uintptr_t>(ptr) % 16) return kErrAlign;
    for (int i = 0; i < 3; ++i)
        if (s[i] < 0 || s[i] % 8) return kErrStride;
    return 0;
}

struct DeviceGuard {
    int prev = -1;
    bool ok = true;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) { ok = false; return; }
        if (prev != dev && cudaSetDevice(dev) != cudaSuccess) ok = false;
        changed = prev != dev;
    }
    ~DeviceGuard() { if (changed && prev >= 0) cudaSetDevice(prev); }
    bool changed = false;
};

// Number of SMs of a device (cached: the attribute query is slow enough to show at small sizes).
static int sm_count(int device) {
    static int cache[64] = {};
    if (device < 0 || device >= 64) return -1;
    if (cache[device] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0) return -1;
        cache[device] = n;
    }
    return cache[device];
}

struct TensorArg {
    const void* ptr;
    const int64_t* strides;   // batch, head, row
    bool q_side;              // [B, Hq, Nq, D] (true) or [B, Hkv, Nk, D] (false)
};

// Raises a kernel's shared-memory limit, once per device: the attribute calls are slow enough to show at
// small sizes.
template <class CFG, class Kernel>
static int prepare_kernel(Kernel kernel, int device, std::atomic<uint64_t>& done) {
    const uint64_t bit = 1ull << device;
    if (done.load(std::memory_order_acquire) & bit) return 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CFG::SMEM_BYTES) != cudaSuccess) return kErrAttr;
    // The kernel's warpgroups trade registers after launch; the trade only balances (and the pointwise
    // warps' request can only ever be met) if the kernel was built with the register count the trade
    // assumes.  Refuse to launch otherwise.
    cudaFuncAttributes a;
    const int regs_at_launch = cudaFuncGetAttributes(&a, kernel) == cudaSuccess ? a.numRegs : 0;
    if (regs_at_launch * CFG::NTHREADS < CFG::NPW * CFG::REGS_POINTWISE + 128 * CFG::REGS_ROLE) return kErrRegs;
    done.fetch_or(bit, std::memory_order_release);
    return 0;
}

template <int MODE, int DPAD, int TN, bool BF16, int NG, int CW, bool ALIAS>
static int launch_sweep(const bob_sm100_geom* g, SweepParams& prm, const TensorArg* tensors,
                        cudaStream_t stream, int counter_slot) {
    using CFG = SweepConfig<MODE, DPAD, TN, NG, CW, ALIAS>;
    using MT = ModeTraits<MODE>;
    constexpr TileType kType = BF16 ? TileType::kBF16 : TileType::kF16;
    auto build = [&](int t, int box_rows) -> int {
        const TensorArg& a = tensors[t];
        if (!a.ptr) return 0;
        int rc = check_strides(a.strides, a.ptr);
        if (rc) return rc;
        return make_tile_map(&prm.map[t], a.ptr, kType, g->D, a.q_side ? g->Nq : g->Nk,
                             a.q_side ? g->Hq : g->Hkv, g->B, a.strides[2], a.strides[1],
                             a.strides[0], box_rows);
    };
    for (int i = 0; i < MT::NOWN; ++i) {
        int rc = build(own_tensor<MODE>(i), 128);
        if (rc) return rc;
    }
    if (CFG::OWN_OUT && !prm.out) {
        int rc = build(kTOUT, 128);
        if (rc) return rc;
    }
    for (int i = 0; i < MT::NOTH; ++i) {
        int rc = build(other_tensor<MODE>(i), TN);
        if (rc) return rc;
    }
    // results: contiguous [B, H, N, D]
    const int n_own = MT::COL ? g->Nk : g->Nq, heads = MT::COL ? g->Hkv : g->Hq;
    auto result = [&](int i, const void* ptr, TileType type) -> int {
        const int64_t sn = g->D, sh = sn * n_own;
        return make_tile_map(&prm.res_map[i], ptr, type, g->D, n_own, heads, g->B, sn, sh, sh * heads, 128);
    };
    if (CFG::N_STAGED > 0) { if (int rc = result(0, prm.res0, kType)) return rc; }
    if (CFG::N_STAGED > 1) { if (int rc = result(1, prm.res1, kType)) return rc; }
    if (CFG::STAGED_PK && prm.pk) { if (int rc = result(2, prm.pk, TileType::kF32)) return rc; }
    if (g->device < 0 || g->device >= 64) return kErrDevice;
    // The second backward has a build of its own for the usual case of three defined tangents.
    constexpr bool kSecond = (MODE == kBwd2Row || MODE == kBwd2Col);
    const bool allt = kSecond && prm.has_uq && prm.has_uk && prm.has_uv;
    auto kernel = allt ? sweep_kernel<MODE, DPAD, TN, BF16, NG, CW, ALIAS, kSecond>
                       : sweep_kernel<MODE, DPAD, TN, BF16, NG, CW, ALIAS, false>;
    static std::atomic<uint64_t> done[2];
    if (int rc = prepare_kernel<CFG>(kernel, g->device, done[allt])) return rc;
    const long long items = (long long)((n_own + 127) / 128) * heads * g->B;
    if (items > 0x7fffffffLL) return kErrGeom;
    const int sms = sm_count(g->device);
    if (sms <= 0) return kErrDevice;
    // One persistent CTA per SM whenever there are more items than SMs; it takes items, longest first, from a
    // counter in the status block (zeroed with it).
    const bool persistent = items > sms;
    dim3 grid((unsigned)(persistent ? sms : items), 1, 1);
    prm.work_counter = persistent ? prm.status + kCounterWord0 + counter_slot : nullptr;
    kernel<<<grid, CFG::NTHREADS, CFG::SMEM_BYTES, stream>>>(prm);
    return cudaGetLastError() == cudaSuccess ? 0 : kErrLaunch;
}

// Tile table (template arguments: head dim, swept-tile width, dtype, pointwise groups, score columns
// per pointwise thread, operands over the scores).
// Head dim <= 64.  Forward: 128-wide tiles, two groups of 128 threads, each thread a whole row, each
// group its own online softmax and output accumulator.  First backward: 64-wide tiles, two groups of 256
// threads.  Second backward: four score accumulators, four operands and two outputs fill tensor memory at
// 64-wide tiles; one group of 256 threads holds a whole tile's columns at 208 registers.
// Head dim 128.  Forward and first backward as above, with the operands over the scores: the output
// accumulators take half of tensor memory.  Second backward: room for 32-wide tiles only.
template <int MODE, bool BF16>
static int dispatch(const bob_sm100_geom* g, SweepParams& prm, const TensorArg* tensors,
                    cudaStream_t stream, int counter_slot) {
    constexpr bool kSecond = (MODE == kBwd2Row || MODE == kBwd2Col);
    if (g->D <= 64) {
        if constexpr (kSecond)           return launch_sweep<MODE, 64, 64, BF16, 1, 32, false>(g, prm, tensors, stream, counter_slot);
        else if constexpr (MODE == kFwd) return launch_sweep<MODE, 64, 128, BF16, 2, 128, false>(g, prm, tensors, stream, counter_slot);
        else                             return launch_sweep<MODE, 64, 64, BF16, 2, 32, false>(g, prm, tensors, stream, counter_slot);
    }
    if constexpr (kSecond)           return launch_sweep<MODE, 128, 32, BF16, 1, 16, false>(g, prm, tensors, stream, counter_slot);
    else if constexpr (MODE == kFwd) return launch_sweep<MODE, 128, 128, BF16, 2, 128, true>(g, prm, tensors, stream, counter_slot);
    else                             return launch_sweep<MODE, 128, 64, BF16, 2, 32, true>(g, prm, tensors, stream, counter_slot);
}

template <int MODE>
static int dispatch_dtype(const bob_sm100_geom* g, SweepParams& prm, const TensorArg* tensors,
                          cudaStream_t stream, int counter_slot) {
    return g->dtype == BOB_SM100_BF16 ? dispatch<MODE, true>(g, prm, tensors, stream, counter_slot)
                                      : dispatch<MODE, false>(g, prm, tensors, stream, counter_slot);
}

// Only builds with -DBOB_TRACE (never the shipped library) read a device pointer (hex) from BOB_SM100_TRACE_PTR.
static long long* trace_pointer() {
#if defined(BOB_TRACE)
    const char* e = std::getenv("BOB_SM100_TRACE_PTR");
    return e ? reinterpret_cast<long long*>(std::strtoull(e, nullptr, 16)) : nullptr;
#else
    return nullptr;
#endif
}

// A per-device word in host memory that kernels can write: a CTA whose bounded wait ran out stores its
// status code there as well as in the workspace, so the host can notice without synchronising
// (bob_sm100_last_status).  Page-locked once per device on first use; null if that failed.
int* sticky_word(int device, bool create) {
    static std::mutex mu;
    static int* host[64] = {};
    static int* dev[64] = {};
    static bool tried[64] = {};
    if (device < 0 || device >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!tried[device] && create) {
        tried[device] = true;
        void* h = nullptr;
        void* d = nullptr;
        if (cudaHostAlloc(&h, 64, cudaHostAllocMapped | cudaHostAllocPortable) == cudaSuccess) {
            std::memset(h, 0, 64);
            if (cudaHostGetDevicePointer(&d, h, 0) == cudaSuccess) {
                host[device] = static_cast<int*>(h);
                dev[device] = static_cast<int*>(d);
            } else {
                cudaFreeHost(h);
            }
        }
        cudaGetLastError();
    }
    return create ? dev[device] : host[device];
}

static void fill_mask(const bob_sm100_geom* g, SweepParams& p) {
    p.is_causal = g->is_causal ? 1 : 0;
    // Lengths are at most 2^28.  Beyond +-2^29 the causal condition has the same outcome for every pair as at
    // the bound; a window moves with the part of the offset that is cut off, and one beyond 2^30 excludes
    // nothing.  32-bit position arithmetic in the kernels then cannot overflow.
    const int64_t kBound = 1 << 29, d = g->q_offset - g->k_offset;
    const int64_t dc = std::min(kBound, std::max(-kBound, d));
    p.delta_off = static_cast<int>(dc);
    p.window = g->window > 0 ? static_cast<int>(std::min<int64_t>(1 << 30, std::max<int64_t>(1, g->window - (d - dc)))) : 0;
}

static void fill_common(const bob_sm100_geom* g, SweepParams& p, void* workspace) {
    std::memset(&p, 0, sizeof(p));
    p.B = g->B; p.Hq = g->Hq; p.Hkv = g->Hkv; p.G = g->Hq / g->Hkv; p.Nq = g->Nq; p.Nk = g->Nk;
    p.D = g->D;
    fill_mask(g, p);
    p.scale = g->scale;
    p.status = static_cast<int*>(workspace);
    p.trace = trace_pointer();
}

static void set_strided(const void*& dst, long long& sb, long long& sh, long long& sn,
                        const void* ptr, const int64_t* s) {
    dst = ptr; sb = s[0]; sh = s[1]; sn = s[2];
}

// ---- forward with a few query rows ------------------------------------------------------------------
// decode_kernel divides a head's keys until kDecodeCtas CTAs are there (two are resident per SM), but not below one
// round of a CTA's warps.  (The numbers are B200's and not asked of the device, so that the workspace's size
// depends on the geometry alone.)
constexpr int kSms = 148, kDecodeCtas = 4 * kSms;
struct DecodePlan { int k_lo, k_hi, splits, split_keys; size_t acc_offset, bytes; };     // offsets in the workspace

static int decode_dpad(const bob_sm100_geom* g) { return g->D <= 32 ? 32 : (g->D <= 64 ? 64 : 128); }

static DecodePlan decode_plan(const bob_sm100_geom* g) {
    DecodePlan d = {};
    SweepParams p;
    fill_mask(g, p);
    int64_t lo = 0, hi = g->Nk;                  // keys that any of the rows attends to
    if (p.is_causal) {
        hi = std::min<int64_t>(hi, (int64_t)g->Nq + p.delta_off);
        if (p.window > 0) lo = std::max<int64_t>(0, (int64_t)p.delta_off - p.window + 1);
    }
    if (hi < lo) hi = lo = 0;
    d.k_lo = (int)lo; d.k_hi = (int)hi;
    const int64_t round = decode_round(decode_dpad(g), g->Nq), rounds = std::max<int64_t>(1, (hi - lo + round - 1) / round);
    const int64_t heads = (int64_t)g->B * g->Hq;
    const int64_t want = std::min<int64_t>({kDecodeMaxSplits, rounds, std::max<int64_t>(1, kDecodeCtas / heads)});
    const int64_t per = (rounds + want - 1) / want;
    d.split_keys = (int)(per * round);
    d.splits = (int)((rounds + per - 1) / per);
    d.bytes = kStatusBlock;
    if (d.splits > 1) {
        const size_t rows = (size_t)heads * d.splits * g->Nq;
        const size_t ml_offset = kStatusBlock + round256(heads * sizeof(int));
        d.acc_offset = ml_offset + round256(rows * 2 * sizeof(float));
        d.bytes = d.acc_offset + rows * g->D * sizeof(float);
    }
    return d;
}

// Whether a forward goes to decode_kernel.  The sweep kernel does the work of 128 rows for a few, but on the tensor cores
// and the special-function unit, and its time grows with the rounds of one CTA per head; decode_kernel's arithmetic grows
// with rows x heads x keys.  Measured, us, decode / sweep kernel, bf16, 4096 keys unless given:
//   one row     128 heads D=64 31.9 / 39.0, D=128 51.4 / 53.4, 512 keys 17.4 / 16.5; 1024 heads D=64 166 / 219; 2 heads 10 / 37
//   four rows   heads x D up to 4096 per round of 148 heads: 64 heads D=64 35 / 38, 32 heads D=128 37 / 47, 160 heads D=32 41 / 68
//               beyond: 96 heads D=64 47 / 38, 64 heads D=128 57 / 49, 148 heads D=128 103 / 56, 512 keys 27 / 17
//               keys for one round of a CTA's warps: 128 heads 64 keys D=128 6 / 12, 1024 heads 24 / 39
// (two and three rows as four).  Without divided keys, which need a workspace of their size (BOB_SM100_SPLIT_KEYS), the
// sweep kernel reads a long head faster.
static bool takes_decode(const bob_sm100_geom* g) {
    if (g->Nq > kDecodeRows) return false;
    const DecodePlan d = decode_plan(g);
    if (d.splits > 1 && !(g->flags & BOB_SM100_SPLIT_KEYS)) return false;
    const int64_t heads = (int64_t)g->B * g->Hq;
    return g->Nq == 1 || d.k_hi - d.k_lo <= decode_round(decode_dpad(g), g->Nq) || heads * decode_dpad(g) <= 4096 * ((heads + kSms - 1) / kSms);
}

template <bool BF16>
static void launch_decode(const bob_sm100_geom* g, const DecodeParams& p, unsigned grid, cudaStream_t s) {
    auto rows = [&](auto dpad_tag) {
        constexpr int DPAD = decltype(dpad_tag)::value;
        if (g->Nq == 1) decode_kernel<DPAD, 1, BF16><<<grid, kDecodeThreads, 0, s>>>(p);
        else decode_kernel<DPAD, kDecodeRows, BF16><<<grid, kDecodeThreads, 0, s>>>(p);
    };
    if (g->D <= 32) rows(IntTag<32>{});
    else if (g->D <= 64) rows(IntTag<64>{});
    else rows(IntTag<128>{});
}

static int run_decode(const bob_sm100_geom* g, const void* q, const void* k, const void* v, void* out, float* lse,
                      void* workspace, cudaStream_t s) {
    // the same layouts as the sweep kernels take
    auto check = [&](const void* ptr, const int64_t* st, int64_t N, int64_t H) -> int {
        if (int rc = check_strides(st, ptr)) return rc;
        int64_t sn = st[2], sh = st[1], sb = st[0];
        return fit_strides(g->D, N, H, g->B, sn, sh, sb, TileType::kF16);
    };
    if (int rc = check(q, g->q_strides, g->Nq, g->Hq)) return rc;
    if (int rc = check(k, g->k_strides, g->Nk, g->Hkv)) return rc;
    if (int rc = check(v, g->v_strides, g->Nk, g->Hkv)) return rc;
    const DecodePlan d = decode_plan(g);
    const int64_t heads = (int64_t)g->B * g->Hq, grid = heads * d.splits;
    if (grid > 0x7fffffffLL) return kErrGeom;
    SweepParams m;
    fill_mask(g, m);
    char* ws = static_cast<char*>(workspace);
    DecodeParams p = {};
    p.q = static_cast<const uint16_t*>(q); p.q_sb = g->q_strides[0]; p.q_sh = g->q_strides[1]; p.q_sn = g->q_strides[2];
    p.k = static_cast<const uint16_t*>(k); p.k_sb = g->k_strides[0]; p.k_sh = g->k_strides[1]; p.k_sn = g->k_strides[2];
    p.v = static_cast<const uint16_t*>(v); p.v_sb = g->v_strides[0]; p.v_sh = g->v_strides[1]; p.v_sn = g->v_strides[2];
    p.Hq = g->Hq; p.G = g->Hq / g->Hkv; p.Nq = g->Nq; p.D = g->D;
    p.causal = m.is_causal; p.window = m.window; p.delta_off = m.delta_off;
    p.k_lo = d.k_lo; p.k_hi = d.k_hi; p.splits = d.splits; p.split_keys = d.split_keys;
    p.scale = g->scale;
    p.out = static_cast<uint16_t*>(out);
    p.lse = lse;
    p.status = reinterpret_cast<int*>(ws);
    if (d.splits > 1) {
        p.arrived = reinterpret_cast<int*>(ws + kStatusBlock);
        p.part_ml = reinterpret_cast<float*>(ws + kStatusBlock + round256(heads * sizeof(int)));
        p.part_acc = reinterpret_cast<float*>(ws + d.acc_offset);
        if (cudaMemsetAsync(p.arrived, 0, heads * sizeof(int), s) != cudaSuccess) return kErrLaunch;
    }
    if (g->dtype == BOB_SM100_BF16) launch_decode<true>(g, p, (unsigned)grid, s);
    else launch_decode<false>(g, p, (unsigned)grid, s);
    return cudaGetLastError() == cudaSuccess ? 0 : kErrLaunch;
}

}  // namespace bob

using namespace bob;

extern "C" int bob_sm100_version(void) { return 100; }

extern "C" const char* bob_sm100_error_string(int code) {
    switch (code) {
        case 0: return "ok";
        case kErrNull: return "null pointer argument";
        case kErrGeom: return "invalid geometry (sizes, heads, window, offsets or scale)";
        case kErrDtype: return "dtype must be fp16 (0) or bf16 (1)";
        case kErrHeadDim: return "head dimension must be a multiple of 16, at most 128";
        case kErrStride: return "tensor strides must be non-negative multiples of 8 elements";
        case kErrWorkspace: return "workspace missing or misaligned";
        case kErrDevice: return "cannot select the device";
        case kErrLaunch: return "kernel launch failed";
        case kErrAttr: return "cannot raise the dynamic shared memory limit";
        case kErrAlign: return "tensor base address must be 16-byte aligned";
        case kErrRegs: return "kernel was built with too few registers for its register rebalancing";
        case kErrNoDriver: return "cuTensorMapEncodeTiled is unavailable in this driver";
        case -11: return "cannot resolve the built-in scratch array on this device";
        case -12: return "problem too large for the built-in scratch (B*Hq*Nq > 1048576 rows)";
        case -101: return "tensor base address must be 16-byte aligned";
        case -102: return "tensor strides unusable for TMA";
        case 77: return "device: the self-test's wait ran out (as it is meant to)";
        case kStatusTimeoutLoad: return "device: a wait for a TMA load ran out";
        case kStatusTimeoutMma: return "device: a wait in the MMA issuer ran out";
        case kStatusMisaligned: return "device: shared memory is not 1024-byte aligned";
        case kStatusTimeoutPw: return "device: a wait in the pointwise threads ran out";
        default: return code < -1000 ? "cuTensorMapEncodeTiled failed" : "unknown code";
    }
}

extern "C" size_t bob_sm100_workspace_bytes(int stage, const bob_sm100_geom* g) {
    if (!g || g->B <= 0 || g->Hq <= 0 || g->Hkv <= 0 || g->Nq <= 0 || g->Nk <= 0) return 0;
    size_t bytes = kStatusBlock;
    if (stage == BOB_SM100_STAGE_BWD2) bytes = bwd2_workspace_bytes(g);
    if (stage == BOB_SM100_STAGE_FWD && takes_decode(g)) bytes = decode_plan(g).bytes;
    return bytes;
}

extern "C" int bob_sm100_kernel_launches(int stage, const bob_sm100_geom* g) {
    (void)g;
    return stage == BOB_SM100_STAGE_FWD ? 1 : 2;    // one sweep, or a row-owned and a column-owned sweep
}

extern "C" int bob_sm100_read_status(const void* workspace, void* stream) {
    if (!workspace) return kErrNull;
    int v = 0;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (cudaMemcpyAsync(&v, workspace, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return kErrLaunch;
    if (cudaStreamSynchronize(s) != cudaSuccess) return kErrLaunch;
    return v;
}

extern "C" int bob_sm100_last_status(int device) {
    int* w = sticky_word(device, false);
    if (!w) return 0;
    return __atomic_exchange_n(w, 0, __ATOMIC_ACQ_REL);
}

// Clears the status block (status word and work counters) of a call's workspace.
static int begin_call(void* workspace, cudaStream_t s) {
    if (!workspace || reinterpret_cast<uintptr_t>(workspace) % 256) return kErrWorkspace;
    return cudaMemsetAsync(workspace, 0, kStatusBlock, s) == cudaSuccess ? 0 : kErrLaunch;
}

extern "C" int bob_sm100_fwd(const bob_sm100_geom* g, const void* q, const void* k, const void* v,
                             void* out, float* lse, void* workspace, void* stream) {
    int rc = check_geom(g);
    if (rc) return rc;
    if (!q || !k || !v || !out || !lse) return kErrNull;
    if ((rc = check_aligned16({out}))) return rc;
    if ((rc = check_aligned4({lse}))) return rc;
    if (!workspace || reinterpret_cast<uintptr_t>(workspace) % 256) return kErrWorkspace;
    DeviceGuard guard(g->device);
    if (!guard.ok) return kErrDevice;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int* sticky = sticky_word(g->device, true);
    if (takes_decode(g)) return run_decode(g, q, k, v, out, lse, workspace, s);
    if ((rc = begin_call(workspace, s))) return rc;

    SweepParams p;
    fill_common(g, p, workspace);
    p.sticky = sticky;
    p.lse = lse;
    p.res0 = out;
    TensorArg t[kNumTensors] = {};
    t[kTQ] = {q, g->q_strides, true};
    t[kTK] = {k, g->k_strides, false};
    t[kTV] = {v, g->v_strides, false};
    return dispatch_dtype<kFwd>(g, p, t, s, 0);
}

extern "C" int bob_sm100_bwd1(const bob_sm100_geom* g, const void* q, const void* k, const void* v,
                              const void* out, const float* lse, const void* dO, void* dQ, void* dK,
                              void* dV, float* delta, float* pk, void* workspace, void* stream) {
    int rc = check_geom(g);
    if (rc) return rc;
    if (!q || !k || !v || !out || !lse || !dO || !dQ || !dK || !dV || !delta) return kErrNull;
    if ((rc = check_aligned16({dQ, dK, dV, pk}))) return rc;
    if ((rc = check_aligned4({lse, delta}))) return rc;
    if (!workspace || reinterpret_cast<uintptr_t>(workspace) % 256) return kErrWorkspace;
    if ((rc = check_strides(g->out_strides, out))) return rc;
    if ((rc = check_strides(g->do_strides, dO))) return rc;
    DeviceGuard guard(g->device);
    if (!guard.ok) return kErrDevice;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if ((rc = begin_call(workspace, s))) return rc;

    TensorArg t[kNumTensors] = {};
    t[kTQ] = {q, g->q_strides, true};
    t[kTK] = {k, g->k_strides, false};
    t[kTV] = {v, g->v_strides, false};
    t[kTDO] = {dO, g->do_strides, true};
    t[kTOUT] = {out, g->out_strides, true};

    SweepParams p;
    fill_common(g, p, workspace);
    p.sticky = sticky_word(g->device, true);
    p.lse = const_cast<float*>(lse);
    p.delta = delta;
    p.pk = pk;
    p.res0 = dQ;
    int64_t sn = g->out_strides[2], sh = g->out_strides[1], sb = g->out_strides[0];
    if (fit_strides(g->D, g->Nq, g->Hq, g->B, sn, sh, sb, TileType::kF16))      // an expanded `out`: no tile of it
        set_strided(p.out, p.out_sb, p.out_sh, p.out_sn, out, g->out_strides);
    rc = dispatch_dtype<kBwd1Row>(g, p, t, s, 0);   // dQ and delta
    if (rc) return rc;
    p.res0 = dK;
    p.res1 = dV;
    return dispatch_dtype<kBwd1Col>(g, p, t, s, 1); // dK and dV (reads delta)
}

int bob::bwd2_impl(const bob_sm100_geom* g, const void* q, const void* k, const void* v, const void* out,
                   const float* lse, const float* delta, const float* pk, const void* dO, const void* dQ,
                   const void* uQ, const void* uK, const void* uV, void* Qbar, void* Kbar, void* Vbar,
                   void* dObar, void* workspace, void* stream, int* sticky, int part) {
    int rc = check_geom(g);
    if (rc) return rc;
    if (!q || !k || !v || !out || !lse || !delta || !pk || !dO || !dQ || !Qbar || !Kbar || !Vbar || !dObar)
        return kErrNull;
    if (part < kPartRow || part > kPartBoth) return kErrGeom;
    if ((rc = check_aligned16({Qbar, Kbar, Vbar, dObar, pk}))) return rc;
    if ((rc = check_aligned4({lse, delta}))) return rc;
    if (!workspace || reinterpret_cast<uintptr_t>(workspace) % 256) return kErrWorkspace;
    if ((rc = check_strides(g->out_strides, out))) return rc;
    if ((rc = check_strides(g->dq_strides, dQ))) return rc;
    DeviceGuard guard(g->device);
    if (!guard.ok) return kErrDevice;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if ((rc = begin_call(workspace, s))) return rc;

    TensorArg t[kNumTensors] = {};
    t[kTQ] = {q, g->q_strides, true};
    t[kTK] = {k, g->k_strides, false};
    t[kTV] = {v, g->v_strides, false};
    t[kTDO] = {dO, g->do_strides, true};
    t[kTUQ] = {uQ, g->uq_strides, true};
    t[kTUK] = {uK, g->uk_strides, false};
    t[kTUV] = {uV, g->uv_strides, false};

    SweepParams p;
    fill_common(g, p, workspace);
    p.sticky = sticky;
    p.has_uq = uQ != nullptr; p.has_uk = uK != nullptr; p.has_uv = uV != nullptr;
    p.lse = const_cast<float*>(lse);
    p.delta = const_cast<float*>(delta);
    p.pk = const_cast<float*>(pk);
    const size_t stat_bytes = round256(static_cast<size_t>(g->B) * g->Hq * g->Nq * sizeof(float));
    p.alpha = reinterpret_cast<float*>(static_cast<char*>(workspace) + kStatusBlock);
    p.ecirc = reinterpret_cast<float*>(static_cast<char*>(workspace) + kStatusBlock + stat_bytes);
    set_strided(p.out, p.out_sb, p.out_sh, p.out_sn, out, g->out_strides);
    set_strided(p.dQ, p.dQ_sb, p.dQ_sh, p.dQ_sn, dQ, g->dq_strides);
    if (part & kPartRow) {
        p.res0 = Qbar;
        p.res1 = dObar;
        rc = dispatch_dtype<kBwd2Row>(g, p, t, s, 0);   // Qbar, dObar, alpha, ecirc
        if (rc) return rc;
    }
    if (part & kPartCol) {
        p.res0 = Kbar;
        p.res1 = Vbar;
        rc = dispatch_dtype<kBwd2Col>(g, p, t, s, 1);   // Kbar, Vbar (reads alpha, ecirc)
    }
    return rc;
}

size_t bob::bwd2_workspace_bytes(const bob_sm100_geom* g) {
    return kStatusBlock + 2 * round256(static_cast<size_t>(g->B) * g->Hq * g->Nq * sizeof(float));
}

extern "C" int bob_sm100_bwd2(const bob_sm100_geom* g, const void* q, const void* k, const void* v,
                              const void* out, const float* lse, const float* delta, const float* pk,
                              const void* dO, const void* dQ, const void* uQ, const void* uK, const void* uV,
                              void* Qbar, void* Kbar, void* Vbar, void* dObar, void* workspace,
                              void* stream) {
    return bwd2_impl(g, q, k, v, out, lse, delta, pk, dO, dQ, uQ, uK, uV, Qbar, Kbar, Vbar, dObar, workspace,
                     stream, g ? sticky_word(g->device, true) : nullptr, kPartBoth);
}

extern "C" int bob_sm100_bwd2_part(int part, const bob_sm100_geom* g, const void* q, const void* k,
                                   const void* v, const void* out, const float* lse, const float* delta,
                                   const float* pk, const void* dO, const void* dQ, const void* uQ,
                                   const void* uK, const void* uV, void* Qbar, void* Kbar, void* Vbar,
                                   void* dObar, void* workspace, void* stream) {
    return bwd2_impl(g, q, k, v, out, lse, delta, pk, dO, dQ, uQ, uK, uV, Qbar, Kbar, Vbar, dObar, workspace,
                     stream, g ? sticky_word(g->device, true) : nullptr, part);
}
