// Forward for a few query rows per head (text generation: one new token, or a handful, against a cache).
//
// What bounds it: reading K and V once (134 MB for 128 heads of 4096 keys at head dim 64, 20 us at 6.65 TB/s).
// The sweep kernel owns 128 query rows per CTA, so with one row it spends its exponentials and products on 127
// rows of padding (2 us per 32 KB of K and V, 1.9 TB/s in all), and it has no more CTAs than heads.  Here the
// arithmetic (two multiply-adds per element and query) stays on the ordinary pipes, in fp32 throughout, and the
// keys of a head are divided between CTAs.  Measured on that case: 31.9 us, against 71.0 us through the sweep kernel.
//
// A key row is read by DPAD / 8 lanes, 16 bytes each, so one warp-wide load takes 32 / (DPAD / 8) keys.  A warp
// asks for U such loads of K and of V before it uses the first (U * 1 KB in flight per warp, 16 warps per SM).
// Every lane group (the lanes that share a key) has a softmax of its own over the keys it reads; groups, warps and
// CTAs are merged in a fixed order, so the result does not depend on the order in which they finish.
#pragma once

#include "sweep.cuh"

namespace bob {

constexpr int kDecodeRows = 4;          // most query rows per head (which calls come here: takes_decode)
constexpr int kDecodeThreads = 256;
constexpr int kDecodeMaxSplits = 64;

struct DecodeParams {
    const uint16_t* q; long long q_sb, q_sh, q_sn;      // element strides: batch, head, row
    const uint16_t* k; long long k_sb, k_sh, k_sn;
    const uint16_t* v; long long v_sb, v_sh, v_sn;
    int Hq, G, Nq, D;
    int causal, window, delta_off;
    int k_lo, k_hi;                     // keys that any query row attends to
    int splits, split_keys;             // CTAs per head, keys of each
    float scale;
    uint16_t* out;                      // [B, Hq, Nq, D]
    float* lse;                         // [B, Hq, Nq]
    // splits > 1: per head and split, Nq rows of (reference, sum) and of D unnormalised columns
    float* part_ml;
    float* part_acc;
    int* arrived;                       // per head: splits that have parked their part (zeroed by the host)
    int* status;
};

// Keys that a CTA takes in one round of its warps.
__host__ __device__ constexpr int decode_unroll(int nq) { return nq == 1 ? 8 : 4; }
__host__ __device__ constexpr int decode_round(int dpad, int nq) { return (kDecodeThreads / 32) * (32 / (dpad / 8)) * decode_unroll(nq); }

template <bool BF16>
__device__ __forceinline__ void unpack8(const uint4 a, float* v) {
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        if constexpr (BF16) {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        } else {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
            v[2 * i] = f.x; v[2 * i + 1] = f.y;
        }
    }
}

__device__ __forceinline__ uint4 load_stream16(const void* p) {          // read once: not kept in L1
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}

template <int DPAD, int NQ, bool BF16>
__global__ void __launch_bounds__(kDecodeThreads, 2) decode_kernel(const __grid_constant__ DecodeParams p) {
    constexpr int LPK = DPAD / 8, KPI = 32 / LPK, U = decode_unroll(NQ), WARPS = kDecodeThreads / 32;
    constexpr float kNone = -1e30f;                      // reference of a softmax without keys
    constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
    __shared__ float sm_ml[2][WARPS][NQ];
    __shared__ __align__(16) float sm_acc[WARPS][NQ][DPAD];
    __shared__ float sm_w[NQ][kDecodeMaxSplits];
    __shared__ float sm_tot[2][NQ];
    __shared__ int sm_last;

    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int chunk = lane % LPK, grp = lane / LPK;
    const int unit = blockIdx.x / p.splits, split = blockIdx.x % p.splits;     // unit = batch * Hq + head
    const int batch = unit / p.Hq, head = unit % p.Hq, kv_head = head / p.G;
    const bool col_ok = chunk * 8 < p.D;
    const float c_exp = p.scale * kLog2e;
    if (blockIdx.x == 0 && tid == 0) *p.status = 0;      // (nothing here waits on anything that could fail)

    float q[NQ][8];
    int lo[NQ], hi[NQ];                                  // keys row i attends to
    #pragma unroll
    for (int i = 0; i < NQ; ++i) {
        uint4 w = make_uint4(0, 0, 0, 0);
        lo[i] = p.k_lo;
        hi[i] = i < p.Nq ? p.k_hi : 0;
        if (i < p.Nq) {
            if (col_ok) w = load_stream16(p.q + batch * p.q_sb + head * p.q_sh + i * p.q_sn + chunk * 8);
            if (p.causal) {
                hi[i] = min(hi[i], i + p.delta_off + 1);
                if (p.window > 0) lo[i] = max(lo[i], i + p.delta_off - p.window + 1);
            }
        }
        unpack8<BF16>(w, q[i]);
    }
    const uint16_t* kp = p.k + batch * p.k_sb + kv_head * p.k_sh + chunk * 8;
    const uint16_t* vp = p.v + batch * p.v_sb + kv_head * p.v_sh + chunk * 8;
    const int first = p.k_lo + split * p.split_keys, last = min(first + p.split_keys, p.k_hi);

    float m[NQ], l[NQ], acc[NQ][8];
    #pragma unroll
    for (int i = 0; i < NQ; ++i) {
        m[i] = kNone; l[i] = 0.f;
        #pragma unroll
        for (int c = 0; c < 8; ++c) acc[i][c] = 0.f;
    }
    for (int base = first + warp * (KPI * U); base < last; base += WARPS * KPI * U) {
        uint4 kw[U], vw[U];
        #pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = base + u * KPI + grp;
            kw[u] = make_uint4(0, 0, 0, 0);
            if (j < last && col_ok) kw[u] = load_stream16(kp + j * p.k_sn);
        }
        #pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = base + u * KPI + grp;
            vw[u] = make_uint4(0, 0, 0, 0);
            if (j < last && col_ok) vw[u] = load_stream16(vp + j * p.v_sn);
        }
        float s[U][NQ];
        #pragma unroll
        for (int u = 0; u < U; ++u) {
            float f[8];
            unpack8<BF16>(kw[u], f);
            #pragma unroll
            for (int i = 0; i < NQ; ++i) {
                float a = q[i][0] * f[0], b = q[i][1] * f[1];
                #pragma unroll
                for (int c = 2; c < 8; c += 2) { a = fmaf(q[i][c], f[c], a); b = fmaf(q[i][c + 1], f[c + 1], b); }
                s[u][i] = a + b;
            }
        }
        #pragma unroll
        for (int o = LPK / 2; o > 0; o >>= 1) {
            #pragma unroll
            for (int u = 0; u < U; ++u) {
                #pragma unroll
                for (int i = 0; i < NQ; ++i) s[u][i] += __shfl_xor_sync(0xffffffffu, s[u][i], o);
            }
        }
        #pragma unroll
        for (int i = 0; i < NQ; ++i) {
            float mt = kNone;                            // in log2 units; the scale is positive
            #pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = base + u * KPI + grp;
                const bool ok = j >= lo[i] && j < min(hi[i], last);
                s[u][i] = ok ? s[u][i] * c_exp : -INFINITY;
                mt = fmaxf(mt, s[u][i]);
            }
            if (mt > m[i]) {
                const float f = fast_exp2(m[i] - mt);
                m[i] = mt;
                l[i] *= f;
                #pragma unroll
                for (int c = 0; c < 8; ++c) acc[i][c] *= f;
            }
            #pragma unroll
            for (int u = 0; u < U; ++u) {
                s[u][i] = fast_exp2(s[u][i] - m[i]);         // probability relative to the reference; 0 where masked
                l[i] += s[u][i];
            }
        }
        #pragma unroll
        for (int u = 0; u < U; ++u) {
            float f[8];
            unpack8<BF16>(vw[u], f);
            #pragma unroll
            for (int i = 0; i < NQ; ++i) {
                #pragma unroll
                for (int c = 0; c < 8; ++c) acc[i][c] = fmaf(s[u][i], f[c], acc[i][c]);
            }
        }
    }

    // ---- lane groups of a warp, then the warps --------------------------------------------------------
    #pragma unroll
    for (int i = 0; i < NQ; ++i) {
        #pragma unroll
        for (int o = LPK; o < 32; o <<= 1) {
            const float mo = __shfl_xor_sync(0xffffffffu, m[i], o), lo_ = __shfl_xor_sync(0xffffffffu, l[i], o);
            const float mn = fmaxf(m[i], mo), fa = fast_exp2(m[i] - mn), fb = fast_exp2(mo - mn);
            l[i] = l[i] * fa + lo_ * fb;
            #pragma unroll
            for (int c = 0; c < 8; ++c) acc[i][c] = acc[i][c] * fa + __shfl_xor_sync(0xffffffffu, acc[i][c], o) * fb;
            m[i] = mn;
        }
        if (grp == 0) {
            #pragma unroll
            for (int c = 0; c < 8; c += 4)
                *reinterpret_cast<float4*>(&sm_acc[warp][i][chunk * 8 + c]) = make_float4(acc[i][c], acc[i][c + 1], acc[i][c + 2], acc[i][c + 3]);
            if (chunk == 0) { sm_ml[0][warp][i] = m[i]; sm_ml[1][warp][i] = l[i]; }
        }
    }
    __syncthreads();
    auto finish = [&](int i, int col, float value, float ref, float sum) {       // row i, column col of the result
        const long long row = (long long)unit * p.Nq + i;
        // no key: zero.  An infinite score makes the sum NaN, and the row with it.
        const float r = sum > 0.f ? value / sum : (ref == INFINITY ? sum : 0.f);
        p.out[row * p.D + col] = static_cast<uint16_t>(pack2<BF16>(r, 0.f));
        if (col == 0) p.lse[row] = sum > 0.f ? (ref + log2f(sum)) * kLn2 : -INFINITY;
    };
    for (int x = tid; x < NQ * DPAD; x += kDecodeThreads) {
        const int i = x / DPAD, col = x % DPAD;
        if (i >= p.Nq || col >= p.D) continue;
        float ref = kNone, sum = 0.f, value = 0.f;
        #pragma unroll
        for (int w = 0; w < WARPS; ++w) ref = fmaxf(ref, sm_ml[0][w][i]);
        #pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float f = fast_exp2(sm_ml[0][w][i] - ref);
            sum = fmaf(f, sm_ml[1][w][i], sum);
            value = fmaf(f, sm_acc[w][i][col], value);
        }
        if (p.splits == 1) {
            finish(i, col, value, ref, sum);
        } else {
            const long long slot = ((long long)unit * p.splits + split) * p.Nq + i;
            p.part_acc[slot * p.D + col] = value;
            if (col == 0) *reinterpret_cast<float2*>(p.part_ml + 2 * slot) = make_float2(ref, sum);
        }
    }
    if (p.splits == 1) return;

    // ---- the CTA that parks a head's last part adds all of them, in the order of the splits ------------
    __threadfence();
    __syncthreads();
    if (tid == 0) sm_last = atomicAdd(p.arrived + unit, 1) == p.splits - 1;
    __syncthreads();
    if (!sm_last) return;
    __threadfence();
    const long long slot0 = (long long)unit * p.splits * p.Nq;
    for (int i = warp; i < p.Nq; i += WARPS) {           // one warp per row: the splits' weights, their sum
        static_assert(kDecodeMaxSplits == 64, "two splits per lane");
        float2 a = make_float2(kNone, 0.f), b = a;
        if (lane < p.splits) a = __ldcg(reinterpret_cast<const float2*>(p.part_ml + 2 * (slot0 + lane * p.Nq + i)));
        if (lane + 32 < p.splits) b = __ldcg(reinterpret_cast<const float2*>(p.part_ml + 2 * (slot0 + (lane + 32) * p.Nq + i)));
        float ref = fmaxf(a.x, b.x);
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) ref = fmaxf(ref, __shfl_xor_sync(0xffffffffu, ref, o));
        const float wa = fast_exp2(a.x - ref), wb = fast_exp2(b.x - ref);
        sm_w[i][lane] = wa;
        sm_w[i][lane + 32] = wb;
        float sum = wa * a.y + wb * b.y;
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) { sm_tot[0][i] = ref; sm_tot[1][i] = sum; }
    }
    __syncthreads();
    // PARTS threads share a column, each with every PARTS-th split
    constexpr int ITEMS = NQ * DPAD, PARTS = ITEMS >= kDecodeThreads ? 1 : kDecodeThreads / ITEMS;
    float* red = &sm_acc[0][0][0];                       // (read for the last time two barriers ago)
    for (int x = tid; x < ITEMS * PARTS; x += kDecodeThreads) {
        const int part = x / ITEMS, i = (x % ITEMS) / DPAD, col = x % DPAD;
        float value = 0.f;
        if (i < p.Nq && col < p.D) {
            #pragma unroll 8
            for (int s = part; s < p.splits; s += PARTS)
                value = fmaf(sm_w[i][s], __ldcg(p.part_acc + (slot0 + (long long)s * p.Nq + i) * p.D + col), value);
            if (PARTS == 1) finish(i, col, value, sm_tot[0][i], sm_tot[1][i]);
        }
        if (PARTS > 1) red[x] = value;
    }
    if (PARTS > 1) {
        __syncthreads();
        if (tid < ITEMS) {
            const int i = tid / DPAD, col = tid % DPAD;
            float value = 0.f;
            #pragma unroll
            for (int part = 0; part < PARTS; ++part) value += red[part * ITEMS + tid];
            if (i < p.Nq && col < p.D) finish(i, col, value, sm_tot[0][i], sm_tot[1][i]);
        }
    }
}

}  // namespace bob
