// conv_gather_f32.cu -- fp32 convolution with a stride on the tensor cores, straight from the packed operands: no prepared
// filter, no workspace.
//
// A reduction step is one filter tap of one 16-channel block: 128 output pixels x 16 channels, gathered from memory (rows of
// 64 bytes, wherever the stride puts them), and the tap's 16 x KT slice of the filter.  Warps load them into registers,
// split every value into two tf32 words there and write the words in the layouts the MMAs read: pixels in rows of 64 bytes
// with the 64-byte swizzle, filter as [c/4][hi k | lo k][4 c].  The two words hold all of a value but,
// at most, its last bit; sums are x_hi * [W_hi | W_lo] + x_lo * W_hi with the cross terms in columns of their own and the
// hi*hi terms in up to six accumulators in turn, because the tensor core truncates when it adds.  Against fp64 the largest error is a half to a third of the FFMA kernel's (3.1e-7 to 4.7e-7 of
// the largest output against 5.2e-7 to 1.5e-6).
//
// What bounds it: no unit (32 -> 64 channels 3x3 at 16x16, 1024 images: L1 and shared memory 66 % of their peak, issue 46 %, the
// unit that feeds the tensor pipe 34 %) but the chain of a step, loads above all.  A step of 64 output channels writes 24 KB of
// words and the MMAs read some 36 KB: 570 to 590 cycles, of which the MMAs alone would need 250.  Copies by cp.async to shared memory with the split there took 760, one
// step at a time in all pixel warps 1200, eight pairs of pixel warps (64 registers a thread) 660.  With 16 input channels it
// is the latency of the loads: 680 cycles, whatever the number of output channels.
// Stride 2, us, FFMA kernel -> this one: 96 -> 192 channels 3x3 at 57x57, 32 images 346 -> 95; 32 -> 64 3x3 at 16x16, 1024
// images 152 -> 35; 16 -> 32 3x3 at 32x32, 1024 images 81 -> 56; 32 -> 64 1x1 at 16x16, 1024 images 31 -> 15; 256 -> 512 3x3 at
// 14x14, 8 images 155 -> 49.
// Tiles are 128 pixels of the whole batch, images run into one another; CTAs are persistent.
#include "tc_common.cuh"

namespace
{
using namespace sb;

constexpr int SLOTS = 8, GROUPS = 4; // operand slots; steps that are prepared at once
constexpr int EPI_WARPS = 8, FIRST_EPI_WARP = 4; // warps 0 and 1: MMAs; 2, 3 and 20..25: filter
constexpr int FIRST_PX_WARP = 12, FIRST_W_WARP = 20, W_WARPS = 8, MMA_WARPS = 2;
constexpr int PX = 8, UNITS = 8; // pixels and filter units of a thread
constexpr int THREADS = 26 * 32; // a slot has the same warps for its pixels, its filter and its MMAs every time: they wait for its next phase
constexpr uint32_t A_PART = 128 * 64, A_BYTES = 2 * A_PART;

struct GArgs
{
    int N, C, K, H, W, Ho, Wo, Fh, Fw, sw, sh, pad_t, pad_l, cbs, taps, steps;
    int px, tiles, KT, k_tiles, total;
    int per_sum, groups, d_cols, d_bufs; // groups: accumulators of an MMA warp
    unsigned slot_bytes, w_at, w_pitch, smem;
    int w_resident;
    float ns;
    int has_bias, accumulate;
    FastDiv by_tiles, by_HoWo, by_Wo, by_taps, by_Fw;
};

// A value as two tf32 words: hi rounded to nearest (half away from zero), lo what is left of it, of which the tensor core
// ignores at most the last bit.  In integer arithmetic: conversions run at a quarter of its rate or less.
__device__ __forceinline__ void split1(float v, float &hi, float &lo)
{
    hi = __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u);
    lo = v - hi; // NaN where v is not finite or rounds to infinity, whatever hi became
}
// Stores the hi words of four values, returns their lo words.
__device__ __forceinline__ float4 split(float4 v, float4 *hi)
{
    float4 h, l;
    split1(v.x, h.x, l.x); split1(v.y, h.y, l.y); split1(v.z, h.z, l.z); split1(v.w, h.w, l.w);
    *hi = h;
    return l;
}

// Bit i: x + i lies in [0, n).
__device__ __forceinline__ uint32_t in_range(int x, int n)
{
    const int lo = min(max(-x, 0), 16), hi = min(max(n - x, 0), 16);
    return hi > lo ? (1u << hi) - (1u << lo) : 0u;
}

__device__ __noinline__ float plain_sum(const GArgs &a, const float *in, const float *filt, int n, int p, int k)
{
    const int oh = p / a.Wo, ow = p - oh * a.Wo;
    float sum = 0.f;
    for (int s = 0; s < a.steps; ++s)
    {
        const int cb = s / a.taps, tap = s - cb * a.taps, r = oh * a.sh - a.pad_t + tap / a.Fw, c = ow * a.sw - a.pad_l + tap % a.Fw;
        if ((uint32_t)r >= (uint32_t)a.H || (uint32_t)c >= (uint32_t)a.W)
            continue;
        const float *x = in + ((((long long)n * a.cbs + cb) * a.H + r) * a.W + c) * CB;
        const float *w = filt + (((long long)(k / CB) * a.steps + s) * CB) * CB + k % CB;
        for (int i = 0; i < CB; ++i)
            sum = fmaf(x[i], w[i * CB], sum);
    }
    return sum;
}

__global__ void __launch_bounds__(THREADS, 1)
conv_gather_f32_kernel(const GArgs a, const float *__restrict__ in, const float *__restrict__ filt, const float *__restrict__ bias,
                       float *__restrict__ out, int *status)
{
    extern __shared__ __align__(1024) uint8_t smem[]; // [slot][pixels hi | pixels lo | filter]
    __shared__ __align__(8) uint64_t full[SLOTS], empty[SLOTS], d_full[2], d_empty[2], w_all; // w_all: a resident filter's every step is there
    __shared__ uint32_t tmem_base_s;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    uint32_t tmem_cols = 32;
    while ((int)tmem_cols < a.d_bufs * a.d_cols)
        tmem_cols <<= 1;
    if (warp == 0)
    {
        if (lane == 0)
        {
            for (int i = 0; i < SLOTS; ++i) { mbar_init(&full[i], 3); mbar_init(&empty[i], 1); }
            for (int i = 0; i < 2; ++i) { mbar_init(&d_full[i], MMA_WARPS); mbar_init(&d_empty[i], EPI_WARPS); }
            mbar_init(&w_all, (uint32_t)a.steps * 32);
            fence_barrier_init();
        }
        __syncwarp();
        tmem_alloc(&tmem_base_s, tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_base_s;
    const int first = blockIdx.x, stride = gridDim.x;

    if (warp < MMA_WARPS)
    {
        // ---------------- MMAs (the whole warp together, one elected lane issues) ----------------
        // Two warps, one for the even slots and one for the odd ones, each with accumulators of its own: waiting for a step and
        // issuing its four to six MMAs takes one warp some 700 cycles, the tensor core under 300.
        bool ok = true;
        int slot = warp, buf = 0, used = 0, s0 = warp;
        uint32_t phase = 0, d_phase = 1;
        const uint64_t x_desc = make_smem_desc(smem_u32(smem), 16, 512, 4);
        const uint32_t w_addr = smem_u32(smem) + a.w_at;
        for (int t = first; t < a.total && ok; t += stride)
        {
            const int kt = a.by_tiles.div(t), kv = min(a.KT, a.K - kt * a.KT);
            const uint32_t idesc = make_idesc(1, 2, 2, 0, 0, 128, (uint32_t)kv), wide = make_idesc(1, 2, 2, 0, 0, 128, 2u * kv);
            const uint64_t w_desc = make_smem_desc(w_addr, (uint32_t)kv * 32, 128, 0);
            // columns of a warp: first hi*hi accumulator, cross terms, further hi*hi accumulators
            const uint32_t d0 = tmem + (uint32_t)(buf * a.d_cols + warp * a.groups * kv), dx = d0 + (uint32_t)kv;
            if (used >= a.d_bufs)
                ok = __all_sync(0xffffffffu, mbar_wait(&d_empty[buf], d_phase, status, 50));
            // A resident filter's step comes with the pixels of its first use.  With an odd number of steps the warps trade steps from
            // one tile to the next, and what the other one has waited for says nothing here.
            if (a.w_resident && used == 1)
                ok = __all_sync(0xffffffffu, ok && mbar_wait(&w_all, 0, status, 55));
            uint32_t dh = d0;
            int in_sum = 0, sum = 0, s = s0;
            for (; s < a.steps && ok; s += MMA_WARPS)
            {
                ok = __all_sync(0xffffffffu, mbar_wait(&full[slot], phase, status, 51));
                if (!ok)
                    break;
                tc_fence_after_sync();
                if (elect_one())
                {
                    const uint64_t off = (uint64_t)((uint32_t)slot * (a.slot_bytes >> 4));
                    const uint64_t xh = x_desc + off, xl = xh + (A_PART >> 4);
                    const uint64_t wh = w_desc + (uint64_t)((uint32_t)(a.w_resident ? s : slot) * (a.w_pitch >> 4)), wl = wh + (uint64_t)kv;
#pragma unroll
                    for (int h = 0; h < 2; ++h) // 8 channels each
                    {
                        const uint64_t xo = (uint64_t)h * 2, wo = (uint64_t)h * kv * 4;
                        const uint32_t on = (in_sum || h) ? 1u : 0u;
                        if (!sum)
                            tc_mma_tf32(d0, xh + xo, wh + wo, wide, on); // [hi*hi | x_hi * W_lo]
                        else
                        {
                            tc_mma_tf32(dh, xh + xo, wh + wo, idesc, on);
                            tc_mma_tf32(dx, xh + xo, wl + wo, idesc, 1u);
                        }
                        tc_mma_tf32(dx, xl + xo, wh + wo, idesc, 1u);
                    }
                    tc_commit(&empty[slot]);
                }
                __syncwarp();
                slot += MMA_WARPS;
                if (slot >= SLOTS) { slot -= SLOTS; phase ^= 1; }
                if (++in_sum == a.per_sum)
                {
                    in_sum = 0; ++sum;
                    dh = d0 + (uint32_t)((sum + 1) * kv);
                }
            }
            if (ok && elect_one())
                tc_commit(&d_full[buf]);
            __syncwarp();
            s0 = s - a.steps;
            ++used;
            if (++buf == a.d_bufs) { buf = 0; d_phase ^= 1; }
        }
    }
    else if (warp >= FIRST_PX_WARP && warp < FIRST_W_WARP)
    {
        // ---------------- pixels ----------------
        // Warps in pairs, each pair a step of its own, four steps at once: a step is a chain of latencies.  A thread has a
        // quarter (4 channels) of eight pixels, 16 rows apart; its loads for the pair's next step are on their way while the
        // other pairs work.
        const int group = (warp - FIRST_PX_WARP) >> 1, g = tid & 63, q = g & 3, m0 = g >> 2;
        const uint32_t at = (uint32_t)m0 * 64 + ((q ^ ((m0 >> 1) & 3)) << 4); // rows 16 apart have the same swizzle
        const int plane = a.H * a.W * CB;
        const float *base = in;
        int rel[PX];       // element offset of the pixel's tap (0, 0) from base
        uint32_t inside[PX]; // bit kh: the tap's row is in the image; bit 16 + kw: its column
        int t = first, s = group - GROUPS, i = s, slot = s + SLOTS;
        uint32_t phase = 0;
        bool ok = true, fresh = true;
        const int count = ((a.total - first + stride - 1) / stride) * a.steps; // steps of this CTA
        float4 v[PX];
        auto load = [&]() { // the pair's next step
            i += GROUPS; s += GROUPS;
            if (i < count)
            {
                while (s >= a.steps) { s -= a.steps; t += stride; fresh = true; }
                if (fresh)
                {
                    fresh = false;
                    const int pt = t - a.by_tiles.div(t) * a.tiles, n0 = a.by_HoWo.div(pt * 128);
                    base = in + (long long)n0 * a.cbs * plane + q * 4;
#pragma unroll
                    for (int j = 0; j < PX; ++j)
                    {
                        const int px = pt * 128 + m0 + 16 * j, pc = min(px, a.px - 1);
                        const int n = a.by_HoWo.div(pc), p = pc - n * a.Ho * a.Wo, oh = a.by_Wo.div(p), ow = p - oh * a.Wo;
                        const int r = oh * a.sh - a.pad_t, c = ow * a.sw - a.pad_l;
                        rel[j] = (n - n0) * a.cbs * plane + (r * a.W + c) * CB;
                        inside[j] = px < a.px ? in_range(r, a.H) | in_range(c, a.W) << 16 : 0u; // past the batch: nothing
                    }
                }
                const int cb = a.by_taps.div(s), tap = s - cb * a.taps, kh = a.by_Fw.div(tap), kw = tap - kh * a.Fw;
                const uint32_t both = 1u << kh | 0x10000u << kw;
                const int shift = cb * plane + (kh * a.W + kw) * CB;
#pragma unroll
                for (int j = 0; j < PX; ++j)
                    v[j] = (inside[j] & both) == both ? __ldg(reinterpret_cast<const float4 *>(base + (rel[j] + shift)))
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        load();
        while (i < count && ok)
        {
            slot += GROUPS;
            if (slot >= SLOTS) { slot -= SLOTS; phase ^= 1; }
            if (i >= SLOTS)
                ok = __all_sync(0xffffffffu, mbar_wait(&empty[slot], phase, status, 52));
            if (!ok)
                break;
            float4 *hi = reinterpret_cast<float4 *>(smem + (size_t)slot * a.slot_bytes + at);
#pragma unroll
            for (int j = 0; j < PX; ++j)
                hi[j * 16 * 4 + A_PART / 16] = split(v[j], hi + j * 16 * 4);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&full[slot]);
            load();
        }
    }
    else if (warp >= FIRST_W_WARP || warp < FIRST_EPI_WARP)
    {
        // ---------------- filter ----------------
        // Each warp a step of its own; where the whole filter has a place in shared memory, once, and then only the signal.  A unit is four channels of one output channel: four reads (lanes take neighbouring
        // output channels of the packed [16 c][16 k] block), one 16-byte write of each word.
        const long long kb_stride = (long long)a.steps * CB * CB;
        const int count = ((a.total - first + stride - 1) / stride) * a.steps;
        int t = first, s = (warp < FIRST_EPI_WARP ? warp - MMA_WARPS : warp - FIRST_W_WARP + FIRST_EPI_WARP - MMA_WARPS) - W_WARPS, i = s, slot = s + SLOTS, kv = 0;
        uint32_t phase = 0;
        bool ok = true;
        float4 v[UNITS];
        auto load = [&]() { // the warp's next step
            i += W_WARPS; s += W_WARPS;
            if (i >= count || (a.w_resident && i >= a.steps))
                return;
            while (s >= a.steps) { s -= a.steps; t += stride; }
            const int kt = a.by_tiles.div(t);
            kv = min(a.KT, a.K - kt * a.KT);
            const float *w = filt + (long long)kt * (a.KT / CB) * kb_stride + (long long)s * CB * CB + (lane & 15) + (lane >> 4) * 64;
#pragma unroll
            for (int j = 0; j < UNITS; ++j) // units lane + 32 j: [16-channel block of k][c/4][16 k]
                if (j * 8 < kv)
                {
                    const float *o = w + (j >> 1) * kb_stride + (j & 1) * 128;
                    v[j] = make_float4(__ldg(o), __ldg(o + 16), __ldg(o + 32), __ldg(o + 48));
                }
        };
        load();
        while (i < count && ok)
        {
            slot += W_WARPS;
            if (slot >= SLOTS) { slot -= SLOTS; phase ^= 1; }
            if (i >= SLOTS)
                ok = __all_sync(0xffffffffu, mbar_wait(&empty[slot], phase, status, 53));
            if (!ok)
                break;
            if (!a.w_resident || i < a.steps)
            {
                uint8_t *wd = smem + a.w_at + (size_t)(a.w_resident ? i : slot) * a.w_pitch +
                              (uint32_t)((lane >> 4) * 2 * kv + (lane & 15)) * 16;
#pragma unroll
                for (int j = 0; j < UNITS; ++j)
                    if (j * 8 < kv)
                    {
                        float4 *o = reinterpret_cast<float4 *>(wd + (uint32_t)((j & 1) * 4 * kv + (j >> 1) * 16) * 16);
                        o[kv] = split(v[j], o);
                    }
                fence_proxy_async();
                if (a.w_resident)
                    mbar_arrive(&w_all);
            }
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&full[slot]);
            load();
        }
    }
    else if (warp >= FIRST_EPI_WARP)
    {
        // ---------------- sums, bias, activation, stores ----------------
        const int quarter = warp & 3, half = (warp - FIRST_EPI_WARP) >> 2, m = quarter * 32 + lane, hw = a.Ho * a.Wo;
        const bool sectors = whole_sectors(out);
        bool ok = true;
        int buf = 0, odd_start = 0;
        uint32_t phase = 0;
        for (int t = first; t < a.total && ok; t += stride)
        {
            // accumulators in use: the warps' steps of this tile, and no accumulator of a warp without any
            const int n0 = (a.steps + 1 - odd_start) / 2, n1 = a.steps - n0;
            const int groups0 = n0 ? (n0 + a.per_sum - 1) / a.per_sum + 1 : 0, groups1 = n1 ? (n1 + a.per_sum - 1) / a.per_sum + 1 : 0;
            odd_start ^= a.steps & 1;
            const int kt = a.by_tiles.div(t), kv = min(a.KT, a.K - kt * a.KT), px = (t - kt * a.tiles) * 128 + m;
            const bool live = px < a.px;
            const int n = live ? a.by_HoWo.div(px) : 0, p = live ? px - n * hw : 0;
            float *o = out + ((long long)n * (a.K / CB) + (long long)kt * (a.KT / CB)) * hw * CB + (long long)p * CB;
            ok = __all_sync(0xffffffffu, mbar_wait(&d_full[buf], phase, status, 54, 1u << 22));
            if (!ok)
                break;
            tc_fence_after_sync();
            const uint32_t d = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * a.d_cols);
            for (int kb = half; kb < kv / CB; kb += 2)
            {
                uint32_t v[16];
                float y[16];
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    y[e] = 0.f;
                for (int i = 0; i < groups0 + groups1; ++i)
                {
                    tmem_ld16(d + (uint32_t)((i < groups0 ? i : a.groups + i - groups0) * kv + kb * CB), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        y[e] += __uint_as_float(v[e]);
                }
                // Outside the finite range the words' sums are not the products' (inf - inf): sum those products themselves.
                bool odd = false;
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    odd = odd || !(fabsf(y[e]) <= 3.402823466e38f);
                if (live && odd)
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        y[e] = plain_sum(a, in, filt, n, p, kt * a.KT + kb * CB + e);
                if (live)
                {
                    float4 *dst = reinterpret_cast<float4 *>(o + (long long)kb * hw * CB);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                    {
                        float4 b = a.has_bias ? __ldg(reinterpret_cast<const float4 *>(bias + kt * a.KT + kb * CB) + j)
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
                        if (a.accumulate)
                        {
                            const float4 r = dst[j];
                            b.x += r.x; b.y += r.y; b.z += r.z; b.w += r.w;
                        }
                        y[4 * j] = apply_act_ns(y[4 * j] + b.x, a.ns); y[4 * j + 1] = apply_act_ns(y[4 * j + 1] + b.y, a.ns);
                        y[4 * j + 2] = apply_act_ns(y[4 * j + 2] + b.z, a.ns); y[4 * j + 3] = apply_act_ns(y[4 * j + 3] + b.w, a.ns);
                    }
                    store8(reinterpret_cast<float *>(dst), y, sectors);
                    store8(reinterpret_cast<float *>(dst + 2), y + 8, sectors);
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&d_empty[buf]);
            if (++buf == a.d_bufs) { buf = 0; phase ^= 1; }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0)
        tmem_dealloc(tmem, tmem_cols);
}

bool plan_gather(const small_b200_layer *L, GArgs &a)
{
    if (L->C <= 0 || L->C % CB || L->K <= 0 || L->K % CB || L->N <= 0 || L->H <= 0 || L->W <= 0 || L->Fh <= 0 || L->Fw <= 0 || L->stride <= 0)
        return false;
    a = GArgs{};
    a.N = L->N; a.C = L->C; a.K = L->K; a.H = L->H; a.W = L->W; a.Fh = L->Fh; a.Fw = L->Fw;
    a.sw = L->stride; a.sh = row_stride(L); a.pad_t = L->pad_t; a.pad_l = L->pad_l;
    a.Ho = out_dim(L->H, L->pad_t, L->pad_b, L->Fh, a.sh);
    a.Wo = out_dim(L->W, L->pad_l, L->pad_r, L->Fw, a.sw);
    const long long px = (long long)a.N * a.Ho * a.Wo;
    if (px <= 0 || px > 0x3fffffffLL || L->Fh > 16 || L->Fw > 16)
        return false; // a pixel's taps are told inside from outside by 16 bits for rows and 16 for columns
    a.cbs = a.C / CB; a.taps = a.Fh * a.Fw;
    if ((127 / ((long long)a.Ho * a.Wo) + 2) * a.C * a.H * a.W > 0x7fffffffLL) // offsets within the images of a tile
        return false;
    if ((long long)a.cbs * a.taps > 192) // three hi*hi accumulators of each MMA warp, at most 32 steps each
        return false;
    a.steps = a.cbs * a.taps;
    a.px = (int)px; a.tiles = (a.px + 127) / 128;
    a.KT = a.K < 64 ? a.K : 64; // a filter step is at most two units for each of the four warps
    a.k_tiles = (a.K + a.KT - 1) / a.KT;
    if ((long long)a.tiles * a.k_tiles > 0x7fffffffLL)
        return false;
    a.total = a.tiles * a.k_tiles;
    const int n0 = (a.steps + 1) / 2; // steps of an MMA warp
    a.per_sum = (n0 + 2) / 3 < 8 ? 8 : (n0 + 2) / 3;
    a.groups = (n0 + a.per_sum - 1) / a.per_sum + 1;
    a.d_cols = MMA_WARPS * a.groups * a.KT;
    a.d_bufs = 2 * a.d_cols <= 512 ? 2 : 1;
    // The filter's words: once per CTA where all of them fit beside the slots, else a step's words in every slot.
    const unsigned w = (unsigned)a.KT * 128;
    a.w_resident = a.k_tiles == 1 && SLOTS * A_BYTES + a.steps * w <= 220u * 1024;
    a.slot_bytes = a.w_resident ? A_BYTES : A_BYTES + w;
    a.w_at = a.w_resident ? SLOTS * A_BYTES : A_BYTES;
    a.w_pitch = a.w_resident ? w : a.slot_bytes;
    a.smem = SLOTS * a.slot_bytes + (a.w_resident ? a.steps * w : 0u);
    a.by_tiles.set(a.tiles); a.by_HoWo.set(a.Ho * a.Wo); a.by_Wo.set(a.Wo); a.by_taps.set(a.taps); a.by_Fw.set(a.Fw);
    return true;
}
} // namespace

namespace sb
{
// Whether the kernel covers a layer and is the better one for it.  Not where 16 input channels leave it a few steps in a few
// CTAs: there it needs some 10 us and the FFMA kernel, whose tiles are smaller, 9 (16 -> 32 channels 3x3, 24 tiles); even at
// about one tile for each SM, ahead from then on and everywhere with more channels.
bool conv_gather_preferred(const small_b200_layer *L)
{
    GArgs a;
    return plan_gather(L, a) && a.px >= 128 && (a.cbs > 1 || a.total >= num_sms());
}

int conv_gather_f32(const small_b200_layer *L, const float *in, const float *filt, const float *bias, float *out, cudaStream_t st)
{
    GArgs a;
    if (!plan_gather(L, a))
        return fail(SMALL_B200_INVALID_ARGUMENT, "Conv2D<float> ERROR: shape not covered by the gathering kernel.");
    a.ns = L->act == SMALL_B200_ACT_RELU ? 0.f : L->act == SMALL_B200_ACT_LEAKY ? L->slope : 1.f;
    a.has_bias = bias != nullptr; a.accumulate = L->accumulate;
    static PerDeviceOnce configured;
    int dev;
    if (configured.needed(&dev))
    {
        SB_CUDA(cudaFuncSetAttribute(conv_gather_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
        configured.mark(dev);
    }
    int *status = device_status_ptr();
    if (!status)
        return fail(SMALL_B200_CUDA_ERROR, "device status word not available");
    const int grid = a.total < num_sms() ? a.total : num_sms();
    conv_gather_f32_kernel<<<(unsigned)grid, THREADS, a.smem, st>>>(a, in, filt, bias, out, status);
    return launched("conv_gather_f32_kernel");
}
} // namespace sb
