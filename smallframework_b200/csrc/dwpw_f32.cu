// dwpw_f32.cu -- fp32 depthwise 3x3 convolution and the 1x1 convolution behind it (a depthwise-separable block,
// include/small/models/MobileNetTiny.hpp) as one kernel: the activation between the two never leaves the SM.
//
// A block moves its input and its output once; as two layers the activation between them is
// written and read again, and the 1x1 layer alone ran at 2 to 3 TB/s because its patches went through shared memory three
// times (bulk copy, operand split, tensor core).  Here what the depthwise warps write to shared memory IS the tensor
// core's operand.
// What bounds it: no unit (16 channels at 48x48, 256 images: issue 37 % of its peak, loads and stores of shared memory 23 %,
// tensor pipe 3 %, DRAM 10 %) but the depthwise warps' chain of reads, sums and stores, 3.6 times the block's bytes at copy
// bandwidth there.  Blocks of so few channels run on the FMA pipe (dwpw_direct_f32.cu, where the rule stands).
//
// A tile is NI images x TH x TW <= 128 output pixels times KT <= 128 output channels.  Roles of a persistent CTA:
//   * one thread keeps patches of 16 channels on their way, one TMA box each (rows of the image are contiguous in it, zeros
//     outside): 70 to 130 KB in flight.  (A first version loaded the inputs from the depthwise warps, three dependent round
//     trips to memory per strip: 385 us for the block of 16 channels at 48x48 on 2048 images.)
//   * eight warps compute the depthwise layer, each one 16-channel block of a tile at a time and on its own (they meet
//     nowhere): a thread owns four channels of a block of R x 3 outputs, reads every input of that block once (2.5 reads
//     per output with R = 4, 4.5 with one row) and the filter's nine 16-byte words again for every output row (up to three per
//     output more: 68 of the 96 registers hold sums and inputs), and writes every value as it is (hi: the tensor core ignores the 13 low mantissa bits of a tf32 operand) and as v - trunc(v)
//     (lo) into rows of 64 bytes in the 64-byte swizzle.  Neighbouring blocks are three pixels apart, an odd number, so the
//     reads of eight lanes fall into different banks (stride 1);
//   * one warp issues the MMAs, kind::tf32, M = 128 pixels: x_hi * [W_hi | W_lo] and x_lo * W_hi.  The cross terms have
//     accumulator columns of their own, and the hi*hi sums change columns after every eight channel blocks: the tensor core
//     truncates when it adds, and this way no accumulator takes more than sixteen full-size terms;
//   * eight warps add up the columns, apply bias and activation and store 64-byte runs.
// tf32 words rather than the block-scaled half-precision ones of conv_f16x3.cu: they need no scale, so a thread can write
// its operands without knowing its neighbours' magnitudes, and the tensor pipe has time to spare (128 -> 128 channels:
// 3072 cycles per tile against 2980 for the tile's bytes).
// An infinity has no second word (inf - inf): outputs whose products sum to an infinity are NaN here.  Making such sums
// again from the products, as conv_gather_f32.cu and conv_f16x3.cu do, was taken back: the code for it, never run, in the
// epilogue, behind a call or behind the last barrier, costs every block 3.5 to 6 % (MobileNet at 2048 images 1092 -> 1130
// to 1160 us).
#include "tc_common.cuh"

namespace sb
{
bool conv_small_preferred(const small_b200_layer *L); // conv_small_f32.cu
double conv_small_us(const small_b200_layer *L);
// dwpw_direct_f32.cu: blocks of few channels on the FMA pipe; -1 where it leaves them to this kernel
int dwpw_direct_f32(const small_b200_layer *D, const small_b200_layer *L, const float *in, const float *dwf, const float *b1, const float *pwf,
                    const float *b2, float *out, cudaStream_t st);
} // namespace sb

namespace
{
using namespace sb;

constexpr int DW_WARPS = 8, P = 3; // outputs of a row that a depthwise thread owns
constexpr int EPI_WARPS = 8, FIRST_EPI_WARP = 4; // warp 0: filter copies, 1: MMAs, 2: patches, 3: slots
constexpr int FIRST_DW_WARP = FIRST_EPI_WARP + EPI_WARPS;
constexpr int THREADS = (FIRST_DW_WARP + DW_WARPS) * 32;
constexpr int A_SLOTS_MAX = 4, P_SLOTS_MAX = DW_WARPS, W_STAGES_MAX = 16;
constexpr uint32_t A_PART = 128 * 64;   // hi (or lo) operand of one channel block: 128 pixels x 16 channels
constexpr uint32_t A_SLOT = 2 * A_PART;
constexpr int CBS_PER_SUM = 8;          // channel blocks per hi*hi accumulator

struct DpArgs
{
    int N, C, K, H, W, Ho, Wo, pad_t, pad_l, cbs;
    int NI, TH, TW, SPR, RB;   // tile: images, rows, columns; blocks of R x P outputs per row and per column of an image
    int PW, PR;                // patch: columns (odd), rows per image
    int tiles_x, tiles_y, px_tiles, KT, k_tiles, total;
    int a_slots, p_slots, w_stages, w_resident, sums, d_bufs, d_cols;
    unsigned p_bytes, p_slot;  // a patch, and its slot (rounded up)
    unsigned p_off, w_off, dwf_off; // shared memory: operand slots, patches, filter stages, depthwise filter + bias
    float ns1, ns2;            // activations as act_neg_scale()
    int has_b1, has_b2;
    FastDiv by_px_tiles, by_tiles_x, by_tiles_y, by_SPR, by_RB, by_TH, by_TW;
};

struct DpTile
{
    int kt, n0, r0, c0;
};
__device__ __forceinline__ DpTile dp_tile(const DpArgs &a, int t)
{
    DpTile T;
    T.kt = a.by_px_tiles.div(t);
    const int p = t - T.kt * a.px_tiles, row = a.by_tiles_x.div(p), n = a.by_tiles_y.div(row);
    T.c0 = (p - row * a.tiles_x) * a.TW;
    T.r0 = (row - n * a.tiles_y) * a.TH;
    T.n0 = n * a.NI;
    return T;
}

// packed 1x1 filter [K/16][C/16][16 c][16 k] -> [K tile][C/16][c/4][hi kv | lo kv][4 c]
__global__ void __launch_bounds__(256) prepare_pw_kernel(int n, int cbs, int K, int KT, const float *__restrict__ w, float *__restrict__ o)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n)
        return;
    const int k16 = i & 15, c = (i >> 4) & 15, cb = (i >> 8) % cbs, k = (i >> 8) / cbs * 16 + k16;
    const int tile = k / KT, kv = min(KT, K - tile * KT);
    const long long at = (long long)tile * KT * cbs * 32 + ((long long)cb * 4 + (c >> 2)) * 2 * kv * 4 + (k - tile * KT) * 4 + (c & 3);
    const float v = w[i];
    o[at] = v;
    o[at + (long long)kv * 4] = v - __uint_as_float(__float_as_uint(v) & 0xffffe000u);
}

__device__ __forceinline__ float4 lo_part(const float4 v)
{
    return make_float4(v.x - __uint_as_float(__float_as_uint(v.x) & 0xffffe000u), v.y - __uint_as_float(__float_as_uint(v.y) & 0xffffe000u),
                       v.z - __uint_as_float(__float_as_uint(v.z) & 0xffffe000u), v.w - __uint_as_float(__float_as_uint(v.w) & 0xffffe000u));
}
__device__ __forceinline__ void fma4(float4 &a, const float4 x, const float4 f)
{
    a.x = fmaf(x.x, f.x, a.x); a.y = fmaf(x.y, f.y, a.y); a.z = fmaf(x.z, f.z, a.z); a.w = fmaf(x.w, f.w, a.w);
}

// Until step `before` has been counted; bounded like mbar_wait().
__device__ __forceinline__ bool wait_step(const int *done, int before, int *status, int code)
{
    for (uint32_t i = 0; i < (1u << 22); ++i)
    {
        if (*reinterpret_cast<const volatile int *>(done) > before)
            return true;
        __nanosleep(20);
        if ((i & 1023u) == 1023u && *reinterpret_cast<volatile int *>(status) != 0)
            return false;
    }
    atomicCAS(status, 0, code);
    return false;
}

template <int S, int R>
__global__ void __launch_bounds__(THREADS, 1)
dwpw_f32_kernel(const __grid_constant__ CUtensorMap map_x, const DpArgs a, const float *__restrict__ dwf, const float *__restrict__ b1,
                const float *__restrict__ pwf, const float *__restrict__ b2, float *__restrict__ out, int *status)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t a_full[A_SLOTS_MAX], a_empty[A_SLOTS_MAX], p_full[P_SLOTS_MAX], p_empty[P_SLOTS_MAX], w_full[W_STAGES_MAX], w_empty[W_STAGES_MAX];
    __shared__ __align__(8) uint64_t d_full[2], d_empty[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ int a_done; // steps whose MMAs have read their operands
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    uint32_t tmem_cols = 32;
    while ((int)tmem_cols < a.d_bufs * a.d_cols)
        tmem_cols <<= 1;
    float *s_dwf = reinterpret_cast<float *>(smem + a.dwf_off); // [cb][9][16], then the bias [C]
    for (int i = tid; i < a.C * 9; i += THREADS)
        s_dwf[i] = dwf[i];
    for (int i = tid; i < a.C; i += THREADS)
        s_dwf[a.C * 9 + i] = a.has_b1 ? b1[i] : 0.f;
    if (warp == 0)
    {
        if (lane == 0)
        {
            for (int i = 0; i < A_SLOTS_MAX; ++i) { mbar_init(&a_full[i], 1); mbar_init(&a_empty[i], 1); }
            a_done = 0;
            for (int i = 0; i < P_SLOTS_MAX; ++i) { mbar_init(&p_full[i], 1); mbar_init(&p_empty[i], 1); }
            for (int i = 0; i < W_STAGES_MAX; ++i) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], 1); }
            for (int i = 0; i < 2; ++i) { mbar_init(&d_full[i], 1); mbar_init(&d_empty[i], a.KT == CB ? EPI_WARPS / 2 : EPI_WARPS); }
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
    const int first = blockIdx.x, step = gridDim.x;

    if (warp == 0)
    {
        if (lane == 0)
        {
            // ---------------- filter copies ----------------
            bool ok = true, again = false;
            int st = 0;
            uint32_t freed = 1;
            for (int t = first; t < a.total && ok; t += step)
            {
                if (again && a.w_resident)
                    break;
                const int kt = a.by_px_tiles.div(t), kv = min(a.KT, a.K - kt * a.KT);
                const float *src = pwf + (long long)kt * a.KT * a.cbs * 32;
                for (int cb = 0; cb < a.cbs && ok; ++cb)
                {
                    if (again)
                        ok = mbar_wait(&w_empty[st], freed, status, 40);
                    if (!ok)
                        break;
                    const uint32_t bytes = (uint32_t)kv * 128;
                    mbar_expect_tx(&w_full[st], bytes);
                    tma_load_1d(smem + a.w_off + (size_t)st * a.KT * 128, src + (long long)cb * kv * 32, bytes, &w_full[st]);
                    if (++st == a.w_stages) { st = 0; freed ^= 1; again = true; }
                }
            }
        }
    }
    else if (warp == 1)
    {
        // ---------------- MMAs ----------------
        // The whole warp walks through the loop with uniform values and one elected lane issues: 42 cycles per instruction
        // instead of the 60 of a loop inside one lane's branch (M = 128, N = 16 back to back).
        bool ok = true;
        int slot = 0, st = 0, buf = 0, used = 0;
        uint32_t a_phase = 0, w_phase = 0, d_phase = 1;
        const uint64_t x_desc = make_smem_desc(smem_u32(smem), 16, 512, 4);
        const uint32_t w_addr = smem_u32(smem + a.w_off);
        int kt_at = -1, kv = 0;
        uint32_t idesc = 0, wide = 0;
        uint64_t w_desc = 0;
        for (int t = first; t < a.total && ok; t += step)
        {
            const int kt = a.k_tiles == 1 ? 0 : a.by_px_tiles.div(t);
            if (kt != kt_at)
            {
                kt_at = kt;
                kv = min(a.KT, a.K - kt * a.KT);
                idesc = make_idesc(1, 2, 2, 0, 0, 128, (uint32_t)kv); wide = make_idesc(1, 2, 2, 0, 0, 128, 2u * kv);
                w_desc = make_smem_desc(w_addr, (uint32_t)kv * 32, 128, 0);
            }
            // columns: hi*hi sums of the first eight channel blocks, cross terms, further hi*hi sums
            const uint32_t d0 = tmem + (uint32_t)(buf * a.d_cols), dx = d0 + (uint32_t)a.KT;
            if (used >= a.d_bufs)
                ok = mbar_wait(&d_empty[buf], d_phase, status, 42);
            for (int cb = 0; cb < a.cbs && ok; ++cb)
            {
                if (!a.w_resident || used == 0)
                    ok = mbar_wait(&w_full[st], w_phase, status, 43);
                ok = ok && mbar_wait(&a_full[slot], a_phase, status, 44);
                ok = __all_sync(0xffffffffu, ok); // the warp stays together (elect_one)
                if (!ok)
                    break;
                tc_fence_after_sync();
                if (elect_one())
                {
                    const int sum = cb / CBS_PER_SUM;
                    const uint32_t dh = sum ? d0 + (uint32_t)((sum + 1) * a.KT) : d0;
                    const uint64_t xh = x_desc + (uint64_t)((uint32_t)slot * (A_SLOT >> 4)), xl = xh + (A_PART >> 4);
                    const uint64_t wh = w_desc + (uint64_t)((uint32_t)st * ((uint32_t)a.KT * 8)), wl = wh + (uint64_t)kv;
                    const bool merged = !sum && kv == a.KT;
#pragma unroll
                    for (int h = 0; h < 2; ++h) // 8 channels each
                    {
                        const uint64_t xo = (uint64_t)h * 2, wo = (uint64_t)h * kv * 4;
                        const uint32_t on = (cb % CBS_PER_SUM || h) ? 1u : 0u;
                        if (merged)
                            tc_mma_tf32(d0, xh + xo, wh + wo, wide, on); // [hi*hi | x_hi * W_lo]
                        else
                        {
                            tc_mma_tf32(dh, xh + xo, wh + wo, idesc, on);
                            tc_mma_tf32(dx, xh + xo, wl + wo, idesc, (cb || h) ? 1u : 0u);
                        }
                        tc_mma_tf32(dx, xl + xo, wh + wo, idesc, 1u);
                    }
                    tc_commit(&a_empty[slot]);
                    if (!a.w_resident)
                        tc_commit(&w_empty[st]);
                    if (cb == a.cbs - 1)
                        tc_commit(&d_full[buf]);
                }
                __syncwarp();
                if (++slot == a.a_slots) { slot = 0; a_phase ^= 1; }
                if (++st == a.w_stages) { st = 0; w_phase ^= a.w_resident ? 0u : 1u; }
            }
            ++used;
            if (++buf == a.d_bufs) { buf = 0; d_phase ^= 1; }
        }
    }
    else if (warp == 3)
    {
        if (lane == 0)
        {
            // ---------------- operand slots come back ----------------
            // The MMAs release operand slots in order; the depthwise warps, more of them than slots, would have to tell
            // phases of a slot's barrier apart that lie two or more uses back.  They wait for a step number instead.
            bool ok = true;
            int slot = 0, done = 0;
            uint32_t phase = 0;
            for (int t = first; t < a.total && ok; t += step)
                for (int cb = 0; cb < a.cbs && ok; ++cb)
                {
                    ok = mbar_wait(&a_empty[slot], phase, status, 48, 1u << 22);
                    if (!ok)
                        break;
                    *reinterpret_cast<volatile int *>(&a_done) = ++done;
                    if (++slot == a.a_slots) { slot = 0; phase ^= 1; }
                }
        }
    }
    else if (warp == 2)
    {
        if (lane == 0)
        {
            // ---------------- patches ----------------
            bool ok = true, again = false;
            int slot = 0;
            uint32_t freed = 1;
            for (int t = first; t < a.total && ok; t += step)
            {
                const DpTile T = dp_tile(a, t);
                for (int cb = 0; cb < a.cbs && ok; ++cb)
                {
                    if (again)
                        ok = mbar_wait(&p_empty[slot], freed, status, 46);
                    if (!ok)
                        break;
                    mbar_expect_tx(&p_full[slot], a.p_bytes);
                    tma_load_4d(smem + a.p_off + (size_t)slot * a.p_slot, &map_x, (T.c0 * S - a.pad_l) * 8, T.r0 * S - a.pad_t, cb, T.n0,
                                &p_full[slot]);
                    if (++slot == a.p_slots) { slot = 0; freed ^= 1; again = true; }
                }
            }
        }
    }
    else if (warp >= FIRST_DW_WARP)
    {
        // ---------------- depthwise layer ----------------
        // As many warps work as there are patch slots, each on a slot of its own: a barrier only tells the last of its
        // phases from the one before, so nobody may wait for a patch two fills ahead of the slot's.
        const int workers = a.p_slots;
        const int q = lane & 3, me = warp - FIRST_DW_WARP, units = a.NI * a.RB * a.SPR;
        bool ok = true;
        int t = first, cb = me, slot = me % a.a_slots, before = me - a.a_slots; // before: the step that used the operand slot last
        uint32_t p_phase = 0;
        while (cb >= a.cbs) { cb -= a.cbs; t += step; }
        while (me < workers && t < a.total && ok)
        {
            ok = mbar_wait(&p_full[me], p_phase, status, 47);
            if (!ok)
                break;
            const float4 *patch = reinterpret_cast<const float4 *>(smem + a.p_off + (size_t)me * a.p_slot) + q;
            uint8_t *hi = smem + (size_t)slot * A_SLOT;
            const float4 *f = reinterpret_cast<const float4 *>(s_dwf + cb * 144) + q;
            const float4 b = reinterpret_cast<const float4 *>(s_dwf + a.C * 9 + cb * CB)[q];
            for (int u0 = 0; u0 < units && ok; u0 += 8)
            {
                const int u = min(u0 + (lane >> 2), units - 1); // neighbouring units are neighbouring blocks of a row
                const int ub = a.by_SPR.div(u), sc = u - ub * a.SPR, ni = a.by_RB.div(ub), r0 = (ub - ni * a.RB) * R;
                const float4 *src = patch + ((ni * a.PR + r0 * S) * a.PW + sc * P * S) * 4;
                constexpr int NC = (P - 1) * S + 3, NR = (R - 1) * S + 3;
                float4 acc[R][P];
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int o = 0; o < P; ++o)
                        acc[r][o] = b;
#pragma unroll
                for (int ih = 0; ih < NR; ++ih)
                {
                    float4 x[NC];
#pragma unroll
                    for (int j = 0; j < NC; ++j)
                        x[j] = src[j * 4];
                    src += a.PW * 4;
#pragma unroll
                    for (int kh = 0; kh < 3; ++kh)
                    {
                        if ((ih - kh) % S != 0 || ih - kh < 0 || (ih - kh) / S >= R)
                            continue;
                        const int r = (ih - kh) / S;
#pragma unroll
                        for (int kw = 0; kw < 3; ++kw)
                        {
                            const float4 fv = f[(kh * 3 + kw) * 4];
#pragma unroll
                            for (int o = 0; o < P; ++o)
                                fma4(acc[r][o], x[o * S + kw], fv);
                        }
                    }
                }
                if (u0 == 0 && before >= 0)
                    ok = wait_step(&a_done, before, status, 41);
                if (ok && u0 + (lane >> 2) < units)
                {
#pragma unroll
                    for (int r = 0; r < R; ++r)
#pragma unroll
                        for (int o = 0; o < P; ++o)
                        {
                            float4 v = acc[r][o];
                            v.x = apply_act_ns(v.x, a.ns1); v.y = apply_act_ns(v.y, a.ns1);
                            v.z = apply_act_ns(v.z, a.ns1); v.w = apply_act_ns(v.w, a.ns1);
                            const int m = (ni * a.TH + r0 + r) * a.TW + sc * P + o;
                            float4 *at = reinterpret_cast<float4 *>(hi + m * 64 + ((q ^ ((m >> 1) & 3)) << 4));
                            if (sc * P + o < a.TW && r0 + r < a.TH) // a last block may reach beyond the tile
                            {
                                at[0] = v;
                                at[A_PART / 16] = lo_part(v);
                            }
                        }
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (ok && lane == 0)
            {
                mbar_arrive(&p_empty[me]);
                mbar_arrive(&a_full[slot]);
            }
            p_phase ^= 1;
            slot += workers;
            while (slot >= a.a_slots)
                slot -= a.a_slots;
            before += workers;
            cb += workers;
            while (cb >= a.cbs) { cb -= a.cbs; t += step; }
        }
    }
    else if (warp >= FIRST_EPI_WARP)
    {
        // ---------------- sums, bias, activation, stores ----------------
        const int quarter = warp & 3, half = (warp - FIRST_EPI_WARP) >> 2;
        const int hw = a.Ho * a.Wo;
        const int m = quarter * 32 + lane, rr = a.by_TW.div(m), ni = a.by_TH.div(rr);
        const int r = rr - ni * a.TH, c = m - rr * a.TW; // this lane's pixel of a tile
        const bool sectors = whole_sectors(out);
        bool ok = true;
        int buf = 0;
        uint32_t phase = 0;
        // one channel block: the two halves of the warps take whole tiles in turn
        const bool alternate = a.KT == CB;
        int turn = 0;
        for (int t = first; t < a.total && ok; t += step, turn ^= 1)
        {
            if (alternate && turn != half)
            {
                if (++buf == a.d_bufs) { buf = 0; phase ^= 1; }
                continue;
            }
            const int kt = a.k_tiles == 1 ? 0 : a.by_px_tiles.div(t), kv = min(a.KT, a.K - kt * a.KT);
            const DpTile T = dp_tile(a, t);
            const int n = T.n0 + ni, oh = T.r0 + r, ow = T.c0 + c;
            const bool live = ni < a.NI && n < a.N && oh < a.Ho && ow < a.Wo;
            float *o = out + ((long long)n * (a.K / CB) + (long long)kt * (a.KT / CB)) * hw * CB + ((long long)oh * a.Wo + ow) * CB;
            ok = mbar_wait(&d_full[buf], phase, status, 45, 1u << 22);
            if (!ok)
                break;
            tc_fence_after_sync();
            const uint32_t d = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * a.d_cols);
            for (int kb = alternate ? 0 : half; kb < kv / CB; kb += alternate ? 1 : 2)
            {
                uint32_t v[16], x[16];
                tmem_ld16(d + (uint32_t)(kb * CB), v);
                tmem_ld16(d + (uint32_t)(a.KT + kb * CB), x);
                tmem_ld_wait();
                float y[16];
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    y[e] = __uint_as_float(v[e]) + __uint_as_float(x[e]);
                for (int g = 1; g < a.sums; ++g)
                {
                    tmem_ld16(d + (uint32_t)((g + 1) * a.KT + kb * CB), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        y[e] += __uint_as_float(v[e]);
                }
                if (live)
                {
                    float4 *dst = reinterpret_cast<float4 *>(o + (long long)kb * hw * CB);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                    {
                        const float4 b = a.has_b2 ? __ldg(reinterpret_cast<const float4 *>(b2 + kt * a.KT + kb * CB) + j)
                                                  : make_float4(0.f, 0.f, 0.f, 0.f);
                        y[4 * j] = apply_act_ns(y[4 * j] + b.x, a.ns2); y[4 * j + 1] = apply_act_ns(y[4 * j + 1] + b.y, a.ns2);
                        y[4 * j + 2] = apply_act_ns(y[4 * j + 2] + b.z, a.ns2); y[4 * j + 3] = apply_act_ns(y[4 * j + 3] + b.w, a.ns2);
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
} // namespace

namespace
{
// The plan of a pair; false where the pair is not covered.
bool plan_dwpw(const small_b200_layer *D, const small_b200_layer *L, DpArgs &a, int &R)
{
    if (!D || !L || D->Fh != 3 || D->Fw != 3 || D->stride < 1 || D->stride > 2 || row_stride(D) != D->stride || D->accumulate ||
        L->accumulate || L->Fh != 1 || L->Fw != 1 || L->stride != 1 || row_stride(L) != 1 || L->pad_t || L->pad_b || L->pad_l || L->pad_r)
        return false;
    if (D->N < 0 || D->H <= 0 || D->W <= 0 || D->C <= 0 || D->C % CB || L->K <= 0 || L->K % CB || L->C != D->C || L->N != D->N ||
        D->pad_t < 0 || D->pad_l < 0 || D->pad_b < 0 || D->pad_r < 0)
        return false;
    a = DpArgs{};
    a.N = D->N; a.C = D->C; a.K = L->K; a.H = D->H; a.W = D->W; a.pad_t = D->pad_t; a.pad_l = D->pad_l;
    a.Ho = out_dim(D->H, D->pad_t, D->pad_b, 3, D->stride);
    a.Wo = out_dim(D->W, D->pad_l, D->pad_r, 3, D->stride);
    if (L->H != a.Ho || L->W != a.Wo || a.Ho == 0 || a.Wo == 0)
        return false;
    a.cbs = a.C / CB;
    if ((long long)a.N * a.Ho * a.Wo > 0x3fffffffLL)
        return false;
    a.KT = a.K < 128 ? a.K : 128;
    a.sums = (a.cbs + CBS_PER_SUM - 1) / CBS_PER_SUM;
    a.d_cols = (a.sums + 1) * a.KT;
    if (a.d_cols > 512)
        return false;
    a.d_bufs = 2 * a.d_cols <= 512 ? 2 : 1;
    // The tile: at most 128 pixels, several images where one does not fill it.  The estimate per tile: bytes of the patch and
    // of the outputs, passes of a depthwise warp (eight blocks each), and what a tile costs whatever it holds.
    // A patch row of at most 31 pixels is one TMA box row.
    const int S = D->stride;
    double best = 0;
    for (int tw = a.Wo < 29 ? a.Wo : 29; tw >= 1; --tw)
        for (int r = S == 1 ? 4 : 3; r >= (S == 1 ? 3 : 2); --r)
        {
            const int spr = (tw + P - 1) / P, odd = ((spr * P - 1) * S + 3) | 1;
            if (odd > 31 || (tw < a.Wo && tw % P))
                continue;
            for (int th = 1; th <= a.Ho && th * tw <= 128; ++th)
            {
                int ni = th == a.Ho && tw == a.Wo ? 128 / (th * tw) : 1;
                ni = ni > a.N ? (a.N > 0 ? a.N : 1) : ni;
                for (; ni >= 1; --ni)
                {
                    const int rb = (th + r - 1) / r, pr = (rb * r - 1) * S + 3;
                    const double tiles = (double)((a.Wo + tw - 1) / tw) * ((a.Ho + th - 1) / th) * ((a.N + ni - 1) / ni);
                    const double passes = (ni * rb * spr + 7) / 8;
                    const double cost = tiles * (odd * pr * ni + tw * th * ni + passes * r * P * S * 10 + 60);
                    if ((size_t)odd * pr * ni * 64 <= 40 * 1024 && (best == 0 || cost < best))
                    {
                        best = cost;
                        R = r; a.TW = tw; a.TH = th; a.NI = ni; a.PW = odd; a.PR = pr; a.SPR = spr; a.RB = rb;
                    }
                }
            }
        }
    if (best == 0)
        return false;
    a.tiles_x = (a.Wo + a.TW - 1) / a.TW; a.tiles_y = (a.Ho + a.TH - 1) / a.TH;
    a.px_tiles = a.tiles_x * a.tiles_y * ((a.N + a.NI - 1) / a.NI);
    a.p_bytes = (unsigned)(a.PW * a.PR * a.NI * 64);
    a.p_slot = (a.p_bytes + 1023u) & ~1023u;
    a.k_tiles = (a.K + a.KT - 1) / a.KT;
    a.total = a.px_tiles * a.k_tiles;
    // Operand slots; the filter whole where it fits beside four patches (and a CTA never changes its channel tile), else a
    // ring; patches for what is left: every depthwise warp holds one while it works.
    const size_t stage = (size_t)a.KT * 128, dw = ((size_t)a.C * 40 + 1023) & ~(size_t)1023, limit = 224 * 1024;
    a.w_resident = 0;
    size_t room = 0;
    for (a.a_slots = A_SLOTS_MAX; a.a_slots >= 2 && !a.w_resident; --a.a_slots)
    {
        room = limit - a.a_slots * (size_t)A_SLOT - dw;
        a.w_resident = a.k_tiles == 1 && a.cbs <= W_STAGES_MAX && a.cbs * stage + 4 * (size_t)a.p_slot <= room;
        if (a.w_resident)
            break;
    }
    if (!a.w_resident)
    {
        a.a_slots = A_SLOTS_MAX;
        room = limit - a.a_slots * (size_t)A_SLOT - dw;
    }
    a.w_stages = a.w_resident ? a.cbs : 4;
    if (a.w_stages * stage + 2 * (size_t)a.p_slot > room)
        return false;
    size_t slots = (room - a.w_stages * stage) / a.p_slot;
    if (slots > P_SLOTS_MAX)
        slots = P_SLOTS_MAX;
    a.p_slots = (int)slots;
    a.p_off = a.a_slots * A_SLOT;
    a.w_off = a.p_off + a.p_slots * a.p_slot;
    a.dwf_off = a.w_off + (unsigned)(a.w_stages * stage);
    a.by_px_tiles.set(a.px_tiles > 0 ? a.px_tiles : 1); a.by_tiles_x.set(a.tiles_x); a.by_tiles_y.set(a.tiles_y);
    a.by_SPR.set(a.SPR); a.by_RB.set(a.RB); a.by_TH.set(a.TH); a.by_TW.set(a.TW);
    return true;
}

template <int S, int R>
int launch_dwpw(const CUtensorMap &mx, const DpArgs &a, const float *dwf, const float *b1, const float *pwf, const float *b2, float *out,
                cudaStream_t st)
{
    static PerDeviceOnce configured;
    int dev;
    if (configured.needed(&dev))
    {
        SB_CUDA(cudaFuncSetAttribute(dwpw_f32_kernel<S, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        configured.mark(dev);
    }
    int *status = device_status_ptr();
    if (!status)
        return fail(SMALL_B200_CUDA_ERROR, "device status word not available");
    const int grid = a.total < num_sms() ? a.total : num_sms();
    const size_t smem = a.dwf_off + (((size_t)a.C * 40 + 1023) & ~(size_t)1023);
    dwpw_f32_kernel<S, R><<<(unsigned)grid, THREADS, smem, st>>>(mx, a, dwf, b1, pwf, b2, out, status);
    return launched("dwpw_f32_kernel");
}
} // namespace

extern "C"
{
int small_b200_dwconv2d_conv2d_f32_supported(const small_b200_layer *dw, const small_b200_layer *pw)
{
    DpArgs a;
    int R;
    return plan_dwpw(dw, pw, a, R) ? 1 : 0;
}

// Layers of a small batch: where the depthwise layer (3 to 4 us) and the latency kernel for the 1x1 layer together stay below
// this kernel's 6 (16 channels) to 13 us (256), two launches are the shorter way.
int small_b200_dwconv2d_conv2d_f32_preferred(const small_b200_layer *dw, const small_b200_layer *pw)
{
    if (!small_b200_dwconv2d_conv2d_f32_supported(dw, pw))
        return 0;
    return conv_small_preferred(pw) && 3.5 + conv_small_us(pw) < 6.5 + 0.03 * dw->C ? 0 : 1;
}

int small_b200_filter_prepare_dwconv2d_conv2d_f32(const small_b200_layer *pw, const float *filt, float *prepared, void *stream)
{
    if (!pw || pw->C <= 0 || pw->K <= 0 || pw->C % CB || pw->K % CB)
        return fail(SMALL_B200_INVALID_ARGUMENT, "DepthwiseConv2D+Conv2D<float> ERROR: channels unsupported.");
    const long long n = (long long)pw->K * pw->C;
    if (n > 0x7fffffffLL)
        return fail(SMALL_B200_INVALID_ARGUMENT, "DepthwiseConv2D+Conv2D<float> ERROR: filter too large.");
    prepare_pw_kernel<<<(unsigned)((n + 255) / 256), 256, 0, as_stream(stream)>>>((int)n, pw->C / CB, pw->K, pw->K < 128 ? pw->K : 128,
                                                                               filt, prepared);
    return launched("prepare_pw_kernel");
}

int small_b200_dwconv2d_conv2d_f32(const small_b200_layer *dw, const small_b200_layer *pw, const float *in, const float *dw_filt,
                                   const float *dw_bias, const float *pw_prepared, const float *pw_bias, float *out, void *stream)
{
    if (int rc = check_window_layer(dw, "DepthwiseConv2D<float>", false, 2))
        return rc;
    if (int rc = check_window_layer(pw, "Conv2D<float>", true, 2))
        return rc;
    DpArgs a;
    int R;
    if (!plan_dwpw(dw, pw, a, R))
        return fail(SMALL_B200_INVALID_ARGUMENT, "DepthwiseConv2D+Conv2D<float> ERROR: pair not covered by the one-kernel form.");
    if (a.N == 0)
        return SMALL_B200_OK;
    a.ns1 = dw->act == SMALL_B200_ACT_RELU ? 0.f : dw->act == SMALL_B200_ACT_LEAKY ? dw->slope : 1.f;
    a.ns2 = pw->act == SMALL_B200_ACT_RELU ? 0.f : pw->act == SMALL_B200_ACT_LEAKY ? pw->slope : 1.f;
    a.has_b1 = dw_bias != nullptr; a.has_b2 = pw_bias != nullptr;
    cudaStream_t st = as_stream(stream);
    const int direct = dwpw_direct_f32(dw, pw, in, dw_filt, dw_bias, pw_prepared, pw_bias, out, st);
    if (direct >= 0)
        return direct;
    CUtensorMap mx; // [N][C/16][H][W x 8 elements of 8 bytes]
    {
        const uint64_t dims[4] = {(uint64_t)a.W * 8, (uint64_t)a.H, (uint64_t)a.cbs, (uint64_t)a.N};
        const uint64_t strides[3] = {(uint64_t)a.W * 64, (uint64_t)a.H * a.W * 64, (uint64_t)a.cbs * a.H * a.W * 64};
        const uint32_t box[4] = {(uint32_t)a.PW * 8, (uint32_t)a.PR, 1, (uint32_t)a.NI};
        if (int rc = make_tensor_map(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, in, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE))
            return rc;
    }
    if (dw->stride == 1)
        return R == 4 ? launch_dwpw<1, 4>(mx, a, dw_filt, dw_bias, pw_prepared, pw_bias, out, st)
                      : launch_dwpw<1, 3>(mx, a, dw_filt, dw_bias, pw_prepared, pw_bias, out, st);
    return R == 3 ? launch_dwpw<2, 3>(mx, a, dw_filt, dw_bias, pw_prepared, pw_bias, out, st)
                  : launch_dwpw<2, 2>(mx, a, dw_filt, dw_bias, pw_prepared, pw_bias, out, st);
}
} // extern "C"
