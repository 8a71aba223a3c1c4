// dwpw_direct_f32.cu -- the depthwise-separable blocks of few channels (dwpw_f32.cu's layers, up to 32 -> 32) on the FMA pipe.
//
// With 16 channels a pixel's 1x1 convolution is 256 multiply-adds: less than what it takes to write the pixel's values as
// two tensor-core operands, issue the MMAs and add up their columns.  Here a thread owns V outputs of a column (4 with 16 output
// channels, 2 with 32) and all their channels.  Four input channels at a time it reads the windows of its outputs, sums the depthwise layer
// in registers, and multiplies the result into its 64 sums; multiply-adds are packed in pairs (fma.rn.f32x2), of channels in the
// depthwise layer, of output channels in the 1x1 layer.  Plain fp32 sums in the order of the two layers: infinities and NaN come out as theirs.
//
// A CTA is one tile: rows of the full width where that is at most 64, one TMA box per 16 channels (zeros outside the image) in the
// 64-byte swizzle, in which the reads of eight neighbouring pixels' same four channels fall into different banks.  Three CTAs an SM
// hide each other's fetches (160 threads of 128 registers; two of 192 take 5 to 10 % longer).
// What bounds it: shared memory (16 -> 16 at 48x48, 1024 images: 52 % of its passes, 54 % of the issue slots, 52 % of the FMA pipe) and
// the latency of a dozen warps; the memory of that block alone is 92 us at 2048 images.
// us, dwpw_f32.cu -> this: 16 -> 16 at 48x48, 2048 images 336 -> 125, 128 images 22.7 -> 11.4, one 5.7 -> 5.2; 32 -> 32 at 24x24, 2048 images
// 118 -> 104; against fp64 4.5e-7 -> 0.9e-7 (2-norm).
#include "tc_common.cuh"

#include <algorithm>

namespace
{
using namespace sb;

constexpr int CTAS = 3, MAX_THREADS = 160, SMEM_LIMIT = 222 * 1024 / CTAS; // CTAs an SM: 128 registers a thread

struct DirectArgs
{
    int N, C, H, W, Ho, Wo, pad_t, pad_l, cbs;
    int TH, TW, PR, PW, tiles_x, tiles_y;
    float ns1, ns2;
    uint32_t patch_bytes;
    FastDiv by_TW, by_tiles_x, by_tiles_y;
};

typedef unsigned long long pair;
__device__ __forceinline__ pair fma2(pair a, pair b, pair c)
{
    pair d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ pair both(float a, float b)
{
    pair d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 parts(pair a)
{
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(a));
    return d;
}

template <int K, int S>
__global__ void __launch_bounds__(MAX_THREADS, CTAS)
dwpw_direct_f32_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ DirectArgs a, const float *__restrict__ dwf,
                       const float *__restrict__ b1, const float *__restrict__ pwf, const float *__restrict__ b2, float *__restrict__ out, int *status)
{
    constexpr int V = 64 / K, WINDOW = (V - 1) * S + 3; // outputs of a thread, rows of input they reach
    extern __shared__ __align__(1024) uint8_t smem[];   // [16-channel block][row][column][16], 64-byte swizzle; then dw [C/16][9][16], pw [C][K], biases
    __shared__ __align__(8) uint64_t full;
    float *s_dw = reinterpret_cast<float *>(smem + a.cbs * a.patch_bytes), *s_pw = s_dw + a.C * 9, *s_b1 = s_pw + a.C * K, *s_b2 = s_b1 + a.C;
    const int tid = threadIdx.x;
    const int t1 = a.by_tiles_x.div(blockIdx.x), n = a.by_tiles_y.div(t1), r0 = (t1 - n * a.tiles_y) * a.TH, c0 = ((int)blockIdx.x - t1 * a.tiles_x) * a.TW;
    if (tid == 0)
    {
        mbar_init(&full, 1);
        fence_barrier_init();
        mbar_expect_tx(&full, a.cbs * a.patch_bytes);
        for (int cb = 0; cb < a.cbs; ++cb)
            tma_load_5d(smem + cb * a.patch_bytes, &map_x, 0, c0 * S - a.pad_l, r0 * S - a.pad_t, cb, n, &full);
    }
    for (int i = tid; i < a.C * 9; i += blockDim.x)
        s_dw[i] = __ldg(dwf + i);
    for (int i = tid; i < a.C * K; i += blockDim.x)
    {
        const int c = i / K, k = i % K; // prepared for dwpw_f32.cu: [c/4][k][4 c], the value itself, then its second word
        s_pw[i] = __ldg(pwf + (c >> 2) * 8 * K + k * 4 + (c & 3));
    }
    for (int i = tid; i < a.C; i += blockDim.x)
        s_b1[i] = b1 ? __ldg(b1 + i) : 0.f;
    if (tid < K)
        s_b2[tid] = b2 ? __ldg(b2 + tid) : 0.f;
    __syncthreads();
    if (!mbar_wait(&full, 0, status, 85))
        return;
    const int strip = a.by_TW.div(tid), x = tid - strip * a.TW, row = strip * V;
    if (row >= a.TH || c0 + x >= a.Wo)
        return;
    pair acc[V][K / 2];
#pragma unroll
    for (int k = 0; k < K / 2; ++k)
    {
        const pair b = *reinterpret_cast<const pair *>(s_b2 + 2 * k);
#pragma unroll
        for (int v = 0; v < V; ++v)
            acc[v][k] = b;
    }
    const uint32_t pitch = (uint32_t)a.PW * 64;
    const uint8_t *window = smem + (uint32_t)(row * S) * pitch + (uint32_t)(x * S) * 64;
    uint32_t swizzle[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
        swizzle[j] = (uint32_t)((x * S + j) >> 1 & 3) << 4;
#pragma unroll 1
    for (int c4 = 0; c4 < a.C / 4; ++c4)
    {
        const uint8_t *p = window + (c4 >> 2) * a.patch_bytes;
        const float *w = s_dw + (c4 >> 2) * 9 * CB + (c4 & 3) * 4;
        const uint8_t *col[3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
            col[j] = p + j * 64 + (swizzle[j] ^ (uint32_t)(c4 & 3) << 4);
        ulonglong2 d[V];
#pragma unroll
        for (int v = 0; v < V; ++v)
            d[v] = *reinterpret_cast<const ulonglong2 *>(s_b1 + c4 * 4);
#pragma unroll
        for (int j = 0; j < 3; ++j) // a column of the window at a time: three taps in registers, not nine
        {
            ulonglong2 taps[3];
#pragma unroll
            for (int t = 0; t < 3; ++t)
                taps[t] = *reinterpret_cast<const ulonglong2 *>(w + (t * 3 + j) * CB);
#pragma unroll
            for (int r = 0; r < WINDOW; ++r)
            {
                const ulonglong2 in = *reinterpret_cast<const ulonglong2 *>(col[j] + r * pitch);
#pragma unroll
                for (int v = 0; v < V; ++v)
                    if (r - v * S >= 0 && r - v * S < 3)
                    {
                        d[v].x = fma2(in.x, taps[r - v * S].x, d[v].x);
                        d[v].y = fma2(in.y, taps[r - v * S].y, d[v].y);
                    }
            }
        }
        float y[V][4];
#pragma unroll
        for (int v = 0; v < V; ++v)
        {
            const float2 lo = parts(d[v].x), hi = parts(d[v].y);
            y[v][0] = apply_act_ns(lo.x, a.ns1); y[v][1] = apply_act_ns(lo.y, a.ns1);
            y[v][2] = apply_act_ns(hi.x, a.ns1); y[v][3] = apply_act_ns(hi.y, a.ns1);
        }
        const float *m = s_pw + c4 * 4 * K;
#pragma unroll
        for (int c = 0; c < 4; ++c)
        {
            pair yy[V];
#pragma unroll
            for (int v = 0; v < V; ++v)
                yy[v] = both(y[v][c], y[v][c]);
#pragma unroll
            for (int k = 0; k < K / 4; ++k)
            {
                const ulonglong2 wk = *reinterpret_cast<const ulonglong2 *>(m + c * K + 4 * k);
#pragma unroll
                for (int v = 0; v < V; ++v)
                {
                    acc[v][2 * k] = fma2(yy[v], wk.x, acc[v][2 * k]);
                    acc[v][2 * k + 1] = fma2(yy[v], wk.y, acc[v][2 * k + 1]);
                }
            }
        }
    }
    float *o = out + (((size_t)n * (K / CB) * a.Ho + r0 + row) * a.Wo + c0 + x) * CB;
#pragma unroll
    for (int v = 0; v < V; ++v)
        if (r0 + row + v < a.Ho && row + v < a.TH)
#pragma unroll
            for (int kb = 0; kb < K / CB; ++kb)
#pragma unroll
                for (int q = 0; q < 2; ++q)
                {
                    float y[8];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                    {
                        const float2 s = parts(acc[v][kb * 8 + 4 * q + e]);
                        y[2 * e] = apply_act_ns(s.x, a.ns2); y[2 * e + 1] = apply_act_ns(s.y, a.ns2);
                    }
                    store8(o + ((size_t)kb * a.Ho + v) * a.Wo * CB + q * 8, y, true);
                }
}

template <int K, int S>
int launch(const CUtensorMap &map, const DirectArgs &a, long long tiles, int threads, size_t smem, const float *dwf, const float *b1, const float *pwf,
           const float *b2, float *out, cudaStream_t st)
{
    auto kern = dwpw_direct_f32_kernel<K, S>;
    static PerDeviceOnce configured;
    int dev;
    if (configured.needed(&dev))
    {
        SB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 110 * 1024));
        configured.mark(dev);
    }
    int *status = device_status_ptr();
    if (!status)
        return fail(SMALL_B200_CUDA_ERROR, "device status word not available");
    kern<<<(unsigned)tiles, threads, smem, st>>>(map, a, dwf, b1, pwf, b2, out, status);
    return launched("dwpw_direct_f32_kernel");
}
} // namespace

namespace sb
{
// The pair of layers, which dwpw_f32.cu has looked over, on the FMA pipe; -1 where it leaves them to the tensor cores.
int dwpw_direct_f32(const small_b200_layer *D, const small_b200_layer *L, const float *in, const float *dwf, const float *b1, const float *pwf,
                    const float *b2, float *out, cudaStream_t st)
{
    const int S = D->stride, K = L->K;
    // Where it is the shorter way, by outputs: 32 channels from 16384 on (24x24: one image 6.4 us there and 7.6 here, 128 images 12.3 and
    // 10.7); a stride of two, where a warp's reads meet in pairs of banks, for 16 -> 32 up to 131072 (48x48: 16 images 6.5 and
    // 5.0, 2048 87 and 89; 32 -> 16 36 and 77) and from 40 on (6x6, one image 5.4 there and 5.7 here, 33x7 6.3 and 4.1).
    const long long outputs = (long long)D->N * L->H * L->W;
    if (S == 2 ? D->C != 16 || K != 32 || outputs < 40 || outputs > 131072 : D->C > 16 && outputs < 16384)
        return -1;
    if (D->C > 32 || (K != 16 && K != 32) || (reinterpret_cast<uintptr_t>(in) & 15) != 0 || (reinterpret_cast<uintptr_t>(out) & 31) != 0)
        return -1;
    DirectArgs a{};
    a.N = D->N; a.C = D->C; a.H = D->H; a.W = D->W; a.Ho = L->H; a.Wo = L->W; a.pad_t = D->pad_t; a.pad_l = D->pad_l; a.cbs = a.C / CB;
    const int V = 64 / K, parts = (a.Wo + 63) / 64;
    a.TW = (a.Wo + parts - 1) / parts;
    a.PW = ((a.TW - 1) * S + 3 + 7) & ~7; // a multiple of eight: the swizzle of a pixel is its column's
    auto rows_in = [&](int TH) { return (TH - 1) * S + 3; };
    auto bytes = [&](int TH) { return a.cbs * rows_in(TH) * a.PW * 64; };
    int TH = V;
    while (TH < a.Ho && a.TW * (TH / V + 1) <= MAX_THREADS && bytes(TH + V) <= SMEM_LIMIT - 6 * 1024)
        TH += V;
    const int ty = (a.Ho + TH - 1) / TH;
    TH = ((a.Ho + ty - 1) / ty + V - 1) / V * V;
    if (bytes(TH) > 100 * 1024 || rows_in(TH) > 256 || a.PW > 256)
        return -1;
    a.TH = TH; a.PR = rows_in(TH); a.tiles_x = parts; a.tiles_y = (a.Ho + TH - 1) / TH;
    a.patch_bytes = (uint32_t)(a.PR * a.PW * 64);
    const long long tiles = (long long)a.N * a.tiles_x * a.tiles_y;
    if (tiles > 0x3fffffff)
        return -1;
    a.ns1 = D->act == SMALL_B200_ACT_RELU ? 0.f : D->act == SMALL_B200_ACT_LEAKY ? D->slope : 1.f;
    a.ns2 = L->act == SMALL_B200_ACT_RELU ? 0.f : L->act == SMALL_B200_ACT_LEAKY ? L->slope : 1.f;
    a.by_TW.set(a.TW); a.by_tiles_x.set(a.tiles_x); a.by_tiles_y.set(a.tiles_y);
    CUtensorMap map; // [N][C/16][H][W][16]
    const uint64_t dims[5] = {16, (uint64_t)a.W, (uint64_t)a.H, (uint64_t)a.cbs, (uint64_t)a.N};
    const uint64_t strides[4] = {64, (uint64_t)a.W * 64, (uint64_t)a.H * a.W * 64, (uint64_t)a.cbs * a.H * a.W * 64};
    const uint32_t box[5] = {16, (uint32_t)a.PW, (uint32_t)a.PR, 1, 1};
    if (int rc = make_tensor_map(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, in, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B))
        return rc;
    const int threads = (a.TW * (TH / V) + 31) & ~31;
    // 32 channels, where the gain is small: not in tiles of one warp, which leave an SM with three of them (18x5, 256 images 7.9 us there and
    // 9.7 here), and not where threads without outputs and pixels fetched for several tiles, or for none, are four times what is
    // needed (5x126, 256 images 22.0 and 27.8).
    const double slots = (double)tiles * threads * V / outputs, fetched = (double)tiles * a.PR * a.PW / outputs;
    if (a.C > CB && (threads == 32 || (K == 32 && slots * fetched > 4)))
        return -1;
    const size_t smem = (size_t)a.cbs * a.patch_bytes + (size_t)(a.C * 9 + a.C * K + a.C + K) * sizeof(float);
#define SB_DIRECT(K_, S_) \
    if (K == K_ && S == S_) \
        return launch<K_, S_>(map, a, tiles, threads, smem, dwf, b1, pwf, b2, out, st);
    SB_DIRECT(16, 1) SB_DIRECT(32, 1) SB_DIRECT(32, 2)
#undef SB_DIRECT
    return -1;
}
} // namespace sb
