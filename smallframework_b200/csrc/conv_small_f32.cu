// conv_small_f32.cu -- fp32 layers that are too small for anything but latency: convolutions of a few million
// multiply-adds (a small network on one image), and the tail of a classifier (global average pool, dense layer, softmax).
//
// What bounds them: nothing but the chain start of a kernel -> loads -> sums -> store.  The tensor-core kernel needs 8 to 10
// us from its first instruction to its last whatever it computes, the staged CUDA-core kernel walks over its channel
// blocks one after the other in a handful of CTAs (22 us for 32 -> 64 channels, stride 2, at 16x16).  Here the reduction is
// what the threads share: a CTA owns 8 output pixels of a row x 16 output channels, its eight warps take the (channel
// block, tap) pairs in turn, and in a warp eight groups of four lanes take the channels; every load is independent
// of every other, and two small reductions (lanes, then warps) end it.  Filter blocks [16 c][16 k] are read as they
// are packed, 512 contiguous bytes per warp and load.
#include "common.cuh"

#include "tc_common.cuh"

namespace
{
using namespace sb;

constexpr int PX = 8, WARPS = 8; // pixels per CTA, warps that share the reduction

struct SmallArgs
{
    int N, C, K, H, W, Ho, Wo, Fh, Fw, sw, sh, pad_t, pad_l, cbs, taps, segs;
    int accumulate, has_bias;
    float ns;
    FastDiv by_taps, by_Fw, by_segs, by_Ho;
};

__global__ void __launch_bounds__(WARPS * 32)
conv_small_f32_kernel(const SmallArgs a, const float *__restrict__ in, const float *__restrict__ filt, const float *__restrict__ bias,
                      float *__restrict__ out)
{
    __shared__ float sums[WARPS][PX * CB];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane & 3, cg = lane >> 2;
    const int kb = blockIdx.y, row = a.by_segs.div((int)blockIdx.x), n = a.by_Ho.div(row);
    const int oh = row - n * a.Ho, ow0 = ((int)blockIdx.x - row * a.segs) * PX;
    const int ih0 = oh * a.sh - a.pad_t, iw0 = ow0 * a.sw - a.pad_l;
    const float *img = in + (long long)n * a.cbs * a.H * a.W * CB + cg;
    const float4 *w = reinterpret_cast<const float4 *>(filt + (long long)kb * a.cbs * a.taps * CB * CB) + cg * 4 + q;
    float4 acc[PX];
#pragma unroll
    for (int p = 0; p < PX; ++p)
        acc[p] = make_float4(0.f, 0.f, 0.f, 0.f);
    // the run of pixels is inside the image for the whole window, as nearly everywhere
    const bool inside = iw0 >= 0 && iw0 + (PX - 1) * a.sw + a.Fw <= a.W;
    for (int pair = warp; pair < a.cbs * a.taps; pair += WARPS)
    {
        const int cb = a.by_taps.div(pair), tap = pair - cb * a.taps, kh = a.by_Fw.div(tap), kw = tap - kh * a.Fw;
        const int ih = ih0 + kh;
        if ((uint32_t)ih >= (uint32_t)a.H)
            continue;
        const float *x = img + ((long long)cb * a.H + ih) * a.W * CB + (long long)(iw0 + kw) * CB;
#pragma unroll
        for (int half = 0; half < 2; ++half) // channels 8 * half + cg
        {
            const float4 f = __ldg(w + pair * 64 + half * 32);
            float v[PX];
#pragma unroll
            for (int p = 0; p < PX; ++p)
                v[p] = (inside || (uint32_t)(iw0 + kw + p * a.sw) < (uint32_t)a.W) ? __ldg(x + p * a.sw * CB + half * 8) : 0.f;
#pragma unroll
            for (int p = 0; p < PX; ++p)
            {
                acc[p].x = fmaf(v[p], f.x, acc[p].x); acc[p].y = fmaf(v[p], f.y, acc[p].y);
                acc[p].z = fmaf(v[p], f.z, acc[p].z); acc[p].w = fmaf(v[p], f.w, acc[p].w);
            }
        }
    }
    // eight channel groups (lane bits 2..4): every step halves the pixels a lane answers for
#pragma unroll
    for (int step = 0, half = PX / 2; step < 3; ++step, half >>= 1)
    {
        const int mask = 16 >> step;
        const bool upper = lane & mask;
#pragma unroll
        for (int p = 0; p < PX / 2; ++p)
            if (p < half)
            {
                const float4 keep = upper ? acc[p + half] : acc[p], give = upper ? acc[p] : acc[p + half];
                acc[p].x = keep.x + __shfl_xor_sync(0xffffffffu, give.x, mask);
                acc[p].y = keep.y + __shfl_xor_sync(0xffffffffu, give.y, mask);
                acc[p].z = keep.z + __shfl_xor_sync(0xffffffffu, give.z, mask);
                acc[p].w = keep.w + __shfl_xor_sync(0xffffffffu, give.w, mask);
            }
    }
    const int mine = (lane & 16 ? 4 : 0) + (lane & 8 ? 2 : 0) + (lane & 4 ? 1 : 0); // the pixel this lane ended with
    *reinterpret_cast<float4 *>(&sums[warp][mine * CB + q * 4]) = acc[0];
    __syncthreads();
    if (tid < PX * CB)
    {
        const int p = tid >> 4, k = tid & 15;
        if (ow0 + p < a.Wo)
        {
            float *o = out + ((((long long)n * (a.K / CB) + kb) * a.Ho + oh) * a.Wo + ow0 + p) * CB + k;
            float y = a.has_bias ? __ldg(bias + kb * CB + k) : 0.f;
            if (a.accumulate)
                y += *o;
#pragma unroll
            for (int g = 0; g < WARPS; ++g)
                y += sums[g][tid];
            *o = apply_act_ns(y, a.ns);
        }
    }
}

// First layer (CI = 1 to 3 interleaved channels): a thread owns four output channels of one pixel.  F: the window's size where
// it is 3x3 (all loads of a thread go out together), 0 for any other.
template <int CI, int F>
__global__ void __launch_bounds__(256)
conv_first_small_f32_kernel(const SmallArgs a, const float *__restrict__ in, const float *__restrict__ filt, const float *__restrict__ bias,
                            float *__restrict__ out)
{
    const int i = blockIdx.x * 256 + threadIdx.x, q = i & 3, px = i >> 2, kb = blockIdx.y;
    if (px >= a.N * a.Ho * a.Wo)
        return;
    const int row = a.by_segs.div(px), ow = px - row * a.Wo, n = a.by_Ho.div(row), oh = row - n * a.Ho; // by_segs: division by Wo here
    float4 acc = a.has_bias ? __ldg(reinterpret_cast<const float4 *>(bias + kb * CB) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 *w = reinterpret_cast<const float4 *>(filt + (long long)kb * a.taps * CI * CB) + q;
    float4 *o = reinterpret_cast<float4 *>(out + ((((long long)n * (a.K / CB) + kb) * a.Ho + oh) * a.Wo + ow) * CB) + q;
    if (a.accumulate)
    {
        const float4 s = *o;
        acc.x += s.x; acc.y += s.y; acc.z += s.z; acc.w += s.w;
    }
    const int ih0 = oh * a.sh - a.pad_t, iw0 = ow * a.sw - a.pad_l;
    const float *x = in + (((long long)n * a.H + ih0) * a.W + iw0) * CI;
    if (F)
    {
        float v[F * F * CI + 1];
#pragma unroll
        for (int kh = 0; kh < F; ++kh)
#pragma unroll
            for (int kw = 0; kw < F; ++kw)
            {
                const bool inside = (uint32_t)(ih0 + kh) < (uint32_t)a.H && (uint32_t)(iw0 + kw) < (uint32_t)a.W;
#pragma unroll
                for (int c = 0; c < CI; ++c)
                    v[(kh * F + kw) * CI + c] = inside ? __ldg(x + (kh * a.W + kw) * CI + c) : 0.f;
            }
#pragma unroll
        for (int t = 0; t < F * F * CI; ++t)
        {
            const float4 f = __ldg(w + t * 4);
            acc.x = fmaf(v[t], f.x, acc.x); acc.y = fmaf(v[t], f.y, acc.y); acc.z = fmaf(v[t], f.z, acc.z); acc.w = fmaf(v[t], f.w, acc.w);
        }
    }
    else
        for (int kh = 0; kh < a.Fh; ++kh)
#pragma unroll 4
            for (int kw = 0; kw < a.Fw; ++kw)
            {
                const bool inside = (uint32_t)(ih0 + kh) < (uint32_t)a.H && (uint32_t)(iw0 + kw) < (uint32_t)a.W;
#pragma unroll
                for (int c = 0; c < CI; ++c)
                {
                    const float v = inside ? __ldg(x + ((long long)kh * a.W + kw) * CI + c) : 0.f;
                    const float4 f = __ldg(w + ((kh * a.Fw + kw) * CI + c) * 4);
                    acc.x = fmaf(v, f.x, acc.x); acc.y = fmaf(v, f.y, acc.y); acc.z = fmaf(v, f.z, acc.z); acc.w = fmaf(v, f.w, acc.w);
                }
            }
    acc.x = apply_act_ns(acc.x, a.ns); acc.y = apply_act_ns(acc.y, a.ns); acc.z = apply_act_ns(acc.z, a.ns); acc.w = apply_act_ns(acc.w, a.ns);
    *o = acc;
}

// Global average pool of an image, a dense layer on the averages, softmax over its (padded) outputs.  One CTA per image.
constexpr int TAIL_THREADS = 256, TAIL_K_MAX = 256, TAIL_C_MAX = 2048;
__global__ void __launch_bounds__(TAIL_THREADS)
pool_dense_softmax_f32_kernel(int C, int hw, float norm, int K, int softmax, float ns, const float *__restrict__ in, const float *__restrict__ filt,
                              const float *__restrict__ bias, float *__restrict__ out)
{
    extern __shared__ float sm[]; // [C] averages, then [16][K] partial sums of the dense layer
    __shared__ float red[TAIL_THREADS / 32];
    const int tid = threadIdx.x;
    const float *x = in + (long long)blockIdx.x * C * hw;
    // a group of four lanes averages a channel block at a time (16-byte reads, 64 bytes per pixel)
    for (int u = tid; u < C / CB * 4 * 8; u += TAIL_THREADS)
    {
        const int q = u & 3, part = (u >> 2) & 7, cb = u >> 5; // a warp per channel block: eight lane groups take the pixels
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int p = part; p < hw; p += 8)
        {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(x + ((long long)cb * hw + p) * CB) + q);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
#pragma unroll
        for (int m = 4; m < 32; m <<= 1)
        {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, m); s.y += __shfl_xor_sync(0xffffffffu, s.y, m);
            s.z += __shfl_xor_sync(0xffffffffu, s.z, m); s.w += __shfl_xor_sync(0xffffffffu, s.w, m);
        }
        if (part == 0)
            *reinterpret_cast<float4 *>(sm + cb * CB + q * 4) = make_float4(s.x * norm, s.y * norm, s.z * norm, s.w * norm);
    }
    __syncthreads();
    // dense: thread (k in a block of 16, slice of the channels); filter [K/16][C/16][16 c][16 k]
    const int k16 = tid & 15, slice = tid >> 4; // 16 slices
    for (int kb = 0; kb < K / CB; ++kb)
    {
        float s = 0.f;
        const float *w = filt + (long long)kb * C * CB + k16;
        for (int c = slice; c < C; c += TAIL_THREADS / 16)
            s = fmaf(sm[c], __ldg(w + c * CB), s);
        sm[C + slice * K + kb * CB + k16] = s;
    }
    __syncthreads();
    float mine = 0.f, e = 0.f;
    const bool live = tid < K;
    if (live)
    {
        mine = bias ? __ldg(bias + tid) : 0.f;
        for (int g = 0; g < TAIL_THREADS / 16; ++g)
            mine += sm[C + g * K + tid];
        mine = apply_act_ns(mine, ns);
    }
    if (!softmax)
    {
        if (live)
            out[(long long)blockIdx.x * K + tid] = mine;
        return;
    }
    e = live ? expf(mine) : 0.f;
    float t = e;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1)
        t += __shfl_xor_sync(0xffffffffu, t, m);
    if ((tid & 31) == 0)
        red[tid >> 5] = t;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int g = 0; g < TAIL_THREADS / 32; ++g)
        total += red[g];
    if (live)
        out[(long long)blockIdx.x * K + tid] = e * (float)(1.0 / (double)total);
}

bool tail_covered(const small_b200_layer *P, const small_b200_layer *D)
{
    return P && D && P->H > 0 && P->W > 0 && P->Fh == P->H && P->Fw == P->W && !P->pad_t && !P->pad_b && !P->pad_l && !P->pad_r && P->C > 0 &&
           P->C % CB == 0 && P->C <= TAIL_C_MAX && D->C == P->C && D->N == P->N && D->H == 1 && D->W == 1 && D->Fh == 1 && D->Fw == 1 &&
           !D->pad_t && !D->pad_b && !D->pad_l && !D->pad_r && !D->accumulate && D->K > 0 && D->K % CB == 0 && D->K <= TAIL_K_MAX;
}
} // namespace

namespace sb
{
// Estimated microseconds of conv_small_f32_kernel: the launch, then waves of CTAs (three on an SM), each a chain of loads
// and reductions plus the pairs its warps walk through (measured: 3.2 us for 16 -> 16 channels 3x3 at 32x32, 5.2 for 64 -> 64
// at 8x8, 9.5 for 2048 CTAs of a single pair).
double conv_small_us(const small_b200_layer *L)
{
    const long long ho = out_dim(L->H, L->pad_t, L->pad_b, L->Fh, row_stride(L)), wo = out_dim(L->W, L->pad_l, L->pad_r, L->Fw, L->stride);
    if (L->C < CB)
        return 2.0 + 1e-6 * (double)L->N * ho * wo * L->K * L->C * L->Fh * L->Fw;
    const long long ctas = (long long)L->N * ho * ((wo + PX - 1) / PX) * (L->K / CB), room = 3LL * num_sms();
    return 1.3 + (double)((ctas + room - 1) / room) * (1.5 + 0.065 * (L->C / CB) * L->Fh * L->Fw);
}
// Where the estimate is below what the tensor-core kernel takes for anything (8 to 10 us), up to 12 Mi multiply-adds.
bool conv_small_preferred(const small_b200_layer *L)
{
    if ((L->C % CB && L->C > 3) || L->N <= 0 || L->C <= 0 || L->K <= 0 || L->K % CB || L->H <= 0 || L->W <= 0 || L->Fh <= 0 || L->Fw <= 0 ||
        L->stride <= 0)
        return false;
    const long long ho = out_dim(L->H, L->pad_t, L->pad_b, L->Fh, row_stride(L)), wo = out_dim(L->W, L->pad_l, L->pad_r, L->Fw, L->stride);
    return (long long)L->N * ho * wo * L->K * L->C * L->Fh * L->Fw <= (12LL << 20) && conv_small_us(L) <= 9.0;
}
int conv_small_f32(const small_b200_layer *L, const float *in, const float *filt, const float *bias, float *out, cudaStream_t st)
{
    SmallArgs a = {};
    a.N = L->N; a.C = L->C; a.K = L->K; a.H = L->H; a.W = L->W; a.Fh = L->Fh; a.Fw = L->Fw;
    a.sw = L->stride; a.sh = row_stride(L); a.pad_t = L->pad_t; a.pad_l = L->pad_l;
    a.Ho = out_dim(L->H, L->pad_t, L->pad_b, L->Fh, a.sh);
    a.Wo = out_dim(L->W, L->pad_l, L->pad_r, L->Fw, a.sw);
    a.cbs = L->C / CB; a.taps = L->Fh * L->Fw; a.segs = (a.Wo + PX - 1) / PX;
    a.accumulate = L->accumulate; a.has_bias = bias != nullptr;
    a.ns = L->act == SMALL_B200_ACT_RELU ? 0.f : L->act == SMALL_B200_ACT_LEAKY ? L->slope : 1.f;
    a.by_taps.set(a.taps); a.by_Fw.set(a.Fw); a.by_segs.set(a.segs); a.by_Ho.set(a.Ho);
    if (a.C < CB)
    {
        a.by_segs.set(a.Wo);
        const dim3 grid((unsigned)(((long long)a.N * a.Ho * a.Wo * 4 + 255) / 256), (unsigned)(a.K / CB));
        const bool f3 = a.Fh == 3 && a.Fw == 3;
#define SB_FIRST(CI) (f3 ? conv_first_small_f32_kernel<CI, 3> : conv_first_small_f32_kernel<CI, 0>)<<<grid, 256, 0, st>>>(a, in, filt, bias, out)
        if (a.C == 3)
            SB_FIRST(3);
        else if (a.C == 2)
            SB_FIRST(2);
        else
            SB_FIRST(1);
#undef SB_FIRST
        return launched("conv_first_small_f32_kernel");
    }
    conv_small_f32_kernel<<<dim3((unsigned)(a.N * a.Ho * a.segs), (unsigned)(a.K / CB)), WARPS * 32, 0, st>>>(a, in, filt, bias, out);
    return launched("conv_small_f32_kernel");
}
} // namespace sb

extern "C"
{
int small_b200_conv2d_f32_small_preferred(const small_b200_layer *L) { return L && conv_small_preferred(L) ? 1 : 0; }

int small_b200_conv2d_f32_small(const small_b200_layer *L, const float *in, const float *filt, const float *bias, float *out, void *stream)
{
    if (int rc = check_window_layer(L, "Conv2D<float>", true, 2))
        return rc;
    if (!conv_small_preferred(L))
        return small_b200_conv2d_f32(L, in, filt, bias, out, stream);
    if (out_dim(L->H, L->pad_t, L->pad_b, L->Fh, row_stride(L)) == 0 || out_dim(L->W, L->pad_l, L->pad_r, L->Fw, L->stride) == 0)
        return SMALL_B200_OK;
    return conv_small_f32(L, in, filt, bias, out, as_stream(stream));
}

int small_b200_avgpool_dense_f32_supported(const small_b200_layer *pool, const small_b200_layer *dense)
{
    return tail_covered(pool, dense) ? 1 : 0;
}

int small_b200_avgpool_dense_f32(const small_b200_layer *pool, const small_b200_layer *dense, int32_t softmax, const float *in,
                                 const float *filt, const float *bias, float *out, void *stream)
{
    if (!tail_covered(pool, dense))
        return fail(SMALL_B200_INVALID_ARGUMENT, "AveragePool2D+Dense<float> ERROR: shapes not covered by the one-kernel form.");
    if (pool->N == 0)
        return SMALL_B200_OK;
    const int hw = pool->H * pool->W;
    const float ns = dense->act == SMALL_B200_ACT_RELU ? 0.f : dense->act == SMALL_B200_ACT_LEAKY ? dense->slope : 1.f;
    const size_t smem = ((size_t)pool->C + 16 * (size_t)dense->K) * sizeof(float);
    pool_dense_softmax_f32_kernel<<<(unsigned)pool->N, TAIL_THREADS, smem, as_stream(stream)>>>(
        pool->C, hw, (float)(1.0 / hw), dense->K, softmax, ns, in, filt, bias, out);
    return launched("pool_dense_softmax_f32_kernel");
}
} // extern "C"
