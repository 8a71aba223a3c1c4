// quint8.cu -- the uint8 layers on the CUDA cores: dense convolution (general shapes),
// depthwise convolution, max / average pooling and ReLU, each followed by the
// reference's fixed-point requantisation.  Replaces
// small::quint8_detail::abstract_layer (include/small/q_abstract_layer.hpp:884-1571) and the
// QUINT8_{CONV,DW,MAX}_TILE_C / QUINT8_QUANTIZE_TILE_C microkernels
// (platforms/reference/intrinsics_quint8.h:191-289, :481-531).
//
// Arithmetic (bit-exact with the reference): zero points are ADDED, padded taps are
// SKIPPED (they contribute nothing, not even zero_in * w), accumulation is int32 and stays
// in registers for the whole reduction -- the reference parks partial sums in the output
// buffer between input-channel blocks (q_abstract_layer.hpp:1144), which is why its
// callers over-allocate outputs four times; nothing of that is needed here.
#include "common.cuh"
#include "tc_common.cuh"

#include <algorithm>

namespace
{
using namespace sb;

struct QArgs
{
    int N, C, K, H, W, Ho, Wo, Fh, Fw, stride, pad_t, pad_l;
    int cib, cbs;
    int zero_in, zero_filt, lshift, rshift, mult, k_zero;
};

__device__ __forceinline__ int byte_of(const uint4 &v, int i)
{
    const unsigned w = (i < 4) ? v.x : (i < 8) ? v.y : (i < 12) ? v.z : v.w;
    return (int)((w >> (8 * (i & 3))) & 0xffu);
}

__device__ __forceinline__ uint4 pack16(const int *v)
{
    uint4 o;
    o.x = (unsigned)v[0] | ((unsigned)v[1] << 8) | ((unsigned)v[2] << 16) | ((unsigned)v[3] << 24);
    o.y = (unsigned)v[4] | ((unsigned)v[5] << 8) | ((unsigned)v[6] << 16) | ((unsigned)v[7] << 24);
    o.z = (unsigned)v[8] | ((unsigned)v[9] << 8) | ((unsigned)v[10] << 16) | ((unsigned)v[11] << 24);
    o.w = (unsigned)v[12] | ((unsigned)v[13] << 8) | ((unsigned)v[14] << 16) | ((unsigned)v[15] << 24);
    return o;
}

// Dense convolution, one thread per output pixel and block of 16 output channels.
// All threads of a CTA share the output-channel block, so filter reads are warp-uniform
// 16-byte loads served by L1.
// PARTIAL (the reference's int32 partial-sum form, one image and one block of output channels): the
// accumulators start from the int32 values the output buffer holds, [pixel][16], and go back there as
// int32; requant_in_place_kernel turns them into bytes afterwards.
template <bool PARTIAL>
__global__ void __launch_bounds__(128)
conv2d_u8_direct_kernel(const QArgs a, const uint8_t *__restrict__ in, const uint8_t *__restrict__ filt,
                        const int32_t *__restrict__ bias, uint8_t *out)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int kb = blockIdx.y, n = blockIdx.z;
    if (p >= a.Ho * a.Wo)
        return;
    const int oh = p / a.Wo, ow = p - oh * a.Wo;
    int acc[CB];
    if (PARTIAL)
    {
        const int4 *seed = reinterpret_cast<const int4 *>(out) + (size_t)p * 4;
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4)
        {
            const int4 v = seed[k4];
            acc[4 * k4] = v.x; acc[4 * k4 + 1] = v.y; acc[4 * k4 + 2] = v.z; acc[4 * k4 + 3] = v.w;
        }
    }
    else
    {
#pragma unroll
        for (int k = 0; k < CB; ++k)
            acc[k] = a.k_zero + (bias ? bias[kb * CB + k] : 0);
    }
    const int taps = a.Fh * a.Fw;
    const uint8_t *img = in + (size_t)n * a.C * a.H * a.W;
    const uint8_t *fk = filt + (size_t)kb * a.cbs * taps * a.cib * CB;
    for (int cb = 0; cb < a.cbs; ++cb)
    {
        const uint8_t *plane = img + (size_t)cb * a.H * a.W * a.cib;
        const uint8_t *fcb = fk + (size_t)cb * taps * a.cib * CB;
        for (int kh = 0; kh < a.Fh; ++kh)
        {
            const int ih = oh * a.stride - a.pad_t + kh;
            if (ih < 0 || ih >= a.H)
                continue;
            for (int kw = 0; kw < a.Fw; ++kw)
            {
                const int iw = ow * a.stride - a.pad_l + kw;
                if (iw < 0 || iw >= a.W)
                    continue;
                const uint8_t *px = plane + ((size_t)ih * a.W + iw) * a.cib;
                const uint4 *fw = reinterpret_cast<const uint4 *>(fcb + (size_t)(kh * a.Fw + kw) * a.cib * CB);
                if (a.cib == CB)
                {
                    const uint4 av = *reinterpret_cast<const uint4 *>(px);
#pragma unroll
                    for (int c = 0; c < CB; ++c)
                    {
                        const int x = byte_of(av, c) + a.zero_in;
                        const uint4 wv = __ldg(fw + c);
#pragma unroll
                        for (int k = 0; k < CB; ++k)
                            acc[k] += x * (byte_of(wv, k) + a.zero_filt);
                    }
                }
                else
                {
                    for (int c = 0; c < a.cib; ++c)
                    {
                        const int x = (int)px[c] + a.zero_in;
                        const uint4 wv = __ldg(fw + c);
#pragma unroll
                        for (int k = 0; k < CB; ++k)
                            acc[k] += x * (byte_of(wv, k) + a.zero_filt);
                    }
                }
            }
        }
    }
    if (PARTIAL)
    {
        int4 *dst = reinterpret_cast<int4 *>(out) + (size_t)p * 4;
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4)
            dst[k4] = make_int4(acc[4 * k4], acc[4 * k4 + 1], acc[4 * k4 + 2], acc[4 * k4 + 3]);
        return;
    }
    *reinterpret_cast<uint4 *>(out + (((size_t)n * (a.K / CB) + kb) * a.Ho * a.Wo + p) * CB) =
        requant_pack16(acc, a.lshift, a.rshift, a.mult);
}

// The int32 accumulators [pixels][16] at the start of a buffer become the bytes [pixels][16] at the start
// of the same buffer.  Pixel p's bytes land on the accumulators of pixel p / 4, so the pass runs as ONE
// CTA that walks the pixels in order, a block of 1024 at a time: read, barrier, write, barrier -- every
// accumulator is read before anything is written over it, as in the reference's sequential loop nest.
__global__ void __launch_bounds__(1024) requant_in_place_kernel(int pixels, const QArgs a, uint8_t *buf)
{
    for (int base = 0; base < pixels; base += 1024)
    {
        const int p = base + (int)threadIdx.x;
        int acc[CB];
        if (p < pixels)
        {
            const int4 *src = reinterpret_cast<const int4 *>(buf) + (size_t)p * 4;
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4)
            {
                const int4 v = src[k4];
                acc[4 * k4] = v.x; acc[4 * k4 + 1] = v.y; acc[4 * k4 + 2] = v.z; acc[4 * k4 + 3] = v.w;
            }
        }
        __syncthreads();
        if (p < pixels)
            *reinterpret_cast<uint4 *>(buf + (size_t)p * CB) = requant_pack16(acc, a.lshift, a.rshift, a.mult);
        __syncthreads();
    }
}

// OP: 0 depthwise conv, 1 max pool, 2 average pool; one thread per output pixel and block
// of 16 channels (one 128-bit load per tap, one 128-bit store).
template <int OP, bool PARTIAL = false>
__global__ void __launch_bounds__(256)
window_u8_kernel(const QArgs a, const uint8_t *__restrict__ in, const uint8_t *__restrict__ filt,
                 const int32_t *__restrict__ bias, uint8_t *out)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)a.N * (a.C / CB) * a.Ho * a.Wo;
    if (i >= total)
        return;
    const long long o = i;
    const int ow = (int)(i % a.Wo); i /= a.Wo;
    const int oh = (int)(i % a.Ho); i /= a.Ho; // i = n*(C/16)+cb
    const int cb = (int)(i % (a.C / CB));
    const uint8_t *plane = in + (size_t)i * a.H * a.W * CB;
    const int h0 = oh * a.stride - a.pad_t, w0 = ow * a.stride - a.pad_l;
    int acc[CB];
#pragma unroll
    for (int k = 0; k < CB; ++k)
        acc[k] = a.k_zero + ((OP == 0 && bias) ? bias[cb * CB + k] : 0);
    if (PARTIAL) // one image, one channel block: o is the pixel
    {
        const int4 *seed = reinterpret_cast<const int4 *>(out) + (size_t)o * 4;
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4)
        {
            const int4 v = seed[k4];
            acc[4 * k4] = v.x; acc[4 * k4 + 1] = v.y; acc[4 * k4 + 2] = v.z; acc[4 * k4 + 3] = v.w;
        }
    }
    if (OP == 1)
    {
        // q_abstract_layer.hpp:277-288: interior tiles are seeded with the RAW first tap
        const bool interior = h0 >= 0 && w0 >= 0 && h0 + a.Fh <= a.H && w0 + a.Fw <= a.W;
        if (interior)
        {
            const uint4 v = *reinterpret_cast<const uint4 *>(plane + ((size_t)h0 * a.W + w0) * CB);
#pragma unroll
            for (int k = 0; k < CB; ++k)
                acc[k] = byte_of(v, k);
        }
    }
    for (int kh = 0; kh < a.Fh; ++kh)
    {
        const int ih = h0 + kh;
        if (ih < 0 || ih >= a.H)
            continue;
        for (int kw = 0; kw < a.Fw; ++kw)
        {
            const int iw = w0 + kw;
            if (iw < 0 || iw >= a.W)
                continue;
            const uint4 v = *reinterpret_cast<const uint4 *>(plane + ((size_t)ih * a.W + iw) * CB);
            if (OP == 0)
            {
                const uint4 f = __ldg(reinterpret_cast<const uint4 *>(
                    filt + (((size_t)cb * a.Fh + kh) * a.Fw + kw) * CB));
#pragma unroll
                for (int k = 0; k < CB; ++k)
                    acc[k] += (byte_of(v, k) + a.zero_in) * (byte_of(f, k) + a.zero_filt);
            }
            else if (OP == 1)
            {
#pragma unroll
                for (int k = 0; k < CB; ++k)
                {
                    const int x = byte_of(v, k) + a.zero_in;
                    acc[k] = x > acc[k] ? x : acc[k];
                }
            }
            else
            {
#pragma unroll
                for (int k = 0; k < CB; ++k)
                    acc[k] += byte_of(v, k) + a.zero_in;
            }
        }
    }
    if (PARTIAL)
    {
        int4 *dst = reinterpret_cast<int4 *>(out) + (size_t)o * 4;
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4)
            dst[k4] = make_int4(acc[4 * k4], acc[4 * k4 + 1], acc[4 * k4 + 2], acc[4 * k4 + 3]);
        return;
    }
    *reinterpret_cast<uint4 *>(out + o * CB) = requant_pack16(acc, a.lshift, a.rshift, a.mult);
}


// ---------------------------------------------------------------------------------------------
// Fast paths for the quantisation every configuration here uses: filter zero point -128 (the
// reference ADDS offsets, so w + zero_filt is a signed byte) and input zero point 0 or -128
// (a + zero_in is an unsigned or a signed byte).  The products then fit dp4a, four per
// instruction.  Padded taps must contribute nothing: their shifted activation is 0.
__device__ __forceinline__ int dp4a_us(unsigned a, unsigned b, int c) // unsigned a bytes x signed b bytes
{
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
template <bool SIGNED_IN>
__device__ __forceinline__ int dp4a_in(unsigned a, unsigned b, int c)
{
    return SIGNED_IN ? __dp4a((int)a, (int)b, c) : dp4a_us(a, b, c);
}

// 4 x 4 byte transpose: r[t] holds 4 channels of tap t; c[j] gets the 4 taps of channel j
__device__ __forceinline__ void transpose4x4(const unsigned r0, const unsigned r1, const unsigned r2,
                                             const unsigned r3, unsigned *c)
{
    const unsigned t0 = __byte_perm(r0, r1, 0x5140), t1 = __byte_perm(r2, r3, 0x5140);
    const unsigned t2 = __byte_perm(r0, r1, 0x7362), t3 = __byte_perm(r2, r3, 0x7362);
    c[0] = __byte_perm(t0, t1, 0x5410); c[1] = __byte_perm(t0, t1, 0x7632);
    c[2] = __byte_perm(t2, t3, 0x5410); c[3] = __byte_perm(t2, t3, 0x7632);
}

// Depthwise convolution: one thread per output pixel and block of 16 channels.  A depthwise sum
// runs over TAPS of one channel while the packed layout keeps CHANNELS of one pixel together, so
// the taps are taken four at a time and byte-transposed (8 PRMT per 4 x 4) into dp4a operands;
// the filter is transposed once per CTA into shared memory as signed bytes.
// QUADS > 0: the number of tap groups is known at compile time and every tap is loaded before
// the arithmetic starts (one round trip to memory instead of one per group).
template <bool SIGNED_IN, int QUADS>
__global__ void __launch_bounds__(256)
dwconv_u8_dp4a_kernel(const QArgs a, const uint8_t *__restrict__ in, const uint8_t *__restrict__ filt,
                      const int32_t *__restrict__ bias, uint8_t *__restrict__ out)
{
    extern __shared__ __align__(16) unsigned sw[]; // [cb][quad][16 ch]: (w ^ 0x80) of 4 taps; then tap -> (kh, kw)
    const int taps = a.Fh * a.Fw, quads = QUADS > 0 ? QUADS : (taps + 3) / 4, cbs = a.C / CB;
    short2 *tap_pos = reinterpret_cast<short2 *>(sw + cbs * quads * CB);
    for (int i = threadIdx.x; i < cbs * quads * CB; i += blockDim.x)
    {
        const int ch = i % CB, q = (i / CB) % quads, cb = i / (CB * quads);
        unsigned wv = 0;
        for (int t = 0; t < 4; ++t)
        {
            const int tap = 4 * q + t;
            if (tap < taps)
                wv |= (unsigned)(filt[((size_t)cb * taps + tap) * CB + ch] ^ 0x80u) << (8 * t);
        }
        sw[i] = wv; // a missing tap keeps weight 0
    }
    for (int i = threadIdx.x; i < quads * 4; i += blockDim.x)
        tap_pos[i] = i < taps ? make_short2((short)(i / a.Fw), (short)(i % a.Fw)) : make_short2(-30000, -30000);
    __syncthreads();

    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)a.N * cbs * a.Ho * a.Wo;
    if (i >= total)
        return;
    const long long o = i;
    const int ow = (int)(i % a.Wo); i /= a.Wo;
    const int oh = (int)(i % a.Ho); i /= a.Ho; // i = n*(C/16)+cb
    const int cb = (int)(i % cbs);
    const uint8_t *plane = in + (size_t)i * a.H * a.W * CB;
    const int h0 = oh * a.stride - a.pad_t, w0 = ow * a.stride - a.pad_l;
    int acc[CB];
#pragma unroll
    for (int k = 0; k < CB; ++k)
        acc[k] = a.k_zero + (bias ? bias[cb * CB + k] : 0);
    const uint4 *wq = reinterpret_cast<const uint4 *>(sw + (size_t)cb * quads * CB);
    if (QUADS > 0)
    {
        uint4 v[QUADS > 0 ? QUADS * 4 : 1];
#pragma unroll
        for (int t = 0; t < QUADS * 4; ++t)
        {
            const short2 pos = tap_pos[t];
            const int ih = h0 + pos.x, iw = w0 + pos.y;
            v[t] = make_uint4(0u, 0u, 0u, 0u);
            if (pos.x >= 0 && ih >= 0 && ih < a.H && iw >= 0 && iw < a.W)
            {
                v[t] = *reinterpret_cast<const uint4 *>(plane + ((size_t)ih * a.W + iw) * CB);
                if (SIGNED_IN)
                {
                    v[t].x ^= 0x80808080u; v[t].y ^= 0x80808080u; v[t].z ^= 0x80808080u; v[t].w ^= 0x80808080u;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < QUADS; ++q)
        {
#pragma unroll
            for (int g = 0; g < 4; ++g)
            {
                unsigned c[4];
                const unsigned r0 = g == 0 ? v[4 * q].x : g == 1 ? v[4 * q].y : g == 2 ? v[4 * q].z : v[4 * q].w;
                const unsigned r1 = g == 0 ? v[4 * q + 1].x : g == 1 ? v[4 * q + 1].y : g == 2 ? v[4 * q + 1].z : v[4 * q + 1].w;
                const unsigned r2 = g == 0 ? v[4 * q + 2].x : g == 1 ? v[4 * q + 2].y : g == 2 ? v[4 * q + 2].z : v[4 * q + 2].w;
                const unsigned r3 = g == 0 ? v[4 * q + 3].x : g == 1 ? v[4 * q + 3].y : g == 2 ? v[4 * q + 3].z : v[4 * q + 3].w;
                transpose4x4(r0, r1, r2, r3, c);
                const uint4 w4 = wq[q * 4 + g];
                acc[4 * g + 0] = dp4a_in<SIGNED_IN>(c[0], w4.x, acc[4 * g + 0]);
                acc[4 * g + 1] = dp4a_in<SIGNED_IN>(c[1], w4.y, acc[4 * g + 1]);
                acc[4 * g + 2] = dp4a_in<SIGNED_IN>(c[2], w4.z, acc[4 * g + 2]);
                acc[4 * g + 3] = dp4a_in<SIGNED_IN>(c[3], w4.w, acc[4 * g + 3]);
            }
        }
    }
    else
    for (int q = 0; q < quads; ++q)
    {
        unsigned r[4][4];
#pragma unroll
        for (int t = 0; t < 4; ++t)
        {
            const short2 pos = tap_pos[4 * q + t];
            const int ih = h0 + pos.x, iw = w0 + pos.y;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (pos.x >= 0 && ih >= 0 && ih < a.H && iw >= 0 && iw < a.W)
            {
                v = *reinterpret_cast<const uint4 *>(plane + ((size_t)ih * a.W + iw) * CB);
                if (SIGNED_IN)
                {
                    v.x ^= 0x80808080u; v.y ^= 0x80808080u; v.z ^= 0x80808080u; v.w ^= 0x80808080u;
                }
            }
            r[t][0] = v.x; r[t][1] = v.y; r[t][2] = v.z; r[t][3] = v.w;
        }
#pragma unroll
        for (int g = 0; g < 4; ++g)
        {
            unsigned c[4];
            transpose4x4(r[0][g], r[1][g], r[2][g], r[3][g], c);
            const uint4 w4 = wq[q * 4 + g];
            acc[4 * g + 0] = dp4a_in<SIGNED_IN>(c[0], w4.x, acc[4 * g + 0]);
            acc[4 * g + 1] = dp4a_in<SIGNED_IN>(c[1], w4.y, acc[4 * g + 1]);
            acc[4 * g + 2] = dp4a_in<SIGNED_IN>(c[2], w4.z, acc[4 * g + 2]);
            acc[4 * g + 3] = dp4a_in<SIGNED_IN>(c[3], w4.w, acc[4 * g + 3]);
        }
    }
    *reinterpret_cast<uint4 *>(out + o * CB) = requant_pack16(acc, a.lshift, a.rshift, a.mult);
}

// Depthwise 3x3, stride 1, through shared memory.  A tile is whole planes (an image's channel block) where they are small,
// else a run of rows of one plane, or of pieces of its rows where two whole rows don't fit (COLS); CTAs are persistent and fetch the next tile before they compute one.  Pixels are copied 16
// bytes a thread (a bulk copy a row took some 50 cycles each, more than all else for rows of 3 or 6 pixels) into a pitch
// that has room for the padding, which holds the byte -zero_in, whose contribution (a + zero_in) * w is nothing: every tap is
// inside.  A thread computes 2 rows x TW pixels of 4 channels.  The four rows a kernel column covers for the two output
// rows are byte-transposed once; against the filter column (w0, w1, w2, 0) they give the upper output, against
// (0, w0, w1, w2) the lower one, so that a transpose of 8 permutes serves up to 24 sums of products.  Filter bytes are
// signed, w' = w - 128, and the input stays unsigned:
//   sum (a + zI)(w + zF) = sum a w' + (128 + zF) sum a + zI sum (w + zF)
// with the last term in the seed of the requantisation and the second one (SUM_A: another three dp4a a column) only
// where zF != -128.  The output goes back through shared memory as one bulk copy.
// What bounds it: instructions (three dp4a, two or three of transposes and loads, four and a half of requantisation per output
// byte): 62 % of the issue slots and 42 % of the ALU at 256 images of 48x48.  Reading strips of a row straight from global memory, 96 bytes apart from lane to lane,
// was bound by L1 wavefronts, with twice the transposes.  2048 images, us before -> now: 16 channels at 48x48 102 -> 70, 32 at
// 24x24 52 -> 36, 64 at 12x12 29 -> 22, 128 at 6x6 16.5 -> 13.6, 256 at 3x3 9.2 -> 10.9 (half the rows of its last pairs
// are nothing); a whole MobileNet's 13 layers 330 -> 285.
// Pieces of rows (from a width of some 380 on; the layer ran one pixel a thread, dwconv_u8_dp4a_kernel, at zero points that kernel
// takes, else tap by tap), 16 channels, us: 416x416, 64 images 367 -> 159, 1080x1920, 8 images 545 -> 241; at zero points
// -113 / -121 477 -> 200 and 710 -> 280.  A row's output is a bulk copy of its own, by a lane of its own.
// TW is odd: eight strips, TW * 16 bytes apart, times four quarters of a pixel then touch all 32 banks.
constexpr int DW_THREADS = 256;
struct DwTile
{
    int N, cbs, H, W, Ho, Wo, pad_t, pad_l;
    int planes;    // planes per tile (more than one only when a tile covers all rows)
    int rows, row_tiles; // output rows per tile (even, or all of them), tiles down a plane
    int strips, pairs, pitch, in_rows; // pitch and in_rows in pixels and rows of shared memory
    int cols, col_tiles; // output columns per tile (COLS: a row is cut into several)
    int zero_in, sum_a;  // sum_a: 128 + zero_filt
    int lshift, rshift, mult, k_zero;
    int tiles;
    unsigned in_bytes, out_bytes, out_at, w_at; // bytes of a stage; offsets
    FastDiv by_row_tiles, by_col_tiles, by_cbs, by_strips, by_pairs, by_pitch, by_in_rows, by_copy_rows, by_W;
};

template <int TW, bool SUM_A, bool COLS>
__global__ void __launch_bounds__(DW_THREADS, 3)
dwconv3x3_u8_tile_kernel(const DwTile a, const uint8_t *__restrict__ in, const uint8_t *__restrict__ filt,
                         const int32_t *__restrict__ bias, uint8_t *__restrict__ out)
{
    extern __shared__ __align__(128) uint8_t smem[]; // [stage][plane][in_rows][pitch][16], [stage][plane][rows][Wo][16], filter
    const int tid = threadIdx.x, first = blockIdx.x, step = gridDim.x;
    // padding: columns, and the rows that are padding in every tile, once for both stages
    const unsigned pad = (unsigned)(-a.zero_in & 255) * 0x01010101u;
    const bool whole = !COLS && a.row_tiles == 1;
    for (int st = 0; !COLS && st < 2 && first + st * step < a.tiles; ++st)
        for (int i = tid; i < a.planes * a.in_rows * a.pitch; i += DW_THREADS)
        {
            const int lr = a.by_pitch.div(i), x = i - lr * a.pitch - a.pad_l, r = lr - a.by_in_rows.div(lr) * a.in_rows - a.pad_t;
            if (x < 0 || x >= a.W || (whole && (r < 0 || r >= a.H)))
                *reinterpret_cast<uint4 *>(smem + st * a.in_bytes + (size_t)i * CB) = make_uint4(pad, pad, pad, pad);
        }
    // per channel block [kw][16] words (w0, w1, w2, 0), then [16] seeds
    unsigned *words = reinterpret_cast<unsigned *>(smem + a.w_at);
    for (int i = tid; i < a.cbs * CB; i += DW_THREADS)
    {
        const int cb = i >> 4, ch = i & 15;
        const uint8_t *w = filt + (size_t)cb * 9 * CB + ch;
        int sum = 0;
#pragma unroll
        for (int kw = 0; kw < 3; ++kw)
        {
            unsigned v = 0;
#pragma unroll
            for (int kh = 0; kh < 3; ++kh)
            {
                const int b = w[(kh * 3 + kw) * CB];
                sum += b - 128 + a.sum_a;
                v |= (unsigned)(b ^ 0x80) << (8 * kh);
            }
            words[(cb * 4 + kw) * CB + ch] = v;
        }
        words[(cb * 4 + 3) * CB + ch] = (unsigned)(a.k_zero + (bias ? bias[cb * CB + ch] : 0) + a.zero_in * sum);
    }
    // Where a tile lies: its first plane, how many, its first output row and column.
    struct Place { int plane0, planes, oh0, ow0; };
    auto place = [&](int tile) {
        const int t = COLS ? a.by_col_tiles.div(tile) : tile, unit = a.by_row_tiles.div(t);
        return Place{unit * a.planes, min(a.planes, a.N * a.cbs - unit * a.planes), (t - unit * a.row_tiles) * a.rows,
                     COLS ? (tile - t * a.col_tiles) * a.cols : 0};
    };
    // A tile's rows: copies of those of the image; rows that are padding (in runs of rows only) are written.
    auto fetch = [&](int tile, int st) {
        const Place p = place(tile);
        const int plane0 = p.plane0, planes = p.planes, top = p.oh0 - a.pad_t;
        if (COLS) // padding on any side: a byte of its own for every pixel outside
        {
            const int left = p.ow0 - a.pad_l;
            const uint8_t *from = in + ((size_t)plane0 * a.H * a.W + left) * CB;
            for (int i = tid; i < a.in_rows * a.pitch; i += DW_THREADS)
            {
                const int lr = a.by_pitch.div(i), x = i - lr * a.pitch, r = lr + top;
                uint8_t *at = smem + st * a.in_bytes + (size_t)i * CB;
                if ((unsigned)r < (unsigned)a.H && (unsigned)(x + left) < (unsigned)a.W)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(at)), "l"(from + ((long long)r * a.W + x) * CB) : "memory");
                else
                    *reinterpret_cast<uint4 *>(at) = make_uint4(pad, pad, pad, pad);
            }
            return;
        }
        const int r_lo = max(top, 0), r_hi = min(top + a.in_rows, a.H), count = max(r_hi - r_lo, 0);
        uint8_t *stage = smem + st * a.in_bytes;
        const uint32_t to = smem_u32(stage) + (uint32_t)(((r_lo - top) * a.pitch + a.pad_l) * CB);
        const uint8_t *from = in + ((size_t)plane0 * a.H + r_lo) * a.W * CB;
        for (int i = tid; i < planes * count * a.W; i += DW_THREADS)
        {
            const int row = a.by_W.div(i), pl = whole ? a.by_copy_rows.div(row) : 0, r = row - pl * count;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + (uint32_t)(((pl * a.in_rows + r) * a.pitch + i - row * a.W) * CB)),
                         "l"(from + (size_t)(pl * (a.H - count) * a.W + i) * CB)
                         : "memory");
        }
        if (!whole && count < a.in_rows)
            for (int i = tid; i < a.in_rows * a.pitch; i += DW_THREADS)
            {
                const int r = a.by_pitch.div(i) + top;
                if (r < r_lo || r >= r_hi)
                    *reinterpret_cast<uint4 *>(stage + (size_t)i * CB) = make_uint4(pad, pad, pad, pad);
            }
    };
    // By the storing threads, after all of them have fenced and met: one copy, or (COLS) one for each row.
    const bool storer = COLS ? tid < a.rows : tid == 0;
    auto store = [&](int tile, int st) {
        const Place p = place(tile);
        const int rows = min(a.rows, a.Ho - p.oh0);
        if (COLS && tid >= rows)
            return;
        const int r = COLS ? tid : 0;
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(out + (((size_t)p.plane0 * a.Ho + p.oh0 + r) * a.Wo + p.ow0) * CB),
                     "r"(smem_u32(smem + a.out_at + st * a.out_bytes) + (unsigned)(r * a.cols * CB)),
                     "r"((unsigned)(COLS ? min(a.cols, a.Wo - p.ow0) * CB : p.planes * rows * a.Wo * CB))
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    };
    __syncthreads();
    fetch(first, 0);
    const bool fast = requant_is_fast(a.lshift, a.rshift, a.mult);
    const int per_plane = a.pairs * a.strips;
    int st = 0;
    for (int tile = first; tile < a.tiles; tile += step)
    {
        // One meeting per tile: this tile's copies have landed, everyone is through with the tile before it (its output can
        // go, its stage be filled again), and the output before that one has been read.
        asm volatile("cp.async.wait_all;" ::: "memory");
        fence_proxy_async();
        if (storer)
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncthreads();
        if (storer && tile != first)
            store(tile - step, st ^ 1);
        if (tile + step < a.tiles)
            fetch(tile + step, st ^ 1);
        const Place p = place(tile);
        const int plane0 = p.plane0, planes = p.planes, rows = min(a.rows, a.Ho - p.oh0);
        const int pitch_out = COLS ? a.cols : a.Wo, cols = COLS ? min(a.cols, a.Wo - p.ow0) : a.Wo;
        const uint8_t *sI = smem + st * a.in_bytes;
        uint8_t *sO = smem + a.out_at + st * a.out_bytes;
        for (int i = tid; i < planes * per_plane * 4; i += DW_THREADS)
        {
            const int q = i & 3, row = a.by_strips.div(i >> 2), strip = (i >> 2) - row * a.strips, pl = a.by_pairs.div(row);
            const int r = 2 * (row - pl * a.pairs), ow0 = strip * TW;
            const unsigned *src = reinterpret_cast<const unsigned *>(sI + ((size_t)(pl * a.in_rows + r) * a.pitch + ow0) * CB) + q;
            const int cb = plane0 + pl - a.by_cbs.div(plane0 + pl) * a.cbs;
            const uint4 *wp = reinterpret_cast<const uint4 *>(words + cb * 4 * CB) + q;
            unsigned w[3][4];
#pragma unroll
            for (int kw = 0; kw < 3; ++kw)
            {
                const uint4 v = wp[kw * 4];
                w[kw][0] = v.x; w[kw][1] = v.y; w[kw][2] = v.z; w[kw][3] = v.w;
            }
            const uint4 sv = wp[12];
            const int seed[4] = {(int)sv.x, (int)sv.y, (int)sv.z, (int)sv.w};
            int acc[2][TW][4];
            int asum[2][SUM_A ? TW : 1][4];
#pragma unroll
            for (int o = 0; o < TW; ++o)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                {
                    acc[0][o][j] = acc[1][o][j] = 0;
                    if (SUM_A)
                        asum[0][o][j] = asum[1][o][j] = 0;
                }
#pragma unroll
            for (int x = 0; x < TW + 2; ++x)
            {
                unsigned c[4];
                transpose4x4(src[x * 4], src[(a.pitch + x) * 4], src[(2 * a.pitch + x) * 4], src[(3 * a.pitch + x) * 4], c);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                {
#pragma unroll
                    for (int kw = 0; kw < 3; ++kw)
                        if (x - kw >= 0 && x - kw < TW)
                        {
                            acc[0][x - kw][j] = dp4a_us(c[j], w[kw][j], acc[0][x - kw][j]);
                            acc[1][x - kw][j] = dp4a_us(c[j], w[kw][j] << 8, acc[1][x - kw][j]);
                            if (SUM_A)
                            {
                                asum[0][x - kw][j] = dp4a_us(c[j], 0x00010101u, asum[0][x - kw][j]);
                                asum[1][x - kw][j] = dp4a_us(c[j], 0x01010100u, asum[1][x - kw][j]);
                            }
                        }
                }
            }
            if (SUM_A)
#pragma unroll
                for (int o = 0; o < TW; ++o)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                    {
                        acc[0][o][j] += a.sum_a * asum[0][o][j];
                        acc[1][o][j] += a.sum_a * asum[1][o][j];
                    }
            long long seeds[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                seeds[j] = requant_seed(seed[j], a.mult);
            unsigned *dst = reinterpret_cast<unsigned *>(sO + ((size_t)(pl * a.rows + r) * pitch_out + ow0) * CB) + q;
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int o = 0; o < TW; ++o)
                    if (ow0 + o < cols && r + h < rows)
                    {
                        unsigned v;
                        if (fast)
                        {
                            const int bit = 1 << (a.rshift - 2), sh1 = a.rshift - 1;
                            v = pack4_sat(requant_seeded_raw(acc[h][o][0], a.mult, seeds[0], bit, sh1),
                                          requant_seeded_raw(acc[h][o][1], a.mult, seeds[1], bit, sh1),
                                          requant_seeded_raw(acc[h][o][2], a.mult, seeds[2], bit, sh1),
                                          requant_seeded_raw(acc[h][o][3], a.mult, seeds[3], bit, sh1));
                        }
                        else
                            v = requant_pack4_general(acc[h][o][0] + seed[0], acc[h][o][1] + seed[1], acc[h][o][2] + seed[2],
                                                      acc[h][o][3] + seed[3], a.lshift, a.rshift, a.mult);
                        dst[(h * pitch_out + o) * 4] = v;
                    }
        }
        st ^= 1;
    }
    fence_proxy_async();
    __syncthreads();
    if (storer)
    {
        store(first + (a.tiles - 1 - first) / step * step, st ^ 1);
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
}

// Dense convolution whose whole reduction is at most 32 bytes: a 1x1 layer on 16 or 32 channels, or a first layer (1..3
// channels, [H][W][C] image) whose window holds at most 32 values, e.g. 3x3 on 3 channels.  These are streaming layers
// with too little arithmetic for the tensor core to matter: what bounds them is the integer pipes (a dp4a for four products,
// four and a half instructions of requantisation per output byte), and before that shared memory, if every
// pixel fetches the filter for itself (64 four-byte broadcasts a pixel; 2.3 of the 3 cycles an output took).  So a thread makes
// PX pixels, 32 apart, and a 16-byte fetch of four channels' filter words feeds 4 * PX dp4a; one pixel a thread where
// there are not enough of them to fill the machine.  Two and not four: with 128 registers the gathers of eight warps a CTA had
// too little to hide behind (first layer 138 us against 100).  2048 images, us before -> now: 3x3 on 3 channels, stride 2
// at 96x96 113 -> 99 (225 -> 100 with padding on all sides); 16 -> 16 channels at 48x48 69 -> 57; 16 -> 32 at 24x24 49 -> 27
// (as an implicit GEMM before).
// Filter bytes are signed, w' = w - 128, the input stays unsigned, taps outside the image hold the byte -zero_in:
//   sum (a + zI)(w + zF) = sum a w' + (128 + zF) sum a + zI sum (w + zF)
// with the last term in the seed of the requantisation and the second one counted once per pixel.
struct OneArgs
{
    int total, H, W, Ho, Wo, C, K, Fh, Fw, R, stride, pad_t, pad_l;
    int zero_in, sum_a; // sum_a: 128 + zero_filt
    int lshift, rshift, mult, k_zero;
    long long in_bytes;
    FastDiv by_hw, by_Wo;
};
enum { ONE_1X1, ONE_333, ONE_FIRST };

// The reduction row of output pixel g: WORDS words of four bytes.
template <int WORDS, int KIND>
__device__ __forceinline__ void one_gather(const OneArgs &a, const uint8_t *__restrict__ in, int g, unsigned pad, unsigned (&x)[WORDS])
{
    const int n = a.by_hw.div(g), p = g - n * a.Ho * a.Wo, oh = a.by_Wo.div(p), ow = p - oh * a.Wo;
    const int ih0 = oh * a.stride - a.pad_t, iw0 = ow * a.stride - a.pad_l;
    if (KIND == ONE_1X1)
    {
        const bool inside = (unsigned)ih0 < (unsigned)a.H && (unsigned)iw0 < (unsigned)a.W;
        const uint8_t *src = in + (((size_t)n * (WORDS / 4) * a.H + ih0) * a.W + iw0) * CB;
#pragma unroll
        for (int cb = 0; cb < WORDS / 4; ++cb)
        {
            const uint4 v = inside ? __ldg(reinterpret_cast<const uint4 *>(src + (size_t)cb * a.H * a.W * CB)) : make_uint4(pad, pad, pad, pad);
            x[4 * cb] = v.x; x[4 * cb + 1] = v.y; x[4 * cb + 2] = v.z; x[4 * cb + 3] = v.w;
        }
        return;
    }
    if (KIND == ONE_333)
    {
        // A kernel row is 9 contiguous bytes: three aligned words and two funnel shifts; where the aligned words would pass an
        // end of the buffer, bytes.
        const uint8_t *row0 = in + ((long long)n * a.H + ih0) * a.W * 3 + iw0 * 3;
        const int vb = min(9, (a.W - iw0) * 3), skip = max(0, -iw0) * 3; // bytes of a row's run inside the image: [skip, vb)
        unsigned r0[3], r1[3], r2[3];
#pragma unroll
        for (int kh = 0; kh < 3; ++kh)
        {
            r0[kh] = r1[kh] = pad; r2[kh] = pad & 0xffu;
            if ((unsigned)(ih0 + kh) >= (unsigned)a.H)
                continue;
            const uint8_t *run = row0 + (long long)kh * a.W * 3;
            const uintptr_t base = reinterpret_cast<uintptr_t>(run) & ~(uintptr_t)3;
            if (base >= reinterpret_cast<uintptr_t>(in) && base + 12 <= reinterpret_cast<uintptr_t>(in) + (uintptr_t)a.in_bytes)
            {
                const unsigned *wp = reinterpret_cast<const unsigned *>(base);
                const unsigned sh = (unsigned)(reinterpret_cast<uintptr_t>(run) & 3) * 8;
                const unsigned w0 = __ldg(wp), w1 = __ldg(wp + 1), w2 = __ldg(wp + 2);
                r0[kh] = __funnelshift_r(w0, w1, sh);
                r1[kh] = __funnelshift_r(w1, w2, sh);
                r2[kh] = (w2 >> sh) & 0xffu;
                if (vb < 9 || skip > 0)
                {
#pragma unroll
                    for (int b = 0; b < 9; ++b)
                        if (b < skip || b >= vb)
                        {
                            unsigned &r = b < 4 ? r0[kh] : b < 8 ? r1[kh] : r2[kh];
                            const unsigned m = 0xffu << (8 * (b & 3));
                            r = (r & ~m) | (pad & m);
                        }
                }
            }
            else
            {
#pragma unroll
                for (int b = 0; b < 9; ++b)
                    if (b >= skip && b < vb)
                    {
                        unsigned &r = b < 4 ? r0[kh] : b < 8 ? r1[kh] : r2[kh];
                        const unsigned m = 0xffu << (8 * (b & 3));
                        r = (r & ~m) | (unsigned)run[b] << (8 * (b & 3));
                    }
            }
        }
        x[0] = r0[0]; x[1] = r1[0];
        x[2] = r2[0] | (r0[1] << 8);
        x[3] = (r0[1] >> 24) | (r1[1] << 8);
        x[4] = (r1[1] >> 24) | (r2[1] << 8) | (r0[2] << 16);
        x[5] = (r0[2] >> 16) | (r1[2] << 16);
        x[6] = (r1[2] >> 16) | (r2[2] << 16);
        return;
    }
    const uint8_t *img = in + (size_t)n * a.C * a.H * a.W;
    int kh = 0, kw = 0, c = 0;
#pragma unroll
    for (int j = 0; j < WORDS; ++j)
        x[j] = 0u;
#pragma unroll
    for (int r = 0; r < 4 * WORDS; ++r) // unrolled: x[] stays in registers
    {
        const int ih = ih0 + kh, iw = iw0 + kw;
        if (r < a.R)
        {
            const unsigned v = (unsigned)ih < (unsigned)a.H && (unsigned)iw < (unsigned)a.W ? img[((size_t)ih * a.W + iw) * a.C + c] : pad & 0xffu;
            x[r >> 2] |= v << (8 * (r & 3));
        }
        if (++c == a.C)
        {
            c = 0;
            if (++kw == a.Fw) { kw = 0; ++kh; }
        }
    }
}

template <int WORDS, int KIND, int PX>
__global__ void __launch_bounds__(256)
conv2d_u8_onestep_kernel(const OneArgs a, const uint8_t *__restrict__ in, const uint8_t *__restrict__ filt,
                         const int32_t *__restrict__ bias, uint8_t *__restrict__ out)
{
    extern __shared__ __align__(16) unsigned smem_u[]; // [K/4][WORDS + 1][4 k]: filter words, then the seeds
    for (int i = threadIdx.x; i < a.K; i += blockDim.x)
    {
        const uint8_t *w = filt + (size_t)(i / CB) * a.R * CB + (i % CB); // filter [K/16][R rows][16 k] for both layouts
        unsigned *row = smem_u + (size_t)(i / 4) * (WORDS + 1) * 4 + (i & 3);
        int sum = 0;
#pragma unroll
        for (int j = 0; j < WORDS; ++j)
        {
            unsigned wv = 0;
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (4 * j + t < a.R)
                {
                    const int b = w[(4 * j + t) * CB];
                    sum += b - 128 + a.sum_a;
                    wv |= (unsigned)(b ^ 0x80) << (8 * t);
                }
            row[j * 4] = wv;
        }
        row[WORDS * 4] = (unsigned)(a.k_zero + (bias ? bias[i] : 0) + a.zero_in * sum);
    }
    __syncthreads();
    const unsigned pad = (unsigned)(-a.zero_in & 255) * 0x01010101u;
    const int hw = a.Ho * a.Wo, kbs = a.K / CB, bit = 1 << max(a.rshift - 2, 0), sh1 = a.rshift - 1;
    const bool fast = requant_is_fast(a.lshift, a.rshift, a.mult);
    // a CTA keeps its copy of the filter for many pixels
    for (long long base = (long long)blockIdx.x * 256 * PX + (threadIdx.x >> 5) * 32 * PX + (threadIdx.x & 31); base < a.total;
         base += (long long)gridDim.x * 256 * PX)
    {
        const int g0 = (int)base;
        unsigned x[PX][WORDS];
        int sa[PX];
#pragma unroll
        for (int t = 0; t < PX; ++t)
            one_gather<WORDS, KIND>(a, in, min(g0 + 32 * t, a.total - 1), pad, x[t]);
#pragma unroll
        for (int t = 0; t < PX; ++t)
        {
            sa[t] = 0;
            if (a.sum_a)
            {
                unsigned s = 0;
#pragma unroll
                for (int j = 0; j < WORDS; ++j)
                    s = __dp4a(x[t][j], 0x01010101u, s);
                sa[t] = a.sum_a * (int)s;
            }
        }
        for (int kb = 0; kb < kbs; ++kb)
        {
            unsigned o[PX][4];
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4)
            {
                const uint4 *w4 = reinterpret_cast<const uint4 *>(smem_u) + (size_t)(kb * 4 + k4) * (WORDS + 1);
                int acc[PX][4];
#pragma unroll
                for (int t = 0; t < PX; ++t)
                    acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = sa[t];
#pragma unroll
                for (int j = 0; j < WORDS; ++j)
                {
                    const uint4 wv = w4[j];
#pragma unroll
                    for (int t = 0; t < PX; ++t)
                    {
                        acc[t][0] = dp4a_us(x[t][j], wv.x, acc[t][0]);
                        acc[t][1] = dp4a_us(x[t][j], wv.y, acc[t][1]);
                        acc[t][2] = dp4a_us(x[t][j], wv.z, acc[t][2]);
                        acc[t][3] = dp4a_us(x[t][j], wv.w, acc[t][3]);
                    }
                }
                const uint4 c = w4[WORDS];
                if (fast)
                {
                    const long long s0 = requant_seed((int)c.x, a.mult), s1 = requant_seed((int)c.y, a.mult),
                                    s2 = requant_seed((int)c.z, a.mult), s3 = requant_seed((int)c.w, a.mult);
#pragma unroll
                    for (int t = 0; t < PX; ++t)
                        o[t][k4] = pack4_sat(requant_seeded_raw(acc[t][0], a.mult, s0, bit, sh1), requant_seeded_raw(acc[t][1], a.mult, s1, bit, sh1),
                                             requant_seeded_raw(acc[t][2], a.mult, s2, bit, sh1), requant_seeded_raw(acc[t][3], a.mult, s3, bit, sh1));
                }
                else
#pragma unroll
                    for (int t = 0; t < PX; ++t)
                        o[t][k4] = requant_pack4_general(acc[t][0] + (int)c.x, acc[t][1] + (int)c.y, acc[t][2] + (int)c.z, acc[t][3] + (int)c.w,
                                                         a.lshift, a.rshift, a.mult);
            }
#pragma unroll
            for (int t = 0; t < PX; ++t)
            {
                const int g = g0 + 32 * t;
                if (g < a.total)
                {
                    const int n = a.by_hw.div(g);
                    *reinterpret_cast<uint4 *>(out + (((size_t)n * kbs + kb) * hw + (g - n * hw)) * CB) = make_uint4(o[t][0], o[t][1], o[t][2], o[t][3]);
                }
            }
        }
    }
}

// Dense convolution of a ONE-channel image (the first layer of the keyword-spotting network):
// the Fw taps of a kernel row are consecutive bytes of the image, so a row of the window is one
// (unaligned) 32-bit word per 4 taps and feeds dp4a directly.  A CTA takes IMGS images: it
// keeps them zero-padded in shared memory (shifted to signed bytes when zero_in = -128) next to
// the filter as [kb][kh][quad][16 k] words of 4 kw-bytes; a thread makes one pixel x 16 channels.
constexpr int C1_IMGS = 2;
template <bool SIGNED_IN>
__global__ void __launch_bounds__(256)
conv2d_u8_c1_dp4a_kernel(const QArgs a, const uint8_t *__restrict__ in, const uint8_t *__restrict__ filt,
                         const int32_t *__restrict__ bias, uint8_t *__restrict__ out, int pitch, int prow)
{
    extern __shared__ __align__(16) unsigned smem_u[];
    const int quads = (a.Fw + 3) / 4, kbs = a.K / CB;
    unsigned *sw = smem_u;                                    // [kb][kh][quad][16]
    uint8_t *simg = reinterpret_cast<uint8_t *>(sw + (size_t)kbs * a.Fh * quads * CB); // [img][prow][pitch]
    const int n0 = blockIdx.x * C1_IMGS;
    const int imgs = (a.N - n0) < C1_IMGS ? (a.N - n0) : C1_IMGS;
    for (int i = threadIdx.x; i < kbs * a.Fh * quads * CB; i += blockDim.x)
    {
        const int k = i % CB, q = (i / CB) % quads, kh = (i / (CB * quads)) % a.Fh, kb = i / (CB * quads * a.Fh);
        unsigned wv = 0;
        for (int t = 0; t < 4; ++t)
        {
            const int kw = 4 * q + t;
            if (kw < a.Fw) // filter [K/16][1][Fh][Fw][1][16]
                wv |= (unsigned)(filt[(((size_t)kb * a.Fh + kh) * a.Fw + kw) * CB + k] ^ 0x80u) << (8 * t);
        }
        sw[i] = wv;
    }
    const int img_bytes = prow * pitch;
    for (int i = threadIdx.x; i < C1_IMGS * img_bytes / 4; i += blockDim.x)
        reinterpret_cast<unsigned *>(simg)[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < imgs * a.H * a.W; i += blockDim.x)
    {
        const int im = i / (a.H * a.W), p = i - im * a.H * a.W;
        const int h = p / a.W, w = p - h * a.W;
        const uint8_t v = in[(size_t)(n0 + im) * a.H * a.W + p];
        simg[(size_t)im * img_bytes + (h + a.pad_t) * pitch + (w + a.pad_l)] = SIGNED_IN ? (uint8_t)(v ^ 0x80u) : v;
    }
    __syncthreads();
    const int px = a.Ho * a.Wo;
    const int items = imgs * kbs * px;
    for (int it = threadIdx.x; it < items; it += blockDim.x)
    {
        const int p = it % px, kb = (it / px) % kbs, im = it / (px * kbs);
        const int oh = p / a.Wo, ow = p - oh * a.Wo;
        int acc[CB];
#pragma unroll
        for (int k = 0; k < CB; ++k)
            acc[k] = a.k_zero + (bias ? bias[kb * CB + k] : 0);
        const uint8_t *row = simg + (size_t)im * img_bytes + (oh * a.stride) * pitch + ow * a.stride;
        const uint4 *wk = reinterpret_cast<const uint4 *>(sw + (size_t)kb * a.Fh * quads * CB);
        for (int kh = 0; kh < a.Fh; ++kh, row += pitch)
        {
            for (int q = 0; q < quads; ++q)
            {
                const uint8_t *pw = row + 4 * q;
                const unsigned *al = reinterpret_cast<const unsigned *>(pw - ((size_t)pw & 3));
                const unsigned aw = __funnelshift_r(al[0], al[1], 8 * (unsigned)((size_t)pw & 3));
                const uint4 *w4 = wk + (kh * quads + q) * 4;
#pragma unroll
                for (int g = 0; g < 4; ++g)
                {
                    const uint4 wv = w4[g];
                    acc[4 * g + 0] = dp4a_in<SIGNED_IN>(aw, wv.x, acc[4 * g + 0]);
                    acc[4 * g + 1] = dp4a_in<SIGNED_IN>(aw, wv.y, acc[4 * g + 1]);
                    acc[4 * g + 2] = dp4a_in<SIGNED_IN>(aw, wv.z, acc[4 * g + 2]);
                    acc[4 * g + 3] = dp4a_in<SIGNED_IN>(aw, wv.w, acc[4 * g + 3]);
                }
            }
        }
        *reinterpret_cast<uint4 *>(out + (((size_t)(n0 + im) * kbs + kb) * px + p) * CB) =
            requant_pack16(acc, a.lshift, a.rshift, a.mult);
    }
}

// Global average pool (window = whole image, no padding) of at most 256 pixels: LANES lanes per image and 16-channel block
// stride over the pixels.  A channel's sum fits 16 bits, so two channels share a register; the last two steps of the
// reduction halve the channels a lane answers for, and four lanes requantise and store four channels each.  A warp for a
// 3x3 plane with every lane adding and requantising all 16 channels took 21.4 us for 2048 images of 256 channels, all of
// it shuffles and multiplications (the bytes are 1 us).  Four lanes up to 64 pixels: beyond, 16 loads a lane and more
// in a row cost more than three steps of shuffles.
template <int LANES>
__global__ void __launch_bounds__(256)
global_avgpool_small_u8_kernel(const QArgs a, const uint8_t *__restrict__ in, uint8_t *__restrict__ out)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, plane = t / LANES;
    const int l = threadIdx.x & (LANES - 1), px = a.H * a.W;
    const bool live = plane < (long long)a.N * (a.C / CB);
    unsigned even[4] = {0u, 0u, 0u, 0u}, odd[4] = {0u, 0u, 0u, 0u};
    if (live)
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(in) + plane * px;
#pragma unroll 4
        for (int p = l; p < px; p += LANES)
        {
            const uint4 v = __ldg(src + p);
            const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                even[k] += w[k] & 0x00ff00ffu;
                odd[k] += (w[k] >> 8) & 0x00ff00ffu;
            }
        }
    }
#pragma unroll
    for (int off = LANES / 2; off > 2; off >>= 1)
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            even[k] += __shfl_xor_sync(0xffffffffu, even[k], off);
            odd[k] += __shfl_xor_sync(0xffffffffu, odd[k], off);
        }
#pragma unroll
    for (int off = 2; off > 0; off >>= 1) // lanes with the bit keep the upper half of what is left
    {
        const bool up = l & off;
#pragma unroll
        for (int k = 0; k < off; ++k)
        {
            const unsigned ge = up ? even[k] : even[k + off], go = up ? odd[k] : odd[k + off];
            const unsigned ke = up ? even[k + off] : even[k], ko = up ? odd[k + off] : odd[k];
            even[k] = ke + __shfl_xor_sync(0xffffffffu, ge, off);
            odd[k] = ko + __shfl_xor_sync(0xffffffffu, go, off);
        }
    }
    if (live && l < 4)
    {
        const int zero = px * a.zero_in + a.k_zero;
        unsigned o = 0;
        const unsigned sums[4] = {even[0] & 0xffffu, odd[0] & 0xffffu, even[0] >> 16, odd[0] >> 16};
#pragma unroll
        for (int k = 0; k < 4; ++k)
            o |= (unsigned)(requant_dev((int)sums[k] + zero, a.lshift, a.rshift, a.mult) & 255) << (8 * k);
        reinterpret_cast<unsigned *>(out)[plane * 4 + l] = o;
    }
}

// The same for larger images: one warp per image and 16-channel block; lanes stride over the pixels, then a shuffle tree adds
// the 16 channel sums.
__global__ void __launch_bounds__(256)
global_avgpool_u8_kernel(const QArgs a, const uint8_t *__restrict__ in, uint8_t *__restrict__ out)
{
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const long long planes = (long long)a.N * (a.C / CB);
    if (warp >= planes)
        return;
    const int px = a.H * a.W;
    const uint4 *plane = reinterpret_cast<const uint4 *>(in + (size_t)warp * px * CB);
    int acc[CB];
#pragma unroll
    for (int k = 0; k < CB; ++k)
        acc[k] = 0;
    for (int p = lane; p < px; p += 32)
    {
        const uint4 v = plane[p];
#pragma unroll
        for (int k = 0; k < CB; ++k)
            acc[k] += byte_of(v, k);
    }
#pragma unroll
    for (int k = 0; k < CB; ++k)
    {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], off);
        acc[k] = requant_dev(acc[k] + px * a.zero_in + a.k_zero, a.lshift, a.rshift, a.mult);
    }
    if (lane == 0)
        *reinterpret_cast<uint4 *>(out + (size_t)warp * CB) = pack16(acc);
}

__global__ void __launch_bounds__(256)
relu_u8_kernel(long long n16, const QArgs a, const uint8_t *in, uint8_t *out) // in may alias out
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride)
    {
        const uint4 v = *reinterpret_cast<const uint4 *>(in + i * 16);
        int r[CB];
#pragma unroll
        for (int k = 0; k < CB; ++k)
        {
            const int x = byte_of(v, k) + a.zero_in;
            r[k] = requant_dev(x > a.k_zero ? x : a.k_zero, a.lshift, a.rshift, a.mult);
        }
        *reinterpret_cast<uint4 *>(out + i * 16) = pack16(r);
    }
}

void fill(const small_b200_layer *L, QArgs &a, bool dense)
{
    a.N = L->N; a.C = L->C; a.K = dense ? L->K : L->C; a.H = L->H; a.W = L->W;
    a.Fh = L->Fh; a.Fw = L->Fw; a.stride = L->stride; a.pad_t = L->pad_t; a.pad_l = L->pad_l;
    a.Ho = out_dim(L->H, L->pad_t, L->pad_b, L->Fh, L->stride);
    a.Wo = out_dim(L->W, L->pad_l, L->pad_r, L->Fw, L->stride);
    a.cib = dense ? eff_block(L->C) : CB;
    a.cbs = L->C / a.cib;
    a.zero_in = L->zero_in; a.zero_filt = L->zero_filt; a.lshift = L->lshift;
    a.rshift = L->rshift; a.mult = L->multiplier; a.k_zero = L->k_zero;
}

int check_quant(const small_b200_layer *L, const char *name)
{
    if (L->lshift < 0 || L->lshift > 31 || L->rshift < 0 || L->rshift > 31)
        return fail(SMALL_B200_INVALID_ARGUMENT, std::string(name) + " ERROR: shift out of range.");
    if (row_stride(L) != L->stride)
        return fail(SMALL_B200_INVALID_ARGUMENT, std::string(name) + " ERROR: stride unsupported (a row stride of its own "
                                                                      "is provided for the fp32 layers only).");
    return SMALL_B200_OK;
}

// The reference's quint8 Partial forms (interface_abstract.hpp:595-767 PartialConv2D, :1194
// PartialDepthwiseConv2D) reuse the uint8 output buffer as int32 storage: the accumulators of output
// channel block k start at BYTE k * Ho*Wo*block and are four times as long as the block's bytes
// (q_abstract_layer.hpp:1135-1144), so the accumulators of one block lie over those of the next three and
// the form has a defined meaning for ONE block of output channels only -- 16 channels on this platform --
// and one image.  There: out holds int32 [Ho*Wo][16] on entry and the bytes [Ho*Wo][16] of
// requantise(entry + convolution) at its start on return.  Anything else is refused.
int check_partial_u8(const small_b200_layer *L, const char *name, int channels, const int32_t *bias)
{
    if (channels != CB || L->N != 1)
        return fail(SMALL_B200_INVALID_ARGUMENT,
                    std::string(name) + " ERROR: the int32 partial sums of different blocks of output channels (and of "
                                        "different images) overlap inside the output buffer; only 16 output channels "
                                        "and one image have a defined result.");
    if (bias)
        return fail(SMALL_B200_INVALID_ARGUMENT, std::string(name) + " ERROR: the partial-sum form takes no bias.");
    return SMALL_B200_OK;
}

// -1: not a shape of the tiled depthwise kernel.
int launch_dw_tile(const small_b200_layer *L, const QArgs &q, const uint8_t *in, const uint8_t *filt, const int32_t *bias, uint8_t *out,
                   cudaStream_t st)
{
    if (q.Fh != 3 || q.Fw != 3 || q.stride != 1 || row_stride(L) != 1 || q.zero_in > 0 || q.zero_in < -255) // padding has to be a byte
        return -1;
    DwTile a{};
    a.N = q.N; a.cbs = q.C / CB; a.H = q.H; a.W = q.W; a.Ho = q.Ho; a.Wo = q.Wo; a.pad_t = q.pad_t; a.pad_l = q.pad_l;
    a.zero_in = q.zero_in; a.sum_a = 128 + q.zero_filt;
    a.lshift = q.lshift; a.rshift = q.rshift; a.mult = q.mult; a.k_zero = q.k_zero;
    const long long total_planes = (long long)q.N * a.cbs;
    // Strips of 5 or of 3, by the instructions they take (two rows, four channels a thread); with sums of the input the
    // accumulators of 5 would not fit the registers.
    auto cost = [&](int tw) { return (q.Wo + tw - 1) / tw * (tw * 76 + (tw + 2) * 14); };
    const int tw = !a.sum_a && cost(5) <= cost(3) ? 5 : 3;
    const long long cap = 72 * 1024, room = 3LL * num_sms(); // three CTAs an SM, what the registers leave
    const int total_strips = (q.Wo + tw - 1) / tw;
    auto width = [&](int strips) { // of a tile
        a.strips = strips; a.cols = strips == total_strips ? q.Wo : strips * tw;
        a.pitch = (strips * tw + 2) | 1; // odd: row pairs, two pitches apart, use different banks
    };
    auto bytes = [&](int planes, int rows) {
        const int in_rows = (rows + 1) / 2 * 2 + 2;
        a.in_bytes = (unsigned)((planes * in_rows * a.pitch * CB + 127) & ~127);
        a.out_bytes = (unsigned)((planes * rows * a.cols * CB + 127) & ~127);
        a.out_at = 2 * a.in_bytes;
        a.w_at = a.out_at + 2 * a.out_bytes;
        return (long long)a.w_at + a.cbs * 4 * CB * 4;
    };
    // The tile: the one with the shortest estimated time, rounds of a CTA's threads plus about half a round for a tile's
    // barrier and copies, with three CTAs an SM, which hide each other's waits.
    int best_planes = 0, best_rows = 0, best_strips = total_strips;
    double best = 1e30;
    auto consider = [&](int planes, int rows, double copies) {
        const long long items = (long long)planes * ((rows + 1) / 2) * a.strips * 4;
        const long long tiles = (total_planes + planes - 1) / planes * ((q.Ho + rows - 1) / rows) * ((total_strips + a.strips - 1) / a.strips);
        const double time = (double)((tiles + room - 1) / room) * ((double)((items + DW_THREADS - 1) / DW_THREADS) + 0.5 + copies);
        if (time < best) { best = time; best_planes = planes; best_rows = rows; best_strips = a.strips; }
    };
    if (q.W <= 4096 && q.H <= 0x10000)
    {
        width(total_strips);
        if (q.W + q.pad_l <= a.pitch)
        {
            for (int planes = 1; planes <= 256 && planes <= total_planes && bytes(planes, q.Ho) <= cap; ++planes)
                consider(planes, q.Ho, 0.0);
            for (int rows = 2; rows < q.Ho && bytes(1, rows) <= cap; rows += 2)
                consider(1, rows, 0.0);
        }
    }
    // Rows that don't fit as a whole, four in and two out, twice (192 bytes a pixel: from a width of some 380 on, less with many
    // channels), are cut.  Whole rows are as fast up to there: 16 channels, 64 images, 376 wide 158 us, 416 wide in pieces 159.
    // Tiles of 4 to 32 rows then, so that few of the rows are copied twice; a sixteenth of a round for a pixel a thread copies.
    const bool cut = !best_planes;
    if (cut)
        for (int pieces = 2; pieces <= total_strips; ++pieces)
        {
            const int strips = (total_strips + pieces - 1) / pieces;
            if (strips == a.strips || strips > 128)
                continue;
            width(strips);
            for (int rows = std::min(4, q.Ho); rows <= std::min(32, q.Ho) && bytes(1, rows) <= cap; rows += rows < q.Ho ? std::min(2, q.Ho - rows) : 1)
                consider(1, rows, ((rows + 1) / 2 * 2 + 2) * a.pitch / (16.0 * DW_THREADS));
            if (strips <= 8)
                break;
        }
    if (!best_planes)
        return -1;
    width(best_strips);
    a.col_tiles = (total_strips + a.strips - 1) / a.strips;
    a.planes = best_planes; a.rows = best_rows;
    a.row_tiles = (q.Ho + a.rows - 1) / a.rows;
    a.pairs = (a.rows + 1) / 2; a.in_rows = 2 * a.pairs + 2;
    const size_t smem = (size_t)bytes(a.planes, a.rows);
    const long long tiles = (total_planes + a.planes - 1) / a.planes * a.row_tiles * a.col_tiles;
    if (tiles > 0x3fffffffLL || total_planes > 0x3fffffffLL)
        return -1;
    a.tiles = (int)tiles;
    const unsigned blocks = (unsigned)(tiles < room ? tiles : room);
    const int copy_rows = cut ? 1 : std::min(a.H, a.in_rows - a.pad_t); // rows of the image in a tile of whole planes
    if (copy_rows <= 0)
        return -1;
    a.by_row_tiles.set(a.row_tiles); a.by_col_tiles.set(a.col_tiles); a.by_cbs.set(a.cbs); a.by_strips.set(a.strips); a.by_pairs.set(a.pairs);
    a.by_pitch.set(a.pitch); a.by_in_rows.set(a.in_rows); a.by_copy_rows.set(copy_rows); a.by_W.set(a.W);
    static PerDeviceOnce configured;
    int dev;
    if (configured.needed(&dev))
    {
        for (auto k : {dwconv3x3_u8_tile_kernel<3, true, false>, dwconv3x3_u8_tile_kernel<3, false, false>, dwconv3x3_u8_tile_kernel<5, false, false>,
                       dwconv3x3_u8_tile_kernel<3, true, true>, dwconv3x3_u8_tile_kernel<3, false, true>, dwconv3x3_u8_tile_kernel<5, false, true>})
            SB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
        configured.mark(dev);
    }
    auto kern = a.sum_a ? (cut ? dwconv3x3_u8_tile_kernel<3, true, true> : dwconv3x3_u8_tile_kernel<3, true, false>)
              : tw == 5 ? (cut ? dwconv3x3_u8_tile_kernel<5, false, true> : dwconv3x3_u8_tile_kernel<5, false, false>)
                        : (cut ? dwconv3x3_u8_tile_kernel<3, false, true> : dwconv3x3_u8_tile_kernel<3, false, false>);
    kern<<<blocks, DW_THREADS, smem, st>>>(a, in, filt, bias, out);
    return launched("dwconv3x3_u8_tile_kernel");
}

template <int OP>
int launch_window(const small_b200_layer *L, const char *name, int max_stride, const uint8_t *in,
                  const uint8_t *filt, const int32_t *bias, uint8_t *out, void *stream)
{
    if (int rc = check_window_layer(L, name, false, max_stride))
        return rc;
    if (int rc = check_quant(L, name))
        return rc;
    QArgs a; fill(L, a, false);
    const long long items = (long long)a.N * (a.C / CB) * a.Ho * a.Wo;
    if (L->accumulate)
    {
        if (OP != 0)
            return fail(SMALL_B200_INVALID_ARGUMENT, std::string(name) + " ERROR: no partial form.");
        if (int rc = check_partial_u8(L, "PartialDepthwiseConv2D<quint8>", L->C, bias))
            return rc;
        if (items == 0)
            return SMALL_B200_OK;
        window_u8_kernel<OP, true><<<(unsigned)((items + 255) / 256), 256, 0, as_stream(stream)>>>(a, in, filt, nullptr, out);
        if (int rc = launched(name))
            return rc;
        requant_in_place_kernel<<<1, 1024, 0, as_stream(stream)>>>(a.Ho * a.Wo, a, out);
        return launched("requant_in_place_kernel");
    }
    if (items == 0)
        return SMALL_B200_OK;
    if (OP == 0)
    {
        const int rc = launch_dw_tile(L, a, in, filt, bias, out, as_stream(stream));
        if (rc >= 0)
            return rc;
    }
    if (OP == 0 && a.zero_filt == -128 && (a.zero_in == 0 || a.zero_in == -128) && a.Fh * a.Fw <= 64 && a.C <= 2048)
    {
        const int quads = (a.Fh * a.Fw + 3) / 4;
        const size_t smem = (size_t)(a.C / CB) * quads * CB * 4 + (size_t)quads * 4 * sizeof(short2);
        const unsigned blocks = (unsigned)((items + 255) / 256);
        const bool sgn = a.zero_in != 0;
        cudaStream_t st = as_stream(stream);
        if (quads == 3) // 3x3
            sgn ? dwconv_u8_dp4a_kernel<true, 3><<<blocks, 256, smem, st>>>(a, in, filt, bias, out)
                : dwconv_u8_dp4a_kernel<false, 3><<<blocks, 256, smem, st>>>(a, in, filt, bias, out);
        else if (quads == 1)
            sgn ? dwconv_u8_dp4a_kernel<true, 1><<<blocks, 256, smem, st>>>(a, in, filt, bias, out)
                : dwconv_u8_dp4a_kernel<false, 1><<<blocks, 256, smem, st>>>(a, in, filt, bias, out);
        else
            sgn ? dwconv_u8_dp4a_kernel<true, 0><<<blocks, 256, smem, st>>>(a, in, filt, bias, out)
                : dwconv_u8_dp4a_kernel<false, 0><<<blocks, 256, smem, st>>>(a, in, filt, bias, out);
        return launched("dwconv_u8_dp4a_kernel");
    }
    if (OP == 2 && a.Fh == a.H && a.Fw == a.W && !L->pad_t && !L->pad_b && !L->pad_l && !L->pad_r)
    {
        const long long warps = (long long)a.N * (a.C / CB);
        const int px = a.H * a.W;
        if (px <= 256)
        {
            const int lanes = px <= 64 ? 4 : 32;
            (lanes == 4 ? global_avgpool_small_u8_kernel<4> : global_avgpool_small_u8_kernel<32>)
                <<<(unsigned)((warps * lanes + 255) / 256), 256, 0, as_stream(stream)>>>(a, in, out);
            return launched("global_avgpool_small_u8_kernel");
        }
        global_avgpool_u8_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, as_stream(stream)>>>(a, in, out);
        return launched("global_avgpool_u8_kernel");
    }
    window_u8_kernel<OP><<<(unsigned)((items + 255) / 256), 256, 0, as_stream(stream)>>>(a, in, filt, bias, out);
    return launched(name);
}
} // namespace

namespace sb
{
// Defined in conv_u8_tc.cu: the tensor-core path for shapes it supports.  Returns -1 when
// the shape is not covered, otherwise a SMALL_B200_* code.
int conv2d_u8_tensor_core(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt,
                          const int32_t *bias, uint8_t *out, cudaStream_t st);
int conv2d_u8_one_channel_tc(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt,
                             const int32_t *bias, uint8_t *out, cudaStream_t st);
// Defined in conv_u8_patch.cu: windows of more than one tap on blocks of channels, for zero points whose padding is a byte.
int conv2d_u8_patch(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt, const int32_t *bias,
                    uint8_t *out, cudaStream_t st);
// Defined in conv_u8_rgb.cu: first layers on many pixels of three channels, where conv2d_u8_onestep would take them; -1 otherwise.
int conv2d_u8_rgb(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt, const int32_t *bias,
                  uint8_t *out, cudaStream_t st);
// Defined in conv_u8_thin.cu: pointwise layers on many pixels of 16, 32 or 64 channels; -1 otherwise.
int conv2d_u8_thin(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt, const int32_t *bias,
                   uint8_t *out, cudaStream_t st);
// Defined in conv_u8_ring.cu: every other window / stride / channel count as an implicit GEMM on the
// tensor core, for the zero points it covers; -1 otherwise.
int conv2d_u8_ring(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt, const int32_t *bias,
                   uint8_t *out, cudaStream_t st);
}

namespace
{
// Layers whose whole reduction is at most 32 bytes and whose padding is a byte.
bool one_step_covers(const small_b200_layer *L)
{
    return (long long)L->C * L->Fh * L->Fw <= 32 && (L->C < CB || (L->Fh == 1 && L->Fw == 1)) && L->zero_in <= 0 && L->zero_in >= -255 &&
           L->K <= 1024;
}
// ... and which the kernel does faster than conv_u8_tc.cu (what conv_u8_rgb.cu and conv_u8_thin.cu do faster never gets here).  2048
// images, us, this kernel and that one: 16 -> 32 channels at 24x24 27 and 49, 16 -> 64 48 and 68, 16 -> 128 at 12x12 25 and 29; but
// 32 -> 32 at 24x24 37 and 34, and a few images of 32 channels 5 and 4.
bool one_step_preferred(const small_b200_layer *L)
{
    return one_step_covers(L) && (L->C < CB || (L->C == CB && L->K <= 128));
}

template <int WORDS, int KIND>
int launch_onestep(const OneArgs &a, const uint8_t *in, const uint8_t *filt, const int32_t *bias, uint8_t *out, cudaStream_t st)
{
    const size_t smem = (size_t)a.K * (WORDS + 1) * 4; // at most 36 KB
    constexpr int PX = 2;
    const long long sms = num_sms(), many = (long long)PX * 256;
    if (a.total >= sms * many) // two pixels a thread once that leaves a CTA for every SM
    {
        const long long nb = std::min((a.total + many - 1) / many, sms * 8);
        conv2d_u8_onestep_kernel<WORDS, KIND, PX><<<(unsigned)nb, 256, smem, st>>>(a, in, filt, bias, out);
    }
    else
        conv2d_u8_onestep_kernel<WORDS, KIND, 1><<<(unsigned)((a.total + 255) / 256), 256, smem, st>>>(a, in, filt, bias, out);
    return launched("conv2d_u8_onestep_kernel");
}

// -1: not covered.
int conv2d_u8_onestep(const small_b200_layer *L, const QArgs &q, const uint8_t *in, const uint8_t *filt, const int32_t *bias, uint8_t *out,
                      cudaStream_t st)
{
    const long long px = (long long)q.Ho * q.Wo;
    if (!one_step_covers(L) || row_stride(L) != q.stride || px > 0x3fffffffLL || reinterpret_cast<uintptr_t>(in) % 16 ||
        reinterpret_cast<uintptr_t>(out) % 16)
        return -1;
    OneArgs a{};
    a.H = q.H; a.W = q.W; a.Ho = q.Ho; a.Wo = q.Wo; a.C = q.C; a.K = q.K; a.Fh = q.Fh; a.Fw = q.Fw; a.R = q.C * q.Fh * q.Fw;
    a.stride = q.stride; a.pad_t = q.pad_t; a.pad_l = q.pad_l;
    a.zero_in = q.zero_in; a.sum_a = 128 + q.zero_filt;
    a.lshift = q.lshift; a.rshift = q.rshift; a.mult = q.mult; a.k_zero = q.k_zero;
    a.by_hw.set((int)px); a.by_Wo.set(q.Wo);
    // images in portions of less than 2^30 pixels
    const long long per = 0x3fffffffLL / px, in_image = (long long)q.C * q.H * q.W, out_image = px * q.K;
    for (long long n = 0; n < q.N; n += per)
    {
        const long long images = std::min(per, (long long)q.N - n);
        a.total = (int)(images * px);
        a.in_bytes = images * in_image;
        const uint8_t *x = in + n * in_image;
        uint8_t *y = out + n * out_image;
        const int rc = q.C >= 2 * CB                                ? launch_onestep<8, ONE_1X1>(a, x, filt, bias, y, st)
                       : q.C == CB                                  ? launch_onestep<4, ONE_1X1>(a, x, filt, bias, y, st)
                       : q.C == 3 && q.Fh == 3 && q.Fw == 3 ? launch_onestep<7, ONE_333>(a, x, filt, bias, y, st)
                                                                    : launch_onestep<8, ONE_FIRST>(a, x, filt, bias, y, st);
        if (rc)
            return rc;
    }
    return SMALL_B200_OK;
}

// path: 0 = the faster kernel for the shape, 1 = CUDA cores only, 2 = tensor cores or an error
int conv2d_u8_dispatch(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt, const int32_t *bias,
                       uint8_t *out, void *stream, int path)
{
    const bool tensor_core = path != 1;
    if (int rc = check_window_layer(L, "Conv2D<quint8>", true, 2))
        return rc;
    if (int rc = check_quant(L, "Conv2D<quint8>"))
        return rc;
    if (L->accumulate)
    {
        if (int rc = check_partial_u8(L, "PartialConv2D<quint8>", L->K, bias))
            return rc;
        if (path == 2)
            return fail(SMALL_B200_INVALID_ARGUMENT, "PartialConv2D<quint8> ERROR: runs on the CUDA cores only.");
        QArgs a; fill(L, a, true);
        if (a.Ho <= 0 || a.Wo <= 0)
            return SMALL_B200_OK;
        dim3 grid((a.Ho * a.Wo + 127) / 128, 1, 1);
        conv2d_u8_direct_kernel<true><<<grid, 128, 0, as_stream(stream)>>>(a, in, filt, nullptr, out);
        if (int rc = launched("conv2d_u8_direct_kernel"))
            return rc;
        requant_in_place_kernel<<<1, 1024, 0, as_stream(stream)>>>(a.Ho * a.Wo, a, out);
        return launched("requant_in_place_kernel");
    }
    QArgs a; fill(L, a, true);
    if (a.N == 0 || a.Ho == 0 || a.Wo == 0)
        return SMALL_B200_OK;
    if (path == 0)
    {
        const int thin = conv2d_u8_thin(L, in, filt, bias, out, as_stream(stream));
        if (thin >= 0)
            return thin;
    }
    if (path == 0 && L->C >= CB && one_step_preferred(L))
    {
        const int one = conv2d_u8_onestep(L, a, in, filt, bias, out, as_stream(stream));
        if (one >= 0)
            return one;
    }
    const int tc = tensor_core ? conv2d_u8_tensor_core(L, in, filt, bias, out, as_stream(stream)) : -1;
    if (tc >= 0)
        return tc;
    if (tensor_core)
    {
        const int tc1 = conv2d_u8_one_channel_tc(L, in, filt, bias, out, as_stream(stream));
        if (tc1 >= 0)
            return tc1;
    }
    if (path == 0 && one_step_preferred(L))
    {
        const int rgb = conv2d_u8_rgb(L, in, filt, bias, out, as_stream(stream));
        if (rgb >= 0)
            return rgb;
    }
    if (path == 1 || (path == 0 && one_step_preferred(L)))
    {
        const int one = conv2d_u8_onestep(L, a, in, filt, bias, out, as_stream(stream));
        if (one >= 0)
            return one;
    }
    if (tensor_core)
    {
        const int tc2 = conv2d_u8_patch(L, in, filt, bias, out, as_stream(stream));
        if (tc2 >= 0)
            return tc2;
    }
    if (tensor_core)
    {
        const int tc2 = conv2d_u8_ring(L, in, filt, bias, out, as_stream(stream));
        if (tc2 >= 0)
            return tc2;
    }
    if (path == 2)
        return fail(SMALL_B200_INVALID_ARGUMENT, "Conv2D<quint8> ERROR: layer not covered by the tensor-core kernels.");
    if (a.C == 1 && a.zero_filt == -128 && (a.zero_in == 0 || a.zero_in == -128))
    {
        // one-channel image: rows of the window are words of the (zero-padded) image
        const int quads = (a.Fw + 3) / 4;
        const int pitch = ((a.W + L->pad_l + L->pad_r + 4 * quads + 8) + 3) & ~3; // room for the unaligned read
        const int prow = a.H + L->pad_t + L->pad_b + 1;
        const size_t smem = (size_t)(a.K / CB) * a.Fh * quads * CB * 4 + (size_t)C1_IMGS * prow * pitch;
        if (smem <= 160 * 1024)
        {
            static PerDeviceOnce configured;
            int dev;
            if (configured.needed(&dev))
            {
                SB_CUDA(cudaFuncSetAttribute(conv2d_u8_c1_dp4a_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
                SB_CUDA(cudaFuncSetAttribute(conv2d_u8_c1_dp4a_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
                configured.mark(dev);
            }
            const unsigned blocks = (unsigned)((a.N + C1_IMGS - 1) / C1_IMGS);
            if (a.zero_in == 0)
                conv2d_u8_c1_dp4a_kernel<false><<<blocks, 256, smem, as_stream(stream)>>>(a, in, filt, bias, out, pitch, prow);
            else
                conv2d_u8_c1_dp4a_kernel<true><<<blocks, 256, smem, as_stream(stream)>>>(a, in, filt, bias, out, pitch, prow);
            return launched("conv2d_u8_c1_dp4a_kernel");
        }
    }
    dim3 grid((a.Ho * a.Wo + 127) / 128, a.K / CB, a.N);
    conv2d_u8_direct_kernel<false><<<grid, 128, 0, as_stream(stream)>>>(a, in, filt, bias, out);
    return launched("conv2d_u8_direct_kernel");
}
} // namespace

extern "C"
{
int small_b200_conv2d_u8(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt,
                         const int32_t *bias, uint8_t *out, void *stream)
{
    return conv2d_u8_dispatch(L, in, filt, bias, out, stream, 0);
}

int small_b200_conv2d_u8_cuda_cores(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt,
                                    const int32_t *bias, uint8_t *out, void *stream)
{
    return conv2d_u8_dispatch(L, in, filt, bias, out, stream, 1);
}

int small_b200_conv2d_u8_tensor_core(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt,
                                     const int32_t *bias, uint8_t *out, void *stream)
{
    return conv2d_u8_dispatch(L, in, filt, bias, out, stream, 2);
}

int small_b200_dwconv2d_u8(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt,
                           const int32_t *bias, uint8_t *out, void *stream)
{
    return launch_window<0>(L, "DepthwiseConv2D<quint8>", 2, in, filt, bias, out, stream);
}

int small_b200_maxpool2d_u8(const small_b200_layer *L, const uint8_t *in, uint8_t *out, void *stream)
{
    return launch_window<1>(L, "MaxPool2D<quint8>", 2, in, nullptr, nullptr, out, stream);
}

int small_b200_avgpool2d_u8(const small_b200_layer *L, const uint8_t *in, uint8_t *out, void *stream)
{
    return launch_window<2>(L, "AveragePool2D<quint8>", 3, in, nullptr, nullptr, out, stream);
}

int small_b200_relu_u8(int64_t n, const small_b200_layer *L, const uint8_t *in, uint8_t *out, void *stream)
{
    if (n < 0 || n % CB != 0)
        return fail(SMALL_B200_INVALID_ARGUMENT, "ReLUActivation<quint8> ERROR: in_channels unsupported.");
    if (int rc = check_quant(L, "ReLUActivation<quint8>"))
        return rc;
    if (n == 0)
        return SMALL_B200_OK;
    QArgs a{};
    a.zero_in = L->zero_in; a.lshift = L->lshift; a.rshift = L->rshift; a.mult = L->multiplier;
    a.k_zero = L->k_zero;
    const long long n16 = n / 16;
    long long blocks = (n16 + 255) / 256;
    const long long cap = (long long)num_sms() * 16;
    if (blocks > cap)
        blocks = cap;
    relu_u8_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(n16, a, in, out);
    return launched("relu_u8");
}
} // extern "C"
