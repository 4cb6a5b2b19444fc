// HBM-bound kernels of the forward pass: layout/precision boundary, pooling, per-channel affine +
// activation, tensor combination, channel-slice copies, softmax, col2im gather, u8 helpers.
// All of them walk channels-innermost tensors in 16-byte channel vectors so that every global access
// of a warp is a run of full sectors.
#include "common.cuh"
#include <type_traits>
#include <float.h>
#include <math.h>

namespace {

// ---- 16-byte channel vectors --------------------------------------------------------------------
template <typename T> struct Vec;
template <> struct Vec<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void load(const float *p, float (&v)[4])
    {
        float4 t = *reinterpret_cast<const float4 *>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
    static __device__ __forceinline__ void store(float *p, const float (&v)[4])
    {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <> struct Vec<__half> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const __half *p, float (&v)[8])
    {
        uint4 t = *reinterpret_cast<const uint4 *>(p);
        const __half2 *h = reinterpret_cast<const __half2 *>(&t);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float2 f = __half22float2(h[i]);
            v[2 * i] = f.x; v[2 * i + 1] = f.y;
        }
    }
    static __device__ __forceinline__ void store(__half *p, const float (&v)[8])
    {
        uint4 t;
        __half2 *h = reinterpret_cast<__half2 *>(&t);
#pragma unroll
        for (int i = 0; i < 4; i++) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
        *reinterpret_cast<uint4 *>(p) = t;
    }
};
template <> struct Vec<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const __nv_bfloat16 *p, float (&v)[8])
    {
        uint4 t = *reinterpret_cast<const uint4 *>(p);
        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&t);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float2 f = __bfloat1622float2(h[i]);
            v[2 * i] = f.x; v[2 * i + 1] = f.y;
        }
    }
    static __device__ __forceinline__ void store(__nv_bfloat16 *p, const float (&v)[8])
    {
        uint4 t;
        __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&t);
#pragma unroll
        for (int i = 0; i < 4; i++) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        *reinterpret_cast<uint4 *>(p) = t;
    }
};
template <> struct Vec<uint8_t> {
    static constexpr int N = 16;
    static __device__ __forceinline__ void load(const uint8_t *p, float (&v)[16])
    {
        uint4 t = *reinterpret_cast<const uint4 *>(p);
        const uint8_t *b = reinterpret_cast<const uint8_t *>(&t);
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = (float)b[i];
    }
    static __device__ __forceinline__ void store(uint8_t *p, const float (&v)[16])
    {
        uint4 t;
        uint8_t *b = reinterpret_cast<uint8_t *>(&t);
#pragma unroll
        for (int i = 0; i < 16; i++) b[i] = (uint8_t)(int)v[i];
        *reinterpret_cast<uint4 *>(p) = t;
    }
};

inline int nblocks(long n, int bs = 256) { return (int)((n + bs - 1) / bs); }

#define DISPATCH_FLOAT_DTYPE(dtype, CALL)                         \
    switch (dtype) {                                               \
    case THB_F32: { using T = float; CALL; break; }                \
    case THB_F16: { using T = __half; CALL; break; }               \
    case THB_BF16: { using T = __nv_bfloat16; CALL; break; }       \
    default: return THB_ERR_UNSUPPORTED;                           \
    }
#define DISPATCH_ANY_DTYPE(dtype, CALL)                            \
    switch (dtype) {                                               \
    case THB_F32: { using T = float; CALL; break; }                \
    case THB_F16: { using T = __half; CALL; break; }               \
    case THB_BF16: { using T = __nv_bfloat16; CALL; break; }       \
    case THB_U8: { using T = uint8_t; CALL; break; }               \
    default: return THB_ERR_UNSUPPORTED;                           \
    }

// ---- preprocess: NCHW fp32 -> normalised NHWC T ---------------------------------------------------
template <typename T>
__global__ void preprocess_kernel(const float *x, float *x_inplace, int N, int C, long HW, float3 mean, float3 std_,
                                  T *y, int y_ld, float q_min, float q_mult)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const long pix = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= (long)N * HW) return;
    const long n = pix / HW, hw = pix - n * HW;
    const float m[3] = {mean.x, mean.y, mean.z}, sd[3] = {std_.x, std_.y, std_.z};
    const float zr = roundf(q_min * q_mult);
    // every stored channel of the pixel is written (y_ld may exceed the rounded channel count: zeros there)
    for (int c0 = 0; c0 < y_ld; c0 += VN) {
        float v[VN];
#pragma unroll
        for (int i = 0; i < VN; i++) {
            const int c = c0 + i;
            float val = 0.f;
            if (c < C) {
                const long idx = (n * C + c) * HW + hw;
                val = x[idx];
                if (c < 3) val = __fdiv_rn(__fsub_rn(val, m[c]), sd[c]);
                if (x_inplace) x_inplace[idx] = val;
                if (sizeof(T) == 1) val = (float)(((int)(roundf(val * q_mult) - zr)) & 255);
            }
            v[i] = val;
        }
        Vec<T>::store(y + pix * y_ld + c0, v);
    }
}

// Space-to-depth variant for a stride-2 first convolution on very few channels: the 2x2 pixel block
// (ph, pw) of channel c becomes channel (ph*2 + pw)*C + c of a half-resolution tensor, so the convolution
// turns into a stride-1 one over 4*C channels whose gathered 16-byte chunks are fully used.
// Rows may be stored row_pitch pixels apart with pad_left zero pixels in front (and zeros behind): every pixel of such
// a row is written here, the padding as zeros.
template <typename T>
__global__ void preprocess_s2d_kernel(const float *x, float *x_inplace, int N, int C, int H, int W, float3 mean,
                                      float3 std_, T *y, int y_ld, int row_pitch, int pad_left)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const int H2 = H / 2, W2 = W / 2;
    const long pix = (long)blockIdx.x * blockDim.x + threadIdx.x;  // over the stored (padded) pixels
    if (pix >= (long)N * H2 * row_pitch) return;
    const long n = pix / ((long)H2 * row_pitch);
    const int rem = (int)(pix - n * (long)H2 * row_pitch), bh = rem / row_pitch, bw = rem - bh * row_pitch - pad_left;
    const bool real = bw >= 0 && bw < W2;
    const float m[3] = {mean.x, mean.y, mean.z}, sd[3] = {std_.x, std_.y, std_.z};
    const int Cs = 4 * C, Cpad = (Cs + VN - 1) / VN * VN;
    // Three planes (every benchmark network): the block's 2 x 2 pixels of every plane as two 8-byte loads per plane (W is
    // even, so a pixel pair never straddles a row and is 8-byte aligned), all issued before any is used, every index
    // known at compile time.  Other plane counts take the element-wise loop below.
    if (C != 3) {
        for (int c0 = 0; c0 < Cpad; c0 += VN) {
            float v[VN];
#pragma unroll
            for (int i = 0; i < VN; i++) {
                const int cs = c0 + i;
                float val = 0.f;
                if (real && cs < Cs) {
                    const int blk = cs / C, c = cs - blk * C;
                    const long idx = ((n * C + c) * H + (2 * bh + (blk >> 1))) * W + 2 * bw + (blk & 1);
                    val = x[idx];
                    if (c < 3) val = __fdiv_rn(__fsub_rn(val, m[c]), sd[c]);
                    if (x_inplace) x_inplace[idx] = val;
                }
                v[i] = val;
            }
            Vec<T>::store(y + pix * y_ld + c0, v);
        }
        return;
    }
    float vals[16];
#pragma unroll
    for (int i = 0; i < 16; i++) vals[i] = 0.f;
    if (real) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
#pragma unroll
            for (int ph = 0; ph < 2; ph++) {
                const long idx = ((n * C + c) * H + (2 * bh + ph)) * W + 2 * bw;
                float2 v = *reinterpret_cast<const float2 *>(x + idx);
                if (c < 3) {
                    v.x = __fdiv_rn(__fsub_rn(v.x, m[c]), sd[c]);
                    v.y = __fdiv_rn(__fsub_rn(v.y, m[c]), sd[c]);
                }
                if (x_inplace) *reinterpret_cast<float2 *>(x_inplace + idx) = v;
                // channel (ph*2 + pw)*3 + c of the regrouped pixel
                vals[(ph * 2) * 3 + c] = v.x;
                vals[(ph * 2 + 1) * 3 + c] = v.y;
            }
        }
    }
#pragma unroll
    for (int c0 = 0; c0 < 16; c0 += VN) {
        if (c0 >= Cpad) break;   // (12 channels rounded up to the type's 16-byte group: 12 for fp32, 16 otherwise)
        float v[VN];
#pragma unroll
        for (int i = 0; i < VN; i++) v[i] = vals[c0 + i];
        Vec<T>::store(y + pix * y_ld + c0, v);
    }
}

// The same for any block size f (a first convolution of stride f), any plane count with C*f*f stored channels or fewer, and
// image sides that f does not divide (the missing pixels are zeros, in uint8 the byte 0.0 quantises to, which the zero point
// cancels).  One thread per stored 16-byte group; SRC: NCHW floats or HWC bytes.
struct S2dArgs {
    const void *src;
    float *x_inplace;  // floats: where the normalised values go back to, or null
    int N, C, H, W, f, stride, bgr;
    float3 mean, std_;  // bytes: 1 / std
    int y_ld, row_pitch, pad_left;
    float q_mult, zr;   // uint8 floats
    int3 q_sub;         // uint8 bytes (lowp_images.c)
    float3 q_mul;
    int q_zero;         // uint8: the byte of 0.0
    int words;          // bytes: every pixel pair starts at an even address
};
template <typename T, bool BYTES>
__global__ void preprocess_s2d_any_kernel(const S2dArgs a, T *y)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const int H2 = (a.H + a.f - 1) / a.f, W2 = (a.W + a.f - 1) / a.f, groups = a.y_ld / VN;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long pix = t / groups;
    if (pix >= (long)a.N * H2 * a.row_pitch) return;
    const int c0 = (int)(t - pix * groups) * VN;
    const long n = pix / ((long)H2 * a.row_pitch);
    const int rem = (int)(pix - n * (long)H2 * a.row_pitch), bh = rem / a.row_pitch, bw = rem - bh * a.row_pitch - a.pad_left;
    const bool real = bw >= 0 && bw < W2;
    const float m[3] = {a.mean.x, a.mean.y, a.mean.z}, sd[3] = {a.std_.x, a.std_.y, a.std_.z};
    const int qs[3] = {a.q_sub.x, a.q_sub.y, a.q_sub.z};
    const float qm[3] = {a.q_mul.x, a.q_mul.y, a.q_mul.z};
    int blk = c0 / a.C, c = c0 - blk * a.C, ph = blk / a.f, pw = blk - ph * a.f;  // stepped, not divided, from here on
    float v[VN];
#pragma unroll
    for (int i = 0; i < VN; i++) {
        float val = 0.f;
        if (real && ph < a.f) {
            const int h = bh * a.f + ph, w = bw * a.f + pw;
            if (h < a.H && w < a.W) {
                if (BYTES) {
                    const uint8_t *px = reinterpret_cast<const uint8_t *>(a.src) + ((size_t)n * a.H + h) * a.stride + (size_t)w * a.C;
                    const float b = (float)px[a.bgr ? a.C - 1 - c : c];
                    if (sizeof(T) == 1) val = (float)((int)roundf(__fmul_rn(b - (float)qs[c], qm[c])) & 255);
                    else val = __fmul_rn(__fsub_rn(__fmul_rn(b, 0.003921568f), m[c]), sd[c]);
                } else {
                    const long idx = ((n * a.C + c) * a.H + h) * a.W + w;
                    val = reinterpret_cast<const float *>(a.src)[idx];
                    if (c < 3) val = __fdiv_rn(__fsub_rn(val, m[c]), sd[c]);
                    if (a.x_inplace) a.x_inplace[idx] = val;
                    if (sizeof(T) == 1) val = (float)(((int)(roundf(val * a.q_mult) - a.zr)) & 255);
                }
            } else if (sizeof(T) == 1)
                val = (float)a.q_zero;
        }
        v[i] = val;
        if (++c == a.C) {
            c = 0;
            if (++pw == a.f) { pw = 0; ph++; }
        }
    }
    Vec<T>::store(y + pix * a.y_ld + c0, v);
}

// uint8 engine, 3x3 / stride 1 / pad 1 first convolution on a three-plane float batch: every pixel's 27 neighbours,
// normalised and quantised as preprocess_kernel does, become the channels of that pixel of an [N][H][W][32] byte tensor
// (channel (r*3 + s)*3 + c = plane c of pixel (h - 1 + r, w - 1 + s)); neighbours outside the image hold the byte that 0.0
// quantises to -- with the input zero point b_offset = roundf(q_min * q_mult) of the convolution (lowp_basic.c:15-29) such a
// byte plus b_offset is exactly 0, so the tap contributes nothing, as in the reference, which never visits it.  The layer
// is then a 1x1 convolution over 27 channels.  The in-place side effect writes each pixel once, as the centre tap.
// A block quantises a tile of 32 x 8 pixels with its halo once, into shared memory, and assembles the neighbours from there: with
// every thread normalising and quantising its own 27 values (27 divisions) the kernel took 74 us for 32 images of 224 x 224,
// where its 70 MB are worth 11.
__global__ void __launch_bounds__(256) preprocess_neigh_u8_kernel(const float *x, int N, int H, int W, float3 mean, float3 std_, uint8_t *y,
                                                                  int y_ld, float q_min, float q_mult)
{
    __shared__ uint8_t q[10][34][4];
    pdl_enter();
    const long HW = (long)H * W;
    const int n = blockIdx.z, h0 = blockIdx.y * 8, w0 = blockIdx.x * 32;
    const float m[3] = {mean.x, mean.y, mean.z}, sd[3] = {std_.x, std_.y, std_.z};
    const float zr = roundf(q_min * q_mult);
    const uint32_t zp = (uint32_t)(-(int)zr) & 255u;
    for (int i = threadIdx.x; i < 340; i += 256) {
        const int r = i / 34, c34 = i - r * 34, h = h0 - 1 + r, w = w0 - 1 + c34;
        uint32_t word = zp | zp << 8 | zp << 16;
        if ((unsigned)h < (unsigned)H && (unsigned)w < (unsigned)W) {
            word = 0;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const float val = __fdiv_rn(__fsub_rn(__ldg(x + ((long)n * 3 + c) * HW + (long)h * W + w), m[c]), sd[c]);
                word |= (uint32_t)(((int)(roundf(val * q_mult) - zr)) & 255) << (8 * c);
            }
        }
        *reinterpret_cast<uint32_t *>(q[r][c34]) = word;
    }
    __syncthreads();
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, h = h0 + ty, w = w0 + tx;
    if (h >= H || w >= W) return;
    uint32_t words[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int t = 0; t < 9; t++) {
        const uint32_t v = *reinterpret_cast<const uint32_t *>(q[ty + t / 3][tx + t % 3]);  // three bytes, at byte 3t of the pixel
        words[3 * t >> 2] |= v << (8 * (3 * t & 3));
        if ((3 * t & 3) > 1) words[(3 * t >> 2) + 1] |= v >> (8 * (4 - (3 * t & 3)));
    }
    uint8_t *at = y + (((long)n * H + h) * W + w) * y_ld;
    uint4 *dst = reinterpret_cast<uint4 *>(at);
    dst[0] = make_uint4(words[0], words[1], words[2], words[3]);
    dst[1] = make_uint4(words[4], words[5], words[6], words[7]);
    for (int c0 = 32; c0 < y_ld; c0 += 16) *reinterpret_cast<uint4 *>(at + c0) = make_uint4(0, 0, 0, 0);
}

// The in-place side effect of the kernel above, as a pass of its own: its blocks read one another's pixels.
__global__ void normalize_kernel(float *x, long total, long HW, float3 mean, float3 std_)
{
    pdl_enter();
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int c = (int)(i / HW % 3);
    x[i] = __fdiv_rn(__fsub_rn(x[i], c == 0 ? mean.x : c == 1 ? mean.y : mean.z), c == 0 ? std_.x : c == 1 ? std_.y : std_.z);
}

// Space-to-depth by two of RGB bytes (any sides): one thread per stored pixel, its twelve bytes as three 2-byte words a row where
// the address and the row pitch allow it, everything unrolled.  (preprocess_s2d_any_kernel, which steps through channels and blocks of any size, took
// 123 us in uint8 for 256 pictures of 224 x 224, 89 MB.)
template <typename T>
__global__ void __launch_bounds__(256) preprocess_s2d_bytes_kernel(const S2dArgs a, T *y)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const int H2 = (a.H + 1) / 2, W2 = (a.W + 1) / 2;
    const long pix = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= (long)a.N * H2 * a.row_pitch) return;
    const long n = pix / ((long)H2 * a.row_pitch);
    const int rem = (int)(pix - n * (long)H2 * a.row_pitch), bh = rem / a.row_pitch, bw = rem - bh * a.row_pitch - a.pad_left;
    const float m[3] = {a.mean.x, a.mean.y, a.mean.z}, sd[3] = {a.std_.x, a.std_.y, a.std_.z};
    const float qs[3] = {(float)a.q_sub.x, (float)a.q_sub.y, (float)a.q_sub.z}, qm[3] = {a.q_mul.x, a.q_mul.y, a.q_mul.z};
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = 0.f;
    if (bw >= 0 && bw < W2) {
#pragma unroll
        for (int ph = 0; ph < 2; ph++) {
            const int h = 2 * bh + ph;
            const uint8_t *row = reinterpret_cast<const uint8_t *>(a.src) + ((size_t)n * a.H + h) * a.stride + 6 * (size_t)bw;
            const bool in_h = h < a.H, two = 2 * bw + 1 < a.W;
            uint32_t b[6];
            if (in_h && two && a.words) {
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const uint32_t u = __ldg(reinterpret_cast<const uint16_t *>(row) + k);
                    b[2 * k] = u & 255u;
                    b[2 * k + 1] = u >> 8;
                }
            } else {
#pragma unroll
                for (int k = 0; k < 6; k++) b[k] = in_h && (k < 3 || two) ? row[k] : 0;
            }
#pragma unroll
            for (int pw = 0; pw < 2; pw++)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const float px = (float)(a.bgr ? b[pw * 3 + 2 - c] : b[pw * 3 + c]);
                    float val;
                    if (sizeof(T) == 1) val = in_h && (pw == 0 || two) ? (float)((int)roundf(__fmul_rn(px - qs[c], qm[c])) & 255) : (float)a.q_zero;
                    else val = in_h && (pw == 0 || two) ? __fmul_rn(__fsub_rn(__fmul_rn(px, 0.003921568f), m[c]), sd[c]) : 0.f;
                    v[(ph * 2 + pw) * 3 + c] = val;
                }
        }
    }
#pragma unroll
    for (int c0 = 0; c0 < 16; c0 += VN) {
        float u[VN];
#pragma unroll
        for (int i = 0; i < VN; i++) u[i] = v[c0 + i];
        Vec<T>::store(y + pix * a.y_ld + c0, u);
    }
}

// u8 HWC images -> normalised NHWC T (thapi.c:20-46: multiply by 0.003921568f and by 1/std)
template <typename T>
__global__ void preprocess_images_kernel(const uint8_t *img, int N, int H, int W, int stride, int cp, int bgr, float3 mean,
                                         float3 istd, T *y, int y_ld)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const long pix = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= (long)N * H * W) return;
    const long n = pix / ((long)H * W);
    const int hw = (int)(pix - n * (long)H * W), h = hw / W, w = hw - h * W;
    const uint8_t *src = img + ((size_t)n * H + h) * stride + (size_t)w * cp;
    const float m[3] = {mean.x, mean.y, mean.z}, is[3] = {istd.x, istd.y, istd.z};
    float v[VN];
#pragma unroll
    for (int i = 0; i < VN; i++) {
        float val = 0.f;
        if (i < cp) {
            const int sc = bgr ? cp - 1 - i : i;
            val = __fmul_rn(__fsub_rn(__fmul_rn((float)src[sc], 0.003921568f), m[i]), is[i]);
        }
        v[i] = val;
    }
    Vec<T>::store(y + pix * y_ld, v);
    // (a pixel stored with more channels than one group: zeros behind)
#pragma unroll
    for (int i = 0; i < VN; i++) v[i] = 0.f;
    for (int c0 = VN; c0 < y_ld; c0 += VN) Vec<T>::store(y + pix * y_ld + c0, v);
}

// One YUYV frame (Y0 U Y1 V per pixel pair) -> normalised NHWC T with three channels, the arithmetic of the reference's
// table-driven converter (thapi.c:48-117): Y' = (Y-16)*298/256, R = sat(Y' + 459*(V-128)/256),
// G = sat(Y' - 137*(U-128)/256 - 55*(V-128)/256), B = sat(Y' + 541*(U-128)/256), every quotient truncated towards zero
// as C integer division does, then (byte * 0.003921568f - mean) * (1/std).  One thread per pixel pair.
template <typename T>
__global__ void preprocess_yuyv_kernel(const uint8_t *frame, int H, int W, float3 mean, float3 istd, T *y, int y_ld)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const long pair = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int W2 = W / 2;
    if (pair >= (long)H * W2) return;
    const uchar4 q = *reinterpret_cast<const uchar4 *>(frame + pair * 4);  // Y0 U Y1 V
    const int u = (int)q.y - 128, v = (int)q.w - 128;
    const int yur = 459 * v / 256, yub = 541 * u / 256, yg = -137 * u / 256 + -55 * v / 256;
    const int ys[2] = {((int)q.x - 16) * 298 / 256, ((int)q.z - 16) * 298 / 256};
    const float m[3] = {mean.x, mean.y, mean.z}, is[3] = {istd.x, istd.y, istd.z};
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int rgb[3] = {min(255, max(0, ys[k] + yur)), min(255, max(0, ys[k] + yg)), min(255, max(0, ys[k] + yub))};
        float out[VN > 4 ? VN : 4];
#pragma unroll
        for (int c = 0; c < (VN > 4 ? VN : 4); c++)
            out[c] = c < 3 ? __fmul_rn(__fsub_rn(__fmul_rn((float)rgb[c], 0.003921568f), m[c]), is[c]) : 0.f;
        // (the row of W pixels is contiguous: pixel index = 2 * pair + k)
        float vv[VN];
#pragma unroll
        for (int c = 0; c < VN; c++) vv[c] = out[c];
        Vec<T>::store(y + (pair * 2 + k) * y_ld, vv);
#pragma unroll
        for (int c = 0; c < VN; c++) vv[c] = 0.f;
        for (int c0 = VN; c0 < y_ld; c0 += VN) Vec<T>::store(y + (pair * 2 + k) * y_ld + c0, vv);
    }
}

// u8 HWC images -> quantised NHWC u8 with the static input range of the lowp image loader
// (lowp/lowp_basic.c:82-131, lowp/lowp_images.c): q = (unsigned char)(int)roundf((px - sub[c]) * mult[c])
__global__ void preprocess_images_u8_kernel(const uint8_t *img, int N, int H, int W, int stride, int bgr, int3 sub, float3 mult,
                                            uint8_t *y, int y_ld)
{
    pdl_enter();
    const long pix = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= (long)N * H * W) return;
    const long n = pix / ((long)H * W);
    const int hw = (int)(pix - n * (long)H * W), h = hw / W, w = hw - h * W;
    const uint8_t *src = img + ((size_t)n * H + h) * stride + (size_t)w * 3;
    const int sb[3] = {sub.x, sub.y, sub.z};
    const float ml[3] = {mult.x, mult.y, mult.z};
    uint32_t word = 0;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const int sc = bgr ? 2 - c : c;
        const int q = (int)roundf(__fmul_rn((float)((int)src[sc] - sb[c]), ml[c]));
        word |= (uint32_t)(q & 0xff) << (8 * c);
    }
    *reinterpret_cast<uint4 *>(y + pix * y_ld) = make_uint4(word, 0, 0, 0);
}

// Range of the normalised input (lowp_basic.c:15-29 starts both ends at 0).  A block scans a piece of one (image, channel)
// plane for its raw extremes with 16-byte loads and normalises only those two: subtraction and division by a positive
// deviation are monotone, so the extremes of the normalised values are the normalised extremes, bit for bit.
__global__ void __launch_bounds__(256) minmax_kernel(const float *x, int C, long HW, int pieces, float3 mean, float3 std_, float *minmax)
{
    pdl_enter();
    const long plane = blockIdx.x / pieces;
    const int piece = blockIdx.x % pieces, c = (int)(plane % C);
    const long per = (HW + pieces - 1) / pieces, i0 = piece * per, i1 = min(HW, i0 + per);
    const float *p = x + plane * HW;
    float mn = INFINITY, mx = -INFINITY;
    if (((HW | per) & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        for (long i = i0 + threadIdx.x * 4; i < i1; i += 1024) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(p + i));
            mn = fminf(fminf(mn, fminf(v.x, v.y)), fminf(v.z, v.w));
            mx = fmaxf(fmaxf(mx, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
        }
    } else {
        for (long i = i0 + threadIdx.x; i < i1; i += 256) {
            const float v = p[i];
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0 && mn <= mx) {
        if (c < 3) {
            const float m = c == 0 ? mean.x : c == 1 ? mean.y : mean.z, sd = c == 0 ? std_.x : c == 1 ? std_.y : std_.z;
            const float a = __fdiv_rn(__fsub_rn(mn, m), sd), b = __fdiv_rn(__fsub_rn(mx, m), sd);
            mn = fminf(a, b);
            mx = fmaxf(a, b);
        }
        // mn <= 0 <= mx is all that matters: negative floats order like their unsigned bit patterns, non-negative like signed ints
        if (mn < 0.f) atomicMax(reinterpret_cast<unsigned int *>(minmax), __float_as_uint(mn));
        if (mx > 0.f) atomicMax(reinterpret_cast<int *>(minmax + 1), __float_as_int(mx));
    }
}

// ---- NHWC Tin -> NCHW Tout through a 32x32 shared-memory transpose ---------------------------------
template <typename Tin, typename Tout>
__global__ void nhwc_to_nchw_kernel(const Tin *x, int HW, int C, int x_ld, float q_sub, float q_invmult, Tout *y,
                                    const int *status, int *status_out)
{
    pdl_enter();
    __shared__ float tile[32][33];
    if (status && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x | threadIdx.y) == 0) *status_out = *status;
    const int n = blockIdx.z, hw0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int hw = hw0 + r, c = c0 + threadIdx.x;
        float v = 0.f;
        if (hw < HW && c < C) {
            v = dt<Tin>::ld(x + ((size_t)n * HW + hw) * x_ld + c);
            if (sizeof(Tin) == 1) v = __fadd_rn(__fmul_rn(v, q_invmult), q_sub);
        }
        tile[r][threadIdx.x] = v;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int c = c0 + r, hw = hw0 + threadIdx.x;
        if (hw < HW && c < C) {
            dt<Tout>::st(y + ((size_t)n * C + c) * HW + hw, tile[threadIdx.x][r]);
        }
    }
}

// The same for one position per image (a classifier's scores): neither side needs transposing, so consecutive threads
// write consecutive values -- `y` may be pinned host memory, where scattered 4-byte stores would cost a transaction each.
template <typename Tin>
__global__ void rows_to_float_kernel(const Tin *x, long total, int C, int x_ld, float q_sub, float q_invmult, float *y,
                                     const int *status, int *status_out)
{
    pdl_enter();
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (status && i == 0) *status_out = *status;
    if (i >= total) return;
    const long n = i / C;
    float v = dt<Tin>::ld(x + n * x_ld + (i - n * C));
    if (sizeof(Tin) == 1) v = __fadd_rn(__fmul_rn(v, q_invmult), q_sub);
    y[i] = v;
}

// ---- pooling ------------------------------------------------------------------------------------------
template <typename T, bool IS_MAX>
__global__ void pool_kernel(const T *x, int N, int H, int W, int C, int x_ld, int kH, int kW, int dH, int dW, int padH,
                            int padW, int oH, int oW, int count_include_pad, T *y, int y_ld)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const int cvecs = (C + VN - 1) / VN;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long)N * oH * oW * cvecs) return;
    const int cv = (int)(idx % cvecs);
    const long opix = idx / cvecs;
    const int ow = (int)(opix % oW), oh = (int)((opix / oW) % oH);
    const long n = opix / ((long)oW * oH);
    int hs = oh * dH - padH, ws = ow * dW - padW;
    float acc[VN];
    int he, we, div = 1;
    if (IS_MAX) {
        he = min(hs + kH, H); we = min(ws + kW, W);
        hs = max(hs, 0); ws = max(ws, 0);
#pragma unroll
        for (int i = 0; i < VN; i++) acc[i] = sizeof(T) == 1 ? 0.f : -FLT_MAX;
    } else {
        he = min(hs + kH, H + padH); we = min(ws + kW, W + padW);
        const int pool = (he - hs) * (we - ws);
        hs = max(hs, 0); ws = max(ws, 0);
        he = min(he, H); we = min(we, W);
        div = count_include_pad ? pool : (he - hs) * (we - ws);
#pragma unroll
        for (int i = 0; i < VN; i++) acc[i] = 0.f;
    }
    for (int h = hs; h < he; h++)
#pragma unroll 4
        for (int w = ws; w < we; w++) {  // (unrolled: four independent loads in flight; a 7x7 global pool is latency-bound)
            float v[VN];
            Vec<T>::load(x + ((size_t)(n * H + h) * W + w) * x_ld + cv * VN, v);
#pragma unroll
            for (int i = 0; i < VN; i++) {
                if (IS_MAX) acc[i] = v[i] > acc[i] ? v[i] : acc[i];
                else acc[i] += v[i];
            }
        }
    if (!IS_MAX) {
#pragma unroll
        for (int i = 0; i < VN; i++) acc[i] = acc[i] / (float)div;
    }
    Vec<T>::store(y + (size_t)opix * y_ld + cv * VN, acc);
}

// Global average pooling (the window is the whole map): the generic kernel would walk the map's pixels one after the
// other in each thread, a chain of dependent load latencies.  Here a block owns one image and 32 channel vectors; its
// eight warps take every eighth pixel (independent loads in flight) and their partial sums meet in shared memory.
template <typename T>
__global__ void __launch_bounds__(256) global_avgpool_kernel(const T *x, int HW, int C, int x_ld, T *y, int y_ld)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    __shared__ float part[8][32][VN + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cvecs = (C + VN - 1) / VN, cv = blockIdx.y * 32 + lane;
    const long n = blockIdx.x;
    float acc[VN];
#pragma unroll
    for (int i = 0; i < VN; i++) acc[i] = 0.f;
    if (cv < cvecs)
        for (int p = warp; p < HW; p += 8) {
            float v[VN];
            Vec<T>::load(x + ((size_t)n * HW + p) * x_ld + cv * VN, v);
#pragma unroll
            for (int i = 0; i < VN; i++) acc[i] += v[i];
        }
#pragma unroll
    for (int i = 0; i < VN; i++) part[warp][lane][i] = acc[i];
    __syncthreads();
    if (warp == 0 && cv < cvecs) {
        float out[VN];
#pragma unroll
        for (int i = 0; i < VN; i++) {
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < 8; w++) s += part[w][lane][i];
            out[i] = s / (float)HW;
        }
        Vec<T>::store(y + (size_t)n * y_ld + cv * VN, out);
    }
}

// maxima of 16-byte vectors without a conversion
template <typename T2> __device__ __forceinline__ uint4 max8(const uint4 &a, const uint4 &b)
{
    uint4 r;
    const T2 *pa = reinterpret_cast<const T2 *>(&a), *pb = reinterpret_cast<const T2 *>(&b);
    T2 *pr = reinterpret_cast<T2 *>(&r);
#pragma unroll
    for (int i = 0; i < 4; i++) pr[i] = __hmax2(pa[i], pb[i]);
    return r;
}
struct U8x4 {};  // sixteen uint8 channels per 16-byte vector, maxima by __vmaxu4
template <> __device__ __forceinline__ uint4 max8<U8x4>(const uint4 &a, const uint4 &b)
{
    return make_uint4(__vmaxu4(a.x, b.x), __vmaxu4(a.y, b.y), __vmaxu4(a.z, b.z), __vmaxu4(a.w, b.w));
}
// four floats; the comparison of the general kernel, so that NaN and signed zeros come out as there
template <> __device__ __forceinline__ uint4 max8<float>(const uint4 &a, const uint4 &b)
{
    auto m = [](uint32_t p, uint32_t q) { return __uint_as_float(q) > __uint_as_float(p) ? q : p; };
    return make_uint4(m(a.x, b.x), m(a.y, b.y), m(a.z, b.z), m(a.w, b.w));
}
// uint8: the sum of a pixel's bytes (channels beyond the real ones are zero), what the next convolution's zero-point correction
// needs.  Its vectors lie in `cvecs` neighbouring lanes, a power of two up to 32; all of them call.
__device__ __forceinline__ void pixel_sum(const uint4 &v, int cvecs, bool write, int *csum)
{
    const int lane = threadIdx.x & 31;
    const uint32_t group = (cvecs == 32 ? 0xffffffffu : (1u << cvecs) - 1u) << (lane & ~(cvecs - 1));
    int sum = (int)__dp4a(v.w, 0x01010101u, __dp4a(v.z, 0x01010101u, __dp4a(v.y, 0x01010101u, __dp4a(v.x, 0x01010101u, 0u))));
    for (int d = 1; d < cvecs; d <<= 1) sum += __shfl_xor_sync(group, sum, d);
    if (write && (lane & (cvecs - 1)) == 0) *csum = sum;
}

// K x K max pooling, any stride and padding: a thread owns one 16-byte vector of an output pixel (ROWS = 2, stride 2: of two, one above
// the other, which share a row of inputs), a block a piece of an output row, so that a pixel costs one division; all of its loads are
// on their way before the first maximum.  HBM-bound.  3x3 stride 2, 112x112x64, us for threads that walked down strips of rows / for
// one row a thread / for two (* chosen):
//   fp16    1 image 6.9 / 6.8 / 6.8*    32 images 13.6 / 12.3 / 11.2*    256 images 107 / 96 / 85* (514 MB: 6.0 TB/s)
//   uint8   1 image 8.6 / 6.6* / 6.6    32 images 16.1 / 11.4* / 11.6    256 images 74 / 77 / 72*
//   fp32    1 image 5.2 / 5.1*          32 images 41 / 26*               256 images 297 / 191*   (strips: the general kernel)
// (48 registers for one row, five blocks to an SM: with 50, and four, fp32 takes 217.)
// VGG-16's five 2x2 poolings in uint8, 32 images, with the sums of the pooled pixels for the next layers: 77 us (28.6 for the first, 129
// MB: 4.5 TB/s) against 119 for the general kernel and 41 for passes of their own over its results.
template <typename T2, int K, int ROWS>
__global__ void __launch_bounds__(256, K == 3 && ROWS == 1 ? 5 : 1) maxpool_kernel(const uint4 *__restrict__ x, int H, int W, int cvecs, int x_ld, int dH, int dW, int padH, int padW,
                                                      int oH, int oW, uint32_t lowest, uint4 *__restrict__ y, int y_ld, int *csum)
{
    pdl_enter();
    constexpr int IN = 2 * (ROWS - 1) + K;  // (ROWS > 1: stride 2)
    const int rows = (oH + ROWS - 1) / ROWS, n = blockIdx.x / rows, oh0 = (blockIdx.x - n * rows) * ROWS, ih0 = oh0 * dH - padH;
    const int it = blockIdx.y * 256 + threadIdx.x, ow = it / cvecs, cv = it - ow * cvecs, iw0 = ow * dW - padW;
    const uint4 *img = x + (size_t)n * H * W * x_ld + cv;
    const uint4 none = make_uint4(lowest, lowest, lowest, lowest);
    uint4 v[IN * K];
#pragma unroll
    for (int k = 0; k < IN * K; k++) {
        const int ih = ih0 + k / K, iw = iw0 + k % K;
        v[k] = ow < oW && (unsigned)ih < (unsigned)H && (unsigned)iw < (unsigned)W ? __ldg(img + ((size_t)ih * W + iw) * x_ld) : none;
    }
    if constexpr (std::is_same<T2, float>::value) {  // in order, so that NaN is passed over wherever it stands; one row, no sums
        uint4 m = none;
#pragma unroll
        for (int k = 0; k < K * K; k++) m = max8<T2>(m, v[k]);
        if (ow < oW) y[((size_t)blockIdx.x * oW + ow) * y_ld + cv] = m;
    } else {
        // the maxima of each row's K once, also for the row that two windows share
#pragma unroll
        for (int r = 0; r < IN; r++)
#pragma unroll
            for (int k = 1; k < K; k++) v[r * K] = max8<T2>(v[r * K], v[r * K + k]);
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            uint4 m = none;
#pragma unroll
            for (int k = 0; k < K; k++) m = max8<T2>(m, v[(2 * r + k) * K]);
            const bool real = ow < oW && (ROWS == 1 || oh0 + r < oH);
            const size_t pix = (ROWS == 1 ? (size_t)blockIdx.x : (size_t)n * oH + oh0 + r) * oW + ow;
            if (real) y[pix * y_ld + cv] = m;
            if (csum) pixel_sum(m, cvecs, real, csum + pix);
        }
    }
}

// ---- y = act(x*scale[c] + shift[c]) ----------------------------------------------------------------------
template <typename T>
__global__ void affine_act_kernel(const T *x, long pixels, int C, int x_ld, const float *scale, const float *shift,
                                  thb_act act, T *y, int y_ld)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const int cvecs = (C + VN - 1) / VN;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= pixels * cvecs) return;
    const int cv = (int)(idx % cvecs);
    const long pix = idx / cvecs;
    float v[VN];
    Vec<T>::load(x + pix * x_ld + cv * VN, v);
#pragma unroll
    for (int i = 0; i < VN; i++) {
        const int c = cv * VN + i;
        if (c < C) {
            float t = v[i];
            if (scale) t = t * scale[c] + (shift ? shift[c] : 0.f);
            else if (shift) t = t + shift[c];
            v[i] = thb_apply_act(t, act.kind, act.threshold, act.value, act.alpha,
                                 act.kind == THB_ACT_PRELU ? act.slope[c] : 0.f);
        } else v[i] = 0.f;
    }
    Vec<T>::store(y + pix * y_ld + cv * VN, v);
}

__global__ void u8_threshold_kernel(const uint8_t *x, long pixels, int C, int x_ld, int thr, int val, uint8_t *y, int y_ld)
{
    pdl_enter();
    const int cvecs = (C + 15) / 16;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= pixels * cvecs) return;
    const int cv = (int)(idx % cvecs);
    const long pix = idx / cvecs;
    uint4 t = *reinterpret_cast<const uint4 *>(x + pix * x_ld + cv * 16);
    uint8_t *b = reinterpret_cast<uint8_t *>(&t);
#pragma unroll
    for (int i = 0; i < 16; i++) b[i] = (cv * 16 + i < C) ? (b[i] > thr ? b[i] : (uint8_t)val) : 0;
    *reinterpret_cast<uint4 *>(y + pix * y_ld + cv * 16) = t;
}

// uint8 a*ca + b*cb with ca, cb in {+1, -1}, both inputs and the output on the same static quantisation
// (sub = -range/2, mult = 255/range, so sub*mult = -127.5): the byte a dequantise -> float combine -> requantise chain
// gives in exact arithmetic, floor(ca*qa + cb*qb - (ca + cb - 1)*127.5) saturated to [0, 255] = `add2`/2 folded into an
// integer addend; an optional Threshold (bytes thr, val; thr < 0: none) follows.  No counterpart in the reference, whose
// lowp engine has no CAddTable.
__global__ void u8_combine_kernel(const uint8_t *a, int a_ld, const uint8_t *b, int b_ld, int ca, int cb, int addend,
                                  int thr, int val, long pixels, int C, uint8_t *y, int y_ld)
{
    pdl_enter();
    const int cvecs = (C + 15) / 16;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= pixels * cvecs) return;
    const int cv = (int)(idx % cvecs);
    const long pix = idx / cvecs;
    uint4 ta = __ldg(reinterpret_cast<const uint4 *>(a + pix * a_ld + cv * 16));
    uint4 tb = __ldg(reinterpret_cast<const uint4 *>(b + pix * b_ld + cv * 16));
    const uint8_t *pa = reinterpret_cast<const uint8_t *>(&ta), *pb = reinterpret_cast<const uint8_t *>(&tb);
    uint4 t;
    uint8_t *o = reinterpret_cast<uint8_t *>(&t);
#pragma unroll
    for (int i = 0; i < 16; i++) {
        int v = ca * (int)pa[i] + cb * (int)pb[i] + addend;
        v = min(255, max(0, v));
        if (thr >= 0) v = v > thr ? v : val;
        o[i] = (cv * 16 + i < C) ? (uint8_t)v : 0;
    }
    *reinterpret_cast<uint4 *>(y + pix * y_ld + cv * 16) = t;
}

struct CombineArgs {
    const void *x[8];
    int ld[8];
    float coef[8];
    int nin;
};
template <typename T>
__global__ void combine_kernel(CombineArgs a, long pixels, int C, T *y, int y_ld)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const int cvecs = (C + VN - 1) / VN;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= pixels * cvecs) return;
    const int cv = (int)(idx % cvecs);
    const long pix = idx / cvecs;
    float acc[VN], v[VN];
    Vec<T>::load(reinterpret_cast<const T *>(a.x[0]) + pix * a.ld[0] + cv * VN, v);
#pragma unroll
    for (int i = 0; i < VN; i++) acc[i] = a.coef[0] * v[i];
    for (int k = 1; k < a.nin; k++) {
        Vec<T>::load(reinterpret_cast<const T *>(a.x[k]) + pix * a.ld[k] + cv * VN, v);
#pragma unroll
        for (int i = 0; i < VN; i++) acc[i] = fmaf(a.coef[k], v[i], acc[i]);
    }
#pragma unroll
    for (int i = 0; i < VN; i++)
        if (cv * VN + i >= C) acc[i] = 0.f;
    Vec<T>::store(y + pix * y_ld + cv * VN, acc);
}

template <typename T>
__global__ void copy_channels_kernel(const T *x, long pixels, int cvecs, int x_ld, T *y, int y_ld)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= pixels * cvecs) return;
    const int cv = (int)(idx % cvecs);
    const long pix = idx / cvecs;
    *reinterpret_cast<uint4 *>(y + pix * y_ld + cv * VN) = *reinterpret_cast<const uint4 *>(x + pix * x_ld + cv * VN);
}

// ---- softmax over channels, one warp per pixel; exp(-d) = 1/(poly(d))^8 in double, 0 from 13 up ------------
__device__ __forceinline__ float exp_minus_approx(float d)
{
    const double x = (double)d;
    if (x < 13.0) {
        double y = 1.0 + x * (0.125 + x * (0.0078125 + x * (0.00032552083 + x * 1.0172526e-5)));
        y *= y; y *= y; y *= y;
        return (float)(1 / y);
    }
    return 0.f;
}
template <typename T>
__global__ void softmax_kernel(const T *x, long pixels, int C, int x_ld, T *y, int y_ld)
{
    pdl_enter();
    const long pix = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (pix >= pixels) return;
    const T *xp = x + pix * x_ld;
    T *yp = y + pix * y_ld;
    float mx = -FLT_MAX;
    for (int c = lane; c < C; c += 32) mx = fmaxf(mx, dt<T>::ld(xp + c));
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.f;
    for (int c = lane; c < C; c += 32) sum += exp_minus_approx(mx - dt<T>::ld(xp + c));
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float inv = 1 / sum;
    for (int c = lane; c < C; c += 32) dt<T>::st(yp + c, exp_minus_approx(mx - dt<T>::ld(xp + c)) * inv);
}

// The same with a block per pixel, for few pixels of many channels (a classifier's scores), and each exponential evaluated once: a
// warp's 32 evaluations per lane, twice, were 11 us for one pixel of 1000 channels and 18 us for 126.  Every warp then adds the
// exponentials up by itself, in softmax_kernel's order: a pixel's bits must not depend on how many pixels are in the launch, which
// differs with the sub-batches and GPUs that a batch is cut into.  (softmax_kernel in the order of a sum by blocks instead: 43 us
// for 50000 pixels of 65 channels, where it takes 31.)
template <typename T>
__global__ void __launch_bounds__(256) softmax_block_kernel(const T *x, int C, int x_ld, T *y, int y_ld)
{
    constexpr int PER = 4;  // channels a thread keeps (the launcher sends C <= 1024 here)
    __shared__ float part[8], ex[256 * PER];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    pdl_enter();
    const T *xp = x + (size_t)blockIdx.x * x_ld;
    float v[PER], mx = -FLT_MAX;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        v[i] = t + i * 256 < C ? dt<T>::ld(xp + t + i * 256) : -FLT_MAX;
        mx = fmaxf(mx, v[i]);
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) part[warp] = mx;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; w++) mx = fmaxf(mx, part[w]);
#pragma unroll
    for (int i = 0; i < PER; i++) {
        v[i] = t + i * 256 < C ? exp_minus_approx(mx - v[i]) : 0.f;
        ex[t + i * 256] = v[i];
    }
    __syncthreads();
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < 256 * PER; c += 32) sum += ex[c + lane];  // (zeros from C on)
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float inv = 1 / sum;
#pragma unroll
    for (int i = 0; i < PER; i++)
        if (t + i * 256 < C) dt<T>::st(y + (size_t)blockIdx.x * y_ld + t + i * 256, v[i] * inv);
}

// ---- col2im gather for the transposed convolution ---------------------------------------------------------
template <typename T>
__global__ void col2im_kernel(const T *cols, int N, int H, int W, int Cout, int kH, int kW, int dH, int dW, int padH,
                              int padW, int oH, int oW, int cols_ld, int Cp, float beta, const float *bias, thb_act act,
                              T *y, int y_ld)
{
    pdl_enter();
    constexpr int VN = Vec<T>::N;
    const int cvecs = Cp / VN;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long)N * oH * oW * cvecs) return;
    const int cv = (int)(idx % cvecs);
    const long opix = idx / cvecs;
    const int ow = (int)(opix % oW), oh = (int)((opix / oW) % oH);
    const long n = opix / ((long)oW * oH);
    float acc[VN];
#pragma unroll
    for (int i = 0; i < VN; i++) acc[i] = 0.f;
    for (int kh = 0; kh < kH; kh++) {
        const int hn = oh + padH - kh;
        if (hn < 0 || hn % dH) continue;
        const int h = hn / dH;
        if (h >= H) continue;
        for (int kw = 0; kw < kW; kw++) {
            const int wn = ow + padW - kw;
            if (wn < 0 || wn % dW) continue;
            const int w = wn / dW;
            if (w >= W) continue;
            float v[VN];
            Vec<T>::load(cols + ((size_t)(n * H + h) * W + w) * cols_ld + (size_t)(kh * kW + kw) * Cp + cv * VN, v);
#pragma unroll
            for (int i = 0; i < VN; i++) acc[i] += v[i];
        }
    }
#pragma unroll
    for (int i = 0; i < VN; i++) {
        const int c = cv * VN + i;
        if (c < Cout) {
            float t = acc[i];
            if (bias) t = beta * t + bias[c];
            acc[i] = thb_apply_act(t, act.kind, act.threshold, act.value, act.alpha,
                                   act.kind == THB_ACT_PRELU ? act.slope[c] : 0.f);
        } else acc[i] = 0.f;
    }
    Vec<T>::store(y + (size_t)opix * y_ld + cv * VN, acc);
}

// G lanes per pixel (a power of two up to 32): neighbouring lanes read neighbouring 16-byte chunks, so a warp's load covers
// whole pixels' contiguous bytes; bytes are summed four at a time (dp4a against ones) and the G partial sums by shuffles.
template <int G>
__global__ void u8_channel_sum_kernel(const uint8_t *x, long pixels, int C, int x_ld, int W, int row_pitch, int pad_left, int *csum)
{
    pdl_enter();
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long pix = t / G;
    const int g = (int)(t % G);
    int s = 0;
    if (pix < pixels) {
        long at = pix;
        if (row_pitch) {  // rows stored with their padding
            const long row = pix / W;
            at = row * row_pitch + pad_left + (pix - row * W);
        }
        const uint8_t *p = x + at * x_ld;
        for (int c0 = g * 16; c0 < C; c0 += G * 16) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p + c0));
            uint32_t w[4] = {v.x, v.y, v.z, v.w};
            if (c0 + 16 > C) {
                // the last chunk: bytes beyond channel C do not count
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int nreal = C - c0 - 4 * i;
                    w[i] &= nreal >= 4 ? 0xffffffffu : nreal <= 0 ? 0u : (1u << (8 * nreal)) - 1u;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) s = (int)__dp4a(w[i], 0x01010101u, (uint32_t)s);
        }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (pix < pixels && g == 0) csum[pix] = s;
}

// the same with a whole block per pixel, for the few-pixel, many-channel inputs of Linear layers
__global__ void u8_channel_sum_wide_kernel(const uint8_t *x, int C, int x_ld, int *csum)
{
    pdl_enter();
    const uint8_t *p = x + (size_t)blockIdx.x * x_ld;
    int s = 0;
    for (int c0 = threadIdx.x * 16; c0 < C; c0 += blockDim.x * 16) {
        const uint4 t = *reinterpret_cast<const uint4 *>(p + c0);
        const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int i = 0; i < 16; i++)
            if (c0 + i < C) s += (w[i >> 2] >> ((i & 3) * 8)) & 0xff;
    }
    __shared__ int part[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int tot = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) tot += part[i];
        csum[blockIdx.x] = tot;
    }
}

}  // namespace

// =================================================================================================
// The static input range of the lowp image loader: its float expressions, in its order (lowp_basic.c:102-119).
static void lowp_image_range(const float *mean3, const float *std3, float *q_sub, float *q_mult, int *sub, float *mul)
{
    float mn = 1e30f, mx = -1e30f, m;
    for (int i = 0; i < 3; i++) {
        if (-mean3[i] / std3[i] < mn) mn = -mean3[i] / std3[i];
        if ((1 - mean3[i]) / std3[i] > mx) mx = (1 - mean3[i]) / std3[i];
    }
    m = (mx - mn) ? 255 / (mx - mn) : 0;
    for (int i = 0; i < 3; i++) {
        sub[i] = (int)roundf(255 * (mean3[i] + std3[i] * mn));
        mul[i] = m / (255 * std3[i]);
    }
    *q_sub = mn;
    *q_mult = m;
}

extern "C" {

int thb_channel_align(int dtype) { return dtype == THB_F32 ? 4 : dtype == THB_U8 ? 16 : 8; }

int thb_preprocess(const float *x, float *x_inplace, int N, int C, int H, int W, const float *mean3, const float *std3,
                   int dtype, void *y, int y_ld, float q_sub, float q_mult, thb_stream s)
{
    const long HW = (long)H * W, pix = (long)N * HW;
    if (pix == 0) return THB_OK;
    float3 m = make_float3(mean3[0], mean3[1], mean3[2]), sd = make_float3(std3[0], std3[1], std3[2]);
    DISPATCH_ANY_DTYPE(dtype, (thb_launch(preprocess_kernel<T>, nblocks(pix), 256, s, x, x_inplace, N, C, HW, m, sd, (T *)y, y_ld, q_sub, q_mult)));
    return THB_LAUNCH_CHECK("preprocess_kernel");
}

int thb_preprocess_s2d_padded(const float *x, float *x_inplace, int N, int C, int H, int W, const float *mean3,
                              const float *std3, int dtype, void *y, int y_ld, int row_pitch, int pad_left, thb_stream s)
{
    if (((H | W) & 1) || pad_left < 0 || row_pitch < pad_left + W / 2) return THB_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(x_inplace)) & 7) {  // the kernel moves pairs of floats
        float q_sub = 0, q_mult = 0;
        if (dtype == THB_U8) return THB_ERR_UNSUPPORTED;
        return thb_preprocess_s2d_any(x, 0, x_inplace, N, C, H, W, 2, 0, 0, mean3, std3, dtype, y, y_ld, row_pitch, pad_left, &q_sub, &q_mult, s);
    }
    const long pix = (long)N * (H / 2) * row_pitch;
    if (pix == 0) return THB_OK;
    float3 m = make_float3(mean3[0], mean3[1], mean3[2]), sd = make_float3(std3[0], std3[1], std3[2]);
    DISPATCH_FLOAT_DTYPE(dtype, (thb_launch(preprocess_s2d_kernel<T>, nblocks(pix), 256, s, x, x_inplace, N, C, H, W, m, sd, (T *)y, y_ld, row_pitch, pad_left)));
    return THB_LAUNCH_CHECK("preprocess_s2d_kernel");
}

int thb_preprocess_s2d_u8(const float *x, float *x_inplace, int N, int C, int H, int W, const float *mean3, const float *std3,
                          void *y, int y_ld, float q_sub, float q_mult, thb_stream s)
{
    if ((H | W) & 1) return THB_ERR_ARG;
    return thb_preprocess_s2d_any(x, 0, x_inplace, N, C, H, W, 2, 0, 0, mean3, std3, THB_U8, y, y_ld, W / 2, 0, &q_sub, &q_mult, s);
}

int thb_preprocess_neigh_u8(const float *x, float *x_inplace, int N, int H, int W, const float *mean3, const float *std3, void *y,
                            int y_ld, float q_sub, float q_mult, thb_stream s)
{
    if (y_ld < 32 || y_ld % 16) return THB_ERR_ARG;
    const long pix = (long)N * H * W;
    if (pix == 0) return THB_OK;
    float3 m = make_float3(mean3[0], mean3[1], mean3[2]), sd = make_float3(std3[0], std3[1], std3[2]);
    for (int n0 = 0; n0 < N; n0 += 65535) {
        const int cnt = N - n0 < 65535 ? N - n0 : 65535;
        const dim3 grid((W + 31) / 32, (H + 7) / 8, cnt);
        thb_launch(preprocess_neigh_u8_kernel, grid, 256, s, x + (long)n0 * 3 * H * W, cnt, H, W, m, sd, (uint8_t *)y + (long)n0 * H * W * y_ld,
                   y_ld, q_sub, q_mult);
    }
    if (x_inplace) {
        const long total = pix * 3;
        thb_launch(normalize_kernel, nblocks(total), 256, s, x_inplace, total, (long)H * W, m, sd);
    }
    return THB_LAUNCH_CHECK("preprocess_neigh_u8_kernel");
}

int thb_preprocess_s2d(const float *x, float *x_inplace, int N, int C, int H, int W, const float *mean3,
                       const float *std3, int dtype, void *y, int y_ld, thb_stream s)
{
    return thb_preprocess_s2d_padded(x, x_inplace, N, C, H, W, mean3, std3, dtype, y, y_ld, W / 2, 0, s);
}

int thb_preprocess_images(const unsigned char *img, int N, int H, int W, int stride, int cp, int bgr, const float *mean3,
                          const float *std3, int dtype, void *y, int y_ld, thb_stream s)
{
    const long pix = (long)N * H * W;
    if (pix == 0) return THB_OK;
    if (cp != 1 && cp != 3) return THB_ERR_ARG;
    float3 m = make_float3(mean3[0], mean3[1], mean3[2]);
    float3 is = make_float3(1 / std3[0], 1 / std3[1], 1 / std3[2]);
    DISPATCH_FLOAT_DTYPE(dtype, (thb_launch(preprocess_images_kernel<T>, nblocks(pix), 256, s, img, N, H, W, stride, cp, bgr, m, is, (T *)y, y_ld)));
    return THB_LAUNCH_CHECK("preprocess_images_kernel");
}

int thb_preprocess_yuyv(const unsigned char *frame, int H, int W, const float *mean3, const float *std3, int dtype, void *y,
                        int y_ld, thb_stream s)
{
    if (H < 1 || W < 2 || (W & 1) || y_ld < 3 || (reinterpret_cast<uintptr_t>(frame) & 3)) return THB_ERR_ARG;
    if (dtype == THB_U8) return THB_ERR_UNSUPPORTED;  // (the reference refuses this entry point on its lowp engine)
    const long pairs = (long)H * (W / 2);
    float3 m = make_float3(mean3[0], mean3[1], mean3[2]);
    float3 is = make_float3(1 / std3[0], 1 / std3[1], 1 / std3[2]);
    DISPATCH_FLOAT_DTYPE(dtype, (thb_launch(preprocess_yuyv_kernel<T>, nblocks(pairs), 256, s, frame, H, W, m, is, (T *)y, y_ld)));
    return THB_LAUNCH_CHECK("preprocess_yuyv_kernel");
}

int thb_preprocess_images_s2d(const unsigned char *img, int N, int H, int W, int stride, int bgr, const float *mean3, const float *std3,
                              int dtype, void *y, int y_ld, int row_pitch, int pad_left, thb_stream s)
{
    if (((H | W) & 1) || y_ld < 12) return THB_ERR_ARG;
    if (dtype != THB_F16 && dtype != THB_BF16) return THB_ERR_UNSUPPORTED;
    float q_sub = 0, q_mult = 0;
    return thb_preprocess_s2d_any(img, 1, 0, N, 3, H, W, 2, stride, bgr, mean3, std3, dtype, y, y_ld, row_pitch, pad_left, &q_sub, &q_mult, s);
}

int thb_preprocess_images_lowp(const unsigned char *img, int N, int H, int W, int stride, int bgr, const float *mean3,
                               const float *std3, void *y, int y_ld, float *q_sub, float *q_mult, thb_stream s)
{
    if (y_ld % 16) return THB_ERR_ARG;
    int sub[3];
    float mul[3];
    lowp_image_range(mean3, std3, q_sub, q_mult, sub, mul);
    const long pix = (long)N * H * W;
    if (pix == 0) return THB_OK;
    thb_launch(preprocess_images_u8_kernel, nblocks(pix), 256, s, img, N, H, W, stride, bgr, make_int3(sub[0], sub[1], sub[2]),
                                                                            make_float3(mul[0], mul[1], mul[2]), (uint8_t *)y, y_ld);
    return THB_LAUNCH_CHECK("preprocess_images_u8_kernel");
}

int thb_preprocess_s2d_any(const void *src, int bytes, float *x_inplace, int N, int C, int H, int W, int f, int stride, int bgr,
                           const float *mean3, const float *std3, int dtype, void *y, int y_ld, int row_pitch, int pad_left,
                           float *q_sub, float *q_mult, thb_stream s)
{
    if (f < 2 || C < 1 || (bytes && C != 3) || y_ld % thb_channel_align(dtype) || y_ld < C * f * f) return THB_ERR_ARG;
    const int W2 = (W + f - 1) / f, H2 = (H + f - 1) / f;
    if (pad_left < 0 || row_pitch < pad_left + W2) return THB_ERR_ARG;
    S2dArgs a;
    a.src = src; a.x_inplace = bytes ? nullptr : x_inplace;
    a.N = N; a.C = C; a.H = H; a.W = W; a.f = f; a.stride = stride; a.bgr = bgr;
    a.mean = make_float3(mean3[0], mean3[1], mean3[2]);
    a.std_ = bytes ? make_float3(1 / std3[0], 1 / std3[1], 1 / std3[2]) : make_float3(std3[0], std3[1], std3[2]);
    a.y_ld = y_ld; a.row_pitch = row_pitch; a.pad_left = pad_left;
    a.words = bytes && !((reinterpret_cast<uintptr_t>(src) | (unsigned)stride) & 1);
    a.q_mult = a.zr = 0; a.q_sub = make_int3(0, 0, 0); a.q_mul = make_float3(0, 0, 0); a.q_zero = 0;
    if (dtype == THB_U8) {
        if (bytes) {
            int sub[3];
            float mul[3];
            lowp_image_range(mean3, std3, q_sub, q_mult, sub, mul);
            a.q_sub = make_int3(sub[0], sub[1], sub[2]);
            a.q_mul = make_float3(mul[0], mul[1], mul[2]);
        }
        a.q_mult = *q_mult;
        a.zr = roundf(*q_sub * *q_mult);
        a.q_zero = (int)-a.zr & 255;
    }
    if (bytes && f == 2 && y_ld == 16) {
        const long pix = (long)N * H2 * row_pitch;
        if (pix == 0) return THB_OK;
        DISPATCH_ANY_DTYPE(dtype, (thb_launch(preprocess_s2d_bytes_kernel<T>, nblocks(pix), 256, s, a, (T *)y)));
        return THB_LAUNCH_CHECK("preprocess_s2d_bytes_kernel");
    }
    const long total = (long)N * H2 * row_pitch * (y_ld / thb_channel_align(dtype));
    if (total == 0) return THB_OK;
    if (bytes) {
        DISPATCH_ANY_DTYPE(dtype, (thb_launch(preprocess_s2d_any_kernel<T, true>, nblocks(total), 256, s, a, (T *)y)));
    } else {
        DISPATCH_ANY_DTYPE(dtype, (thb_launch(preprocess_s2d_any_kernel<T, false>, nblocks(total), 256, s, a, (T *)y)));
    }
    return THB_LAUNCH_CHECK("preprocess_s2d_any_kernel");
}

int thb_minmax_normalized(const float *x, int N, int C, int H, int W, const float *mean3, const float *std3,
                          float *minmax2, thb_stream s)
{
    const long HW = (long)H * W, total = (long)N * C * HW;
    cudaError_t e = cudaMemsetAsync(minmax2, 0, 2 * sizeof(float), (cudaStream_t)s);
    if (e != cudaSuccess) return thb_note_launch(e, "minmax memset");
    if (total == 0) return THB_OK;
    float3 m = make_float3(mean3[0], mean3[1], mean3[2]), sd = make_float3(std3[0], std3[1], std3[2]);
    // pieces of a plane per block: enough blocks for a few waves, pieces a multiple of four elements long where possible
    const long planes = (long)N * C;
    int pieces = (int)((148L * 16 + planes - 1) / planes);
    if (pieces < 1) pieces = 1;
    while (pieces > 1 && ((HW + pieces - 1) / pieces < 4096 || (HW % (4L * pieces)))) pieces--;
    if (planes * pieces > 0x7fffffffL) return THB_ERR_UNSUPPORTED;
    thb_launch(minmax_kernel, (unsigned)(planes * pieces), 256, s, x, C, HW, pieces, m, sd, minmax2);
    return THB_LAUNCH_CHECK("minmax_kernel");
}

int thb_postprocess_status(const void *x, int dtype, int N, int H, int W, int C, int x_ld, float q_sub, float q_invmult,
                           float *y, const int *status, int *status_out, thb_stream s)
{
    const int HW = H * W;
    if ((long)N * HW * C == 0) return THB_OK;
    if (HW == 1) {
        const long total = (long)N * C;
        DISPATCH_ANY_DTYPE(dtype, (thb_launch(rows_to_float_kernel<T>, nblocks(total), 256, s, (const T *)x, total, C, x_ld, q_sub, q_invmult, y, status, status_out)));
        return THB_LAUNCH_CHECK("rows_to_float_kernel");
    }
    dim3 grid((HW + 31) / 32, (C + 31) / 32, N), block(32, 8);
    DISPATCH_ANY_DTYPE(dtype, (thb_launch(nhwc_to_nchw_kernel<T, float>, grid, block, s, (const T *)x, HW, C, x_ld, q_sub, q_invmult, y, status, status_out)));
    return THB_LAUNCH_CHECK("nhwc_to_nchw_kernel");
}

int thb_postprocess(const void *x, int dtype, int N, int H, int W, int C, int x_ld, float q_sub, float q_invmult,
                    float *y, thb_stream s)
{
    return thb_postprocess_status(x, dtype, N, H, W, C, x_ld, q_sub, q_invmult, y, 0, 0, s);
}

int thb_to_nchw(int dtype, const void *x, int N, int H, int W, int C, int x_ld, void *y, thb_stream s)
{
    const int HW = H * W;
    if ((long)N * HW * C == 0) return THB_OK;
    dim3 grid((HW + 31) / 32, (C + 31) / 32, N), block(32, 8);
    DISPATCH_ANY_DTYPE(dtype, (thb_launch(nhwc_to_nchw_kernel<T, T>, grid, block, s, (const T *)x, HW, C, x_ld, 0.f, 1.f, (T *)y, nullptr, nullptr)));
    return THB_LAUNCH_CHECK("nhwc_to_nchw_kernel");
}

int thb_maxpool(int dtype, const void *x, int N, int H, int W, int C, int x_ld, int kH, int kW, int dH, int dW, int padH,
                int padW, int oH, int oW, void *y, int y_ld, thb_stream s)
{
    return thb_maxpool_sums(dtype, x, N, H, W, C, x_ld, kH, kW, dH, dW, padH, padW, oH, oW, y, y_ld, 0, s);
}

int thb_maxpool_sums_supported(int C, int kH, int kW, int x_ld, int y_ld)
{
    const int cvecs = (C + 15) / 16;
    return kH == kW && (kH == 2 || kH == 3) && cvecs <= 32 && !(cvecs & (cvecs - 1)) && x_ld % 16 == 0 && y_ld % 16 == 0;
}

int thb_maxpool_sums(int dtype, const void *x, int N, int H, int W, int C, int x_ld, int kH, int kW, int dH, int dW, int padH, int padW,
                     int oH, int oW, void *y, int y_ld, int *csum, thb_stream s)
{
    const int al = thb_channel_align(dtype);
    if (csum && (dtype != THB_U8 || !thb_maxpool_sums_supported(C, kH, kW, x_ld, y_ld))) return THB_ERR_UNSUPPORTED;
    const long total = (long)N * oH * oW * ((C + al - 1) / al);
    if (total == 0) return THB_OK;
    const int cvecs = (C + al - 1) / al;
    const bool vectors = x_ld % al == 0 && y_ld % al == 0 && (((uintptr_t)x | (uintptr_t)y) & 15) == 0;
    // (uint8: the maximum starts from byte 0 as lowp_SpatialMaxPooling.c does; fp32: from the smallest finite value)
    const uint32_t lowest = dtype == THB_F16 ? 0xFC00FC00u : dtype == THB_BF16 ? 0xFF80FF80u : dtype == THB_U8 ? 0u : 0xFF7FFFFFu;
    const bool by_vectors = kH == kW && (kH == 2 || kH == 3) && vectors && (long)N * oH <= 0x7fffffffL && ((long)oW * cvecs + 255) / 256 <= 65535;
    if (csum && !by_vectors) return THB_ERR_UNSUPPORTED;  // (the other kernel knows no sums)
    if (by_vectors) {
        // two rows of outputs a thread (see maxpool_kernel); uint8 from four waves of blocks on (three of them fit an SM)
        const int pieces = (oW * cvecs + 255) / 256;
        const bool two = kH == 3 && dH == 2 && (dtype == THB_F16 || dtype == THB_BF16 || (dtype == THB_U8 && (long)N * ((oH + 1) / 2) * pieces >= 4 * 3 * 148));
        const dim3 grid((unsigned)(N * (two ? (oH + 1) / 2 : oH)), (unsigned)pieces);
#define MAXPOOL_KERNEL(K, ROWS) \
    (dtype == THB_F16 ? maxpool_kernel<__half2, K, ROWS> : dtype == THB_BF16 ? maxpool_kernel<__nv_bfloat162, K, ROWS> : dtype == THB_U8 ? maxpool_kernel<U8x4, K, ROWS> : maxpool_kernel<float, K, 1>)
        const auto kern = kH == 2 ? MAXPOOL_KERNEL(2, 1) : two ? MAXPOOL_KERNEL(3, 2) : MAXPOOL_KERNEL(3, 1);
#undef MAXPOOL_KERNEL
        thb_launch(kern, grid, 256, s, (const uint4 *)x, H, W, cvecs, x_ld / al, dH, dW, padH, padW, oH, oW, lowest, (uint4 *)y, y_ld / al, csum);
        return THB_LAUNCH_CHECK("maxpool_kernel");
    }
    DISPATCH_ANY_DTYPE(dtype, (thb_launch(pool_kernel<T, true>, nblocks(total), 256, s, (const T *)x, N, H, W, C, x_ld, kH, kW, dH, dW, padH, padW, oH, oW, 0, (T *)y, y_ld)));
    return THB_LAUNCH_CHECK("pool_kernel<max>");
}

int thb_avgpool(int dtype, const void *x, int N, int H, int W, int C, int x_ld, int kH, int kW, int dH, int dW, int padH,
                int padW, int oH, int oW, int count_include_pad, void *y, int y_ld, thb_stream s)
{
    const int al = thb_channel_align(dtype);
    const long total = (long)N * oH * oW * ((C + al - 1) / al);
    if (total == 0) return THB_OK;
    if (kH == H && kW == W && padH == 0 && padW == 0 && oH == 1 && oW == 1 && x_ld % al == 0 && y_ld % al == 0) {
        const dim3 grid((unsigned)N, (unsigned)(((C + al - 1) / al + 31) / 32));
        DISPATCH_ANY_DTYPE(dtype, (thb_launch(global_avgpool_kernel<T>, grid, 256, s, (const T *)x, H * W, C, x_ld, (T *)y, y_ld)));
        return THB_LAUNCH_CHECK("global_avgpool_kernel");
    }
    DISPATCH_ANY_DTYPE(dtype, (thb_launch(pool_kernel<T, false>, nblocks(total), 256, s, (const T *)x, N, H, W, C, x_ld, kH, kW, dH, dW, padH, padW, oH, oW,
                                    count_include_pad, (T *)y, y_ld)));
    return THB_LAUNCH_CHECK("pool_kernel<avg>");
}

int thb_affine_act(int dtype, const void *x, long pixels, int C, int x_ld, const float *scale, const float *shift,
                   const thb_act *act, void *y, int y_ld, thb_stream s)
{
    const int al = thb_channel_align(dtype);
    const long total = pixels * ((C + al - 1) / al);
    if (total == 0) return THB_OK;
    thb_act a = {THB_ACT_NONE, 0, 0, 0, nullptr};
    if (act) a = *act;
    DISPATCH_FLOAT_DTYPE(dtype, (thb_launch(affine_act_kernel<T>, nblocks(total), 256, s, (const T *)x, pixels, C, x_ld, scale, shift, a, (T *)y, y_ld)));
    return THB_LAUNCH_CHECK("affine_act_kernel");
}

int thb_u8_threshold(const void *x, long pixels, int C, int x_ld, int thr, int val, void *y, int y_ld, thb_stream s)
{
    const long total = pixels * ((C + 15) / 16);
    if (total == 0) return THB_OK;
    thb_launch(u8_threshold_kernel, nblocks(total), 256, s, (const uint8_t *)x, pixels, C, x_ld, thr, val,
                                                                     (uint8_t *)y, y_ld);
    return THB_LAUNCH_CHECK("u8_threshold_kernel");
}

int thb_u8_combine(const void *a, int a_ld, const void *b, int b_ld, int ca, int cb, int thr, int val, long pixels, int C,
                   void *y, int y_ld, thb_stream s)
{
    if ((ca != 1 && ca != -1) || (cb != 1 && cb != -1)) return THB_ERR_UNSUPPORTED;
    const long total = pixels * ((C + 15) / 16);
    if (total == 0) return THB_OK;
    /* floor(-(ca + cb - 1) * 127.5): +1+1 -> -128, +1-1 -> +127, -1-1 -> +382 */
    const int twice = -(ca + cb - 1) * 255;
    const int addend = twice >= 0 ? twice / 2 : -((-twice + 1) / 2);
    thb_launch(u8_combine_kernel, nblocks(total), 256, s, (const uint8_t *)a, a_ld, (const uint8_t *)b, b_ld, ca, cb,
                                                                   addend, thr, val, pixels, C, (uint8_t *)y, y_ld);
    return THB_LAUNCH_CHECK("u8_combine_kernel");
}

int thb_combine(int dtype, int nin, const void *const *x_host, const int *ld_host, const float *coef_host, long pixels,
                int C, void *y, int y_ld, thb_stream s)
{
    if (nin < 1 || nin > 8) return THB_ERR_UNSUPPORTED;
    CombineArgs a;
    a.nin = nin;
    for (int i = 0; i < nin; i++) {
        a.x[i] = x_host[i];
        a.ld[i] = ld_host[i];
        a.coef[i] = coef_host[i];
    }
    const int al = thb_channel_align(dtype);
    const long total = pixels * ((C + al - 1) / al);
    if (total == 0) return THB_OK;
    DISPATCH_FLOAT_DTYPE(dtype, (thb_launch(combine_kernel<T>, nblocks(total), 256, s, a, pixels, C, (T *)y, y_ld)));
    return THB_LAUNCH_CHECK("combine_kernel");
}

int thb_copy_channels(int dtype, const void *x, long pixels, int C, int x_ld, void *y, int y_ld, thb_stream s)
{
    const int al = thb_channel_align(dtype);
    const int cvecs = (C + al - 1) / al;
    const long total = pixels * cvecs;
    if (total == 0) return THB_OK;
    DISPATCH_ANY_DTYPE(dtype, (thb_launch(copy_channels_kernel<T>, nblocks(total), 256, s, (const T *)x, pixels, cvecs, x_ld, (T *)y, y_ld)));
    return THB_LAUNCH_CHECK("copy_channels_kernel");
}

int thb_softmax(int dtype, const void *x, long pixels, int C, int x_ld, void *y, int y_ld, thb_stream s)
{
    if (pixels == 0) return THB_OK;
    // up to two waves of eight blocks on each of 148 SMs; beyond, a warp per pixel fills the chip (both compute the same bits)
    if (C > 64 && C <= 1024 && pixels <= 2 * 8 * 148) {
        DISPATCH_FLOAT_DTYPE(dtype, (thb_launch(softmax_block_kernel<T>, (unsigned)pixels, 256, s, (const T *)x, C, x_ld, (T *)y, y_ld)));
        return THB_LAUNCH_CHECK("softmax_block_kernel");
    }
    DISPATCH_FLOAT_DTYPE(dtype, (thb_launch(softmax_kernel<T>, nblocks(pixels * 32), 256, s, (const T *)x, pixels, C, x_ld, (T *)y, y_ld)));
    return THB_LAUNCH_CHECK("softmax_kernel");
}

int thb_col2im(int dtype, const void *cols, int N, int H, int W, int Cout, int kH, int kW, int dH, int dW, int padH,
               int padW, int oH, int oW, int cols_ld, float beta, const float *bias, const thb_act *act, void *y,
               int y_ld, thb_stream s)
{
    const int al = thb_channel_align(dtype);
    const int Cp = (Cout + al - 1) / al * al;
    const long total = (long)N * oH * oW * (Cp / al);
    if (total == 0) return THB_OK;
    thb_act a = {THB_ACT_NONE, 0, 0, 0, nullptr};
    if (act) a = *act;
    DISPATCH_FLOAT_DTYPE(dtype, (thb_launch(col2im_kernel<T>, nblocks(total), 256, s, (const T *)cols, N, H, W, Cout, kH, kW, dH, dW, padH, padW, oH, oW, cols_ld, Cp, beta,
                                    bias, a, (T *)y, y_ld)));
    return THB_LAUNCH_CHECK("col2im_kernel");
}

int thb_u8_channel_sum(const void *x, long pixels, int C, int x_ld, int *csum, thb_stream s)
{
    return thb_u8_channel_sum_rows(x, pixels, C, x_ld, 1, 0, 0, csum, s);
}

int thb_u8_channel_sum_rows(const void *x, long pixels, int C, int x_ld, int W, int row_pitch, int pad_left, int *csum, thb_stream s)
{
    if (pixels == 0) return THB_OK;
    if (W < 1 || (row_pitch && row_pitch < pad_left + W)) return THB_ERR_ARG;
    if (!row_pitch && C >= 2048 && pixels <= 65535) {
        thb_launch(u8_channel_sum_wide_kernel, (unsigned)pixels, 256, s, (const uint8_t *)x, C, x_ld, csum);
        return THB_LAUNCH_CHECK("u8_channel_sum_wide_kernel");
    }
    const int chunks = (C + 15) / 16;
#define CSUM_CASE(G)                                                                                                      \
    thb_launch(u8_channel_sum_kernel<G>, nblocks(pixels * G), 256, s, (const uint8_t *)x, pixels, C, x_ld, W, row_pitch, pad_left, csum)
    if (chunks <= 1) CSUM_CASE(1);
    else if (chunks <= 2) CSUM_CASE(2);
    else if (chunks <= 4) CSUM_CASE(4);
    else if (chunks <= 8) CSUM_CASE(8);
    else if (chunks <= 16) CSUM_CASE(16);
    else CSUM_CASE(32);
#undef CSUM_CASE
    return THB_LAUNCH_CHECK("u8_channel_sum_kernel");
}

}  // extern "C"
