// fp32 implicit-GEMM convolution by chains of FFMA: for layers that conv_f32_tc.cu does not take (few products a sum, channel counts
// that neither its copies nor its gather fit), and for callers that hold no split copy of the weights.
//
// D[pixel][cout] = sum_k A[pixel][k] * Wk[k][cout], k = tap*Cin_pad + c over NHWC fp32 activations.
//
// What bounds it is the FP32 pipe (61 TFLOP/s measured in a loop without loads) once operands reach the registers cheaply, so:
//   * a thread owns 8 pixels x 8 channels and multiplies with fma.rn.f32x2, two channels an instruction, which leaves half
//     of the issue slots to the loads and to the duplication of the pixel operand;
//   * a CTA's tile is 128 x 64, 128 x 128 or 64 x 128 (pixels x channels), the K block 32; both operands arrive by 16-byte
//     cp.async (channel chunks of pixels through the gather table, zeros outside the image) in a ring of three stages, pixel
//     rows of 128 bytes swizzled by XOR so that neither the copies nor the 16-byte reads of four k at a time meet in a bank;
//   * launches of few tiles: the K blocks of a tile are shared by the S CTAs of a thread-block cluster.  Each leaves its
//     partial tile in its shared memory, and every CTA adds the S parts of its share of the rows, in rank order, through
//     distributed shared memory (no atomics, the result does not depend on timing).
// Measured: the table at thb_conv_simt_splits.
#include "common.cuh"
#include "conv_maps.cuh"
#include <cooperative_groups.h>
#include <stdlib.h>
#include <string.h>
namespace cg = cooperative_groups;

namespace {

constexpr int BK = 32, STAGES = 3;

struct ConvSimtParams {
    const float *x, *w;
    float *y;
    const int *kinfo;
    int P, H, W, in_ld, oW, oHW, dH, dW, padH, padW, Cout, Cout_pad, out_ld, Ktot, n_kchunks;
    const float *scale, *shift, *slope, *res;
    int res_ld;
    float self_coef, res_coef;
    int act_kind;
    float act_th, act_val, act_alpha;
    int splits, pdl;
};

int g_no_split = -1;  // THB200_NO_SPLITK, read once

__device__ __forceinline__ uint64_t dup2(float a)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ uint64_t pair2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpair2(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t &c, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }

// Four channels of one pixel: y = act(self * (acc * scale + shift) + res_coef * residual), channels >= Cout zero.
struct Affine4 {
    float sc[4], sh[4], sl[4];
    __device__ Affine4(const ConvSimtParams &p, int c0)
    {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int c = c0 + j;
            sc[j] = c < p.Cout ? (p.scale ? p.scale[c] : 1.f) : 0.f;
            sh[j] = c < p.Cout ? (p.shift ? p.shift[c] : 0.f) : 0.f;
            sl[j] = (c < p.Cout && p.slope) ? p.slope[c] : 0.f;
        }
    }
    __device__ void store(const ConvSimtParams &p, int pm, int c0, const float (&acc)[4]) const
    {
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.res) r = *reinterpret_cast<const float4 *>(p.res + (size_t)pm * p.res_ld + c0);
        const float rr[4] = {r.x, r.y, r.z, r.w};
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float val = acc[j] * sc[j] + sh[j];
            if (p.res) val = p.self_coef * val + p.res_coef * rr[j];
            if (p.act_kind == THB_ACT_THRESHOLD) val = val > p.act_th ? val : p.act_val;
            else if (p.act_kind != THB_ACT_NONE) val = thb_apply_act(val, p.act_kind, p.act_th, p.act_val, p.act_alpha, sl[j]);
            v[j] = (c0 + j < p.Cout) ? val : 0.f;
        }
        *reinterpret_cast<float4 *>(p.y + (size_t)pm * p.out_ld + c0) = make_float4(v[0], v[1], v[2], v[3]);
    }
};

template <int BM, int BN, bool SPLIT>
__global__ void __launch_bounds__(BM * BN / 64, BM * BN == 128 * 64 ? 3 : 2) conv_simt_kernel(const ConvSimtParams p)
{
    constexpr int NT = BM * BN / 64, A_BYTES = BM * 128, B_BYTES = BK * BN * 4, STAGE = A_BYTES + B_BYTES;
    constexpr int A_ROWS = BM * 8 / NT, B_ROWS = BK * (BN / 4) / NT;
    extern __shared__ __align__(1024) uint8_t smem[];

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int tx = lane & 7, ty = lane >> 3;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int wm = (warp % (BM / 32)) * 32, wn = (warp / (BM / 32)) * 64;  // this warp's 32 pixels x 64 channels

    // this thread's share of the copies: one 16-byte chunk of K of A_ROWS pixel rows, B_ROWS chunks of weight rows
    const int chunk = t & 7;
    int a_ih[A_ROWS], a_iw[A_ROWS], a_pix[A_ROWS];  // position of tap (0, 0); first pixel of the image, -1: no pixel
#pragma unroll
    for (int j = 0; j < A_ROWS; j++) {
        const int pm = m0 + (t >> 3) + j * (NT / 8);
        a_pix[j] = -1;
        a_ih[j] = a_iw[j] = 0;
        if (pm < p.P) {
            const int n = pm / p.oHW, rem = pm - n * p.oHW;
            const int oh = rem / p.oW, ow = rem - oh * p.oW;
            a_ih[j] = oh * p.dH - p.padH;
            a_iw[j] = ow * p.dW - p.padW;
            a_pix[j] = n * p.H * p.W;
        }
    }
    const int b_row = t / (BN / 4), b_c = (t % (BN / 4)) * 4;

    const int nkb = (p.Ktot + BK - 1) / BK;
    const int kb0 = SPLIT ? (int)((long)nkb * blockIdx.z / gridDim.z) : 0;
    const int kb1 = SPLIT ? (int)((long)nkb * (blockIdx.z + 1) / gridDim.z) : nkb;

    auto load_b = [&](int kb, int s) {
        const uint32_t dst = smem_u32(smem + s * STAGE + A_BYTES);
#pragma unroll
        for (int j = 0; j < B_ROWS; j++) {
            const int r = b_row + j * (NT / (BN / 4)), k = kb * BK + r;
            cp_async16(dst + (r * BN + b_c) * 4, p.w + (size_t)(k < p.Ktot ? k : 0) * p.Cout_pad + n0 + b_c, k < p.Ktot ? 16u : 0u);
        }
    };
    // (the gather word of a K block is read a block ahead: the warps that multiply would wait for it)
    auto kinfo_of = [&](int kb) {
        const int g = kb * 8 + chunk;
        return g < p.n_kchunks ? __ldg(p.kinfo + g) : -1;
    };
    int ki_next = kinfo_of(kb0);
    auto load_a = [&](int kb, int s) {
        const int ki = ki_next;
        ki_next = kinfo_of(kb + 1);
        const int dh = (ki >> 24) & 0x7f, dw = (ki >> 16) & 0xff, coff = (ki & 0xffff) * 4;
        const uint32_t dst = smem_u32(smem + s * STAGE);
#pragma unroll
        for (int j = 0; j < A_ROWS; j++) {
            const int r = (t >> 3) + j * (NT / 8);
            const int ih = a_ih[j] + dh, iw = a_iw[j] + dw;
            const bool ok = ki >= 0 && a_pix[j] >= 0 && (unsigned)ih < (unsigned)p.H && (unsigned)iw < (unsigned)p.W;
            const float *src = ok ? p.x + (size_t)(a_pix[j] + ih * p.W + iw) * p.in_ld + coff : p.x;
            cp_async16(dst + r * 128 + ((chunk ^ (r & 7)) << 4), src, ok ? 16u : 0u);
        }
    };

    // (weights do not depend on the launch before: their first copies go out ahead of the wait)
    int next = kb0;
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++)
        if (kb0 + s < kb1) load_b(kb0 + s, s);
    if (p.pdl) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) {
        if (next < kb1) load_a(next++, s);
        cp_async_commit();
    }

    uint64_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0;

    int s = 0;
    for (int kb = kb0; kb < kb1; kb++) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        {
            const int ns = s == 0 ? STAGES - 1 : s - 1;  // the stage everyone has just left
            if (next < kb1) {
                load_b(next, ns);
                load_a(next, ns);
                next++;
            }
            cp_async_commit();
        }
        const uint8_t *sA = smem + s * STAGE + (wm + ty) * 128;
        const float *sB = reinterpret_cast<const float *>(smem + s * STAGE + A_BYTES) + wn + tx * 4;
#pragma unroll
        for (int kc = 0; kc < 8; kc++) {
            const int off0 = (kc ^ ty) << 4, off1 = off0 ^ 64;  // rows ty + 4i: (row & 7) is ty for even i, ty + 4 for odd
            float4 a[8];
#pragma unroll
            for (int i = 0; i < 8; i++) a[i] = *reinterpret_cast<const float4 *>(sA + i * 512 + (i & 1 ? off1 : off0));
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float4 b0 = *reinterpret_cast<const float4 *>(sB + (kc * 4 + k) * BN);
                const float4 b1 = *reinterpret_cast<const float4 *>(sB + (kc * 4 + k) * BN + 32);
                const uint64_t b[4] = {pair2(b0.x, b0.y), pair2(b0.z, b0.w), pair2(b1.x, b1.y), pair2(b1.z, b1.w)};
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const uint64_t av = dup2(k == 0 ? a[i].x : k == 1 ? a[i].y : k == 2 ? a[i].z : a[i].w);
#pragma unroll
                    for (int j = 0; j < 4; j++) fma2(acc[i][j], av, b[j]);
                }
            }
        }
        if (++s == STAGES) s = 0;
    }
    cp_async_wait<0>();

    if (!SPLIT) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int c0 = n0 + wn + tx * 4 + 32 * h;
            if (c0 >= p.Cout) continue;
            const Affine4 f(p, c0);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int pm = m0 + wm + ty + 4 * i;
                if (pm >= p.P) continue;
                const float2 u = unpair2(acc[i][2 * h]), v = unpair2(acc[i][2 * h + 1]);
                const float o[4] = {u.x, u.y, v.x, v.y};
                f.store(p, pm, c0, o);
            }
        }
        return;
    }
    float *red = reinterpret_cast<float *>(smem);  // this CTA's part of the tile, [BM][BN], over the stages
    __syncthreads();                               // (everyone has left them)
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float2 u = unpair2(acc[i][2 * h]), v = unpair2(acc[i][2 * h + 1]);
            *reinterpret_cast<float4 *>(red + (wm + ty + 4 * i) * BN + wn + tx * 4 + 32 * h) = make_float4(u.x, u.y, v.x, v.y);
        }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int S = (int)gridDim.z, rows = BM / S, r0 = (int)blockIdx.z * rows;
    for (int it = t; it < rows * (BN / 4); it += NT) {
        const int r = r0 + it / (BN / 4), c = (it % (BN / 4)) * 4, pm = m0 + r, c0 = n0 + c;
        if (pm >= p.P || c0 >= p.Cout) continue;
        float acc4[4] = {0.f, 0.f, 0.f, 0.f};
        for (int q = 0; q < S; q++) {
            const float4 v = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(red, q) + r * BN + c);
            acc4[0] += v.x; acc4[1] += v.y; acc4[2] += v.z; acc4[3] += v.w;
        }
        const Affine4 f(p, c0);
        f.store(p, pm, c0, acc4);
    }
    cluster.sync();  // the parts must outlive the reads above
}

template <int BM, int BN, bool SPLIT> int launch_simt(const ConvSimtParams &p, int sms, cudaStream_t st)
{
    auto kern = conv_simt_kernel<BM, BN, SPLIT>;
    constexpr int need = STAGES * (BM * 128 + BK * BN * 4);
    static bool set[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 115712);
        if (e == cudaSuccess && SPLIT) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return thb_note_launch(e, "conv_simt_kernel attributes");
        if (dev >= 0 && dev < 64) set[dev] = true;
    }
    // A launch of one to two CTAs per SM: three would fit, and the scheduler packs clusters before it spreads them (240 CTAs in
    // clusters of two ran on 80 SMs: 90 us instead of 65), so they ask for the shared memory that leaves room for two.
    const long ctas = (long)((p.P + BM - 1) / BM) * (p.Cout_pad / BN) * p.splits;
    const int smem = ctas > sms && ctas <= 2L * sms && need < 115712 ? 115712 : need;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.P + BM - 1) / BM, p.Cout_pad / BN, p.splits);
    cfg.blockDim = dim3(BM * BN / 64);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (SPLIT) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = p.splits;
        n++;
    }
    if (p.pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, p);
    return thb_note_launch(le != cudaSuccess ? le : cudaGetLastError(), "conv_simt_kernel");
}

}  // namespace

// (library-internal: thb_conv_reload_knobs() calls it so that a test can switch THB200_NO_SPLITK between cases)
extern "C" void thb_simt_reload_knobs(void) { g_no_split = -1; }

// A split launch works on tiles of 64 pixels x 128 channels where it can: fewer wasted rows (49 pixels of a 7 x 7 map, 169 of a
// 13 x 13 one), and 2 to 5 % where the rows come out even.  us, 128 x 64 / 64 x 128: 3x3 512->512 @7x7, 1 image 32.1 / 19.2;
// 384->256 @13x13, 1 image 26.2 / 15.9; 256->256 @14x14, 2 images 29.9 / 20.3, 8 images 61.6 / 58.3; 128->128 @29x29, 9 images
// 62.9 / 61.4.
static bool low_tiles(const thb_conv_desc *d) { return d->Cout_pad % 128 == 0; }

// The reduction split while that leaves at most three CTAs to an SM (what its registers hold), in 16 parts where that leaves two at
// most.  Tiles are those of a split launch (low_tiles): 64 x 128 for 128, 256 and 512 output channels, 128 x 64 for 64 and 192.
// Measured, us in 1 / 2 / 4 / 8 / 16 parts (16 in clusters beyond the portable size); * the rule's choice:
//   64->64 3x3 @57x57, 9 images, 229 tiles of 18 K blocks      61* / 65 / 66 / 80 / 132
//   128->128 3x3 @29x29, 9 images, 119 of 36                   65 / 62* / 60 / 68 / 89
//   256->256 3x3 @15x15, 9 images, 64 of 72                   126 / 67 / 60* / 73 / 83
//   512->512 3x3 @8x8, 9 images, 36 of 144                    252 / 128 / 115 / 88* / 87
//   64->192 5x5 @27x27, 1 image, 18 of 50                      89 / 49 / 28 / 27 / 27*
//   256->256 3x3 @14x14, 2 images, 14 of 72                   124 / 67 / 35 / 20 / 21*
//   384->256 3x3 @13x13, 1 image, 6 of 108                    188 / 97 / 50 / 28 / 17*
//   512->512 3x3 @7x7, 1 image, 4 of 144                      250 / 127 / 65 / 35 / 20*
// Unsplit large layers: tiles of 128 channels (128->128 3x3 @28x28, 64 images: 332 with 64, 320 with 128).
extern "C" int thb_conv_simt_splits(const thb_conv_desc *d)
{
    if (g_no_split < 0) {
        const char *e = getenv("THB200_NO_SPLITK");
        g_no_split = e && atoi(e) ? 1 : 0;
    }
    const int sms = thb_conv_launch_knobs().sms, nkb = (d->Ktot_pad + BK - 1) / BK;
    const long P = (long)d->N * d->oH * d->oW;
    const long tiles = low_tiles(d) ? (P + 63) / 64 * (d->Cout_pad / 128) : (P + 127) / 128 * (d->Cout_pad / 64);
    int S = 1;
    if (!g_no_split) {
        while (S < 8 && tiles * 2 * S <= 3L * sms && nkb >= 2 * S) S *= 2;
        if (S == 8 && tiles * 16 <= 2L * sms && nkb >= 32) S = 16;
    }
    return S;
}

extern "C" int thb_conv_fwd_simt(const thb_conv_desc *d, const void *x, void *y, thb_stream s)
{
    if (!d->w || !d->kinfo) return THB_ERR_ARG;
    if (d->in_ld % 4 || d->out_ld % 4 || (d->res && d->res_ld % 4)) return THB_ERR_ARG;
    ConvSimtParams p;
    memset(&p, 0, sizeof(p));
    p.x = (const float *)x; p.w = (const float *)d->w; p.y = (float *)y; p.kinfo = d->kinfo;
    p.P = d->N * d->oH * d->oW;
    p.H = d->H; p.W = d->W; p.in_ld = d->in_ld; p.oW = d->oW; p.oHW = d->oH * d->oW;
    p.dH = d->dH; p.dW = d->dW; p.padH = d->padH; p.padW = d->padW;
    p.Cout = d->Cout; p.Cout_pad = d->Cout_pad; p.out_ld = d->out_ld;
    p.Ktot = d->Ktot_pad; p.n_kchunks = d->Ktot_pad / 4;
    p.scale = d->scale; p.shift = d->shift; p.slope = d->act.kind == THB_ACT_PRELU ? d->act.slope : nullptr;
    p.res = (const float *)d->res; p.res_ld = d->res_ld; p.self_coef = d->self_coef; p.res_coef = d->res_coef;
    p.act_kind = d->act.kind; p.act_th = d->act.threshold; p.act_val = d->act.value; p.act_alpha = d->act.alpha;
    if (p.P <= 0) return THB_OK;
    const ThbConvLaunch kn = thb_conv_launch_knobs();
    p.pdl = kn.pdl;
    const cudaStream_t st = (cudaStream_t)s;
    const long tiles = (long)((p.P + 127) / 128) * (d->Cout_pad / 64);
    p.splits = d->splits > 0 && d->splits <= 16 && !(d->splits & (d->splits - 1)) ? d->splits : thb_conv_simt_splits(d);
    // (64 x 128 tiles give the same sums as 128 x 64 ones)
    if (p.splits > 1) return low_tiles(d) ? launch_simt<64, 128, true>(p, kn.sms, st) : launch_simt<128, 64, true>(p, kn.sms, st);
    if (d->Cout_pad % 128 == 0 && tiles >= 200) return launch_simt<128, 128, false>(p, kn.sms, st);
    return launch_simt<128, 64, false>(p, kn.sms, st);
}
