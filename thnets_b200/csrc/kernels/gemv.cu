// Batch-small Linear (N <= 8 rows of x): y[n][m] = act((sum_k W[m][k] x[n][k]) * scale[m] + shift[m]).
// HBM-bound on the weight matrix: W is streamed once with 16-byte loads (four to eight in flight per thread, marked to leave the
// L2 first: as ordinary lines they push the convolutions' weights out, AlexNet fp32 on one image 120 -> 125 us of kernels), the x
// rows stay in L1/L2, sums are fp32.
// A CTA takes 4, 2 or 1 rows of W at a time: a batch is one vector a thread of each of four rows, two of each of two, four of one.  Four
// rows read x a quarter as often, and short reductions fill their batches; where a CTA has one or two rows in all, groups of four would
// leave most of its loads empty (the sums are the same bits).  us a launch in a chain, weights from HBM, one row at a time by an earlier
// kernel / four rows always / by the CTA's rows:
//                 fp32, 1 row of x     fp16, 1             fp32, 8             fp16, 8
//   9216->4096    22.9 / 22.7 / 22.7   18.9 / 13.2 / 13.0  61.5 / 47.5 / 41.1  80.8 / 37.3 / 33.9
//   4096->1000    3.43 / 4.27 / 3.42   3.43 / 3.25 / 2.77  9.06 / 7.07 / 6.70  12.3 / 5.81 / 5.84
//   2048->1000    2.78 / 2.78 / 2.35   2.80 / 2.58 / 2.23  6.19 / 4.45 / 4.49  7.93 / 4.21 / 4.19
//   512->1000     2.53 / 2.13 / 2.11   2.55 / 2.06 / 2.14  4.16 / 3.04 / 3.07  4.92 / 3.10 / 3.17
//   8192->300     3.09 / 5.52 / 3.84   2.82 / 4.75 / 2.74  8.21 / 9.70 / 5.98  10.7 / 8.07 / 6.56
//   1024->30000   43.7 / 20.5 / 20.4   53.3 / 19.5 / 17.5  95.4 / 65.0 / 64.1  122 / 61.8 / 62.6
// A ring of cp.async in shared memory in place of the registers: as fast, but such copies cannot be marked: 130 us for AlexNet's
// forward instead of 120.
#include "common.cuh"

namespace {

template <typename T> struct V16;
template <> struct V16<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void unpack(const uint4 &t, float (&v)[4])
    {
        v[0] = __uint_as_float(t.x); v[1] = __uint_as_float(t.y); v[2] = __uint_as_float(t.z); v[3] = __uint_as_float(t.w);
    }
};
template <> struct V16<__half> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void unpack(const uint4 &t, float (&v)[8])
    {
        const __half2 *h = reinterpret_cast<const __half2 *>(&t);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float2 f = __half22float2(h[i]);
            v[2 * i] = f.x; v[2 * i + 1] = f.y;
        }
    }
};
template <> struct V16<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void unpack(const uint4 &t, float (&v)[8])
    {
        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&t);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float2 f = __bfloat1622float2(h[i]);
            v[2 * i] = f.x; v[2 * i + 1] = f.y;
        }
    }
};

// A CTA owns a contiguous range of rows and takes them ROWS at a time: a thread owns the vectors tid, tid + 256, ... of each, and a
// batch is VECS of them of every row, each multiplied by one vector of x per image.  The batch after the one being multiplied is
// already in flight (two register buffers, running on into the CTA's next rows), so the stream of loads never drains.
constexpr int ctas_per_sm(int nb) { return nb <= 2 ? 4 : 2; }

template <typename T, int NB, int ROWS>
__global__ void __launch_bounds__(256, ctas_per_sm(NB)) gemv_kernel(const T *x, int K, int x_ld, const T *w, int M, const float *scale,
                                                                    const float *shift, thb_act act, T *y, int y_ld)
{
    constexpr int VN = V16<T>::N, VECS = 4 / ROWS;
    __shared__ float part[2][8][ROWS * NB];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nvec = K / VN, nkb = (nvec + 256 * VECS - 1) / (256 * VECS);
    const int r0 = (int)((long long)M * blockIdx.x / gridDim.x), r1 = (int)((long long)M * (blockIdx.x + 1) / gridDim.x);
    const uint4 *wv = reinterpret_cast<const uint4 *>(w) + tid;

    int lrow = r0, lkb = 0;  // next batch to load
    auto load = [&](uint4 (&buf)[4]) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = i / VECS, v = (lkb * VECS + i % VECS) * 256;
            if (v + tid < nvec && lrow + r < r1) buf[i] = __ldcs(wv + (size_t)(lrow + r) * nvec + v);
        }
        if (++lkb == nkb) { lkb = 0; lrow += ROWS; }
    };
    uint4 buf0[4] = {}, buf1[4] = {};
    // Programmatic dependent launch: the weights do not depend on the kernel before this one, so the first two
    // batches of every CTA are on their way while that kernel drains (and the next kernel of the stream may start its own
    // in the same way); x is read and y written only after the wait.
    load(buf0);
    load(buf1);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (blockIdx.x == 0) {
        // channels of the padded tail of y are kept at exact zero
        const int m = M + tid;
        if (m < (M + VN - 1) / VN * VN && m < y_ld)
            for (int n = 0; n < NB; n++) dt<T>::st(y + (size_t)n * y_ld + m, 0.f);
    }
    float acc[ROWS][NB];
#pragma unroll
    for (int r = 0; r < ROWS; r++)
#pragma unroll
        for (int n = 0; n < NB; n++) acc[r][n] = 0.f;
    int row = r0, kb = 0, parity = 0;

    auto consume = [&](const uint4 (&buf)[4]) {
#pragma unroll
        for (int j = 0; j < VECS; j++) {
            const int v = (kb * VECS + j) * 256 + tid;
            if (v >= nvec) break;
            float wf[ROWS][VN];
#pragma unroll
            for (int r = 0; r < ROWS; r++) V16<T>::unpack(buf[r * VECS + j], wf[r]);
#pragma unroll
            for (int n = 0; n < NB; n++) {
                float xf[VN];
                V16<T>::unpack(*reinterpret_cast<const uint4 *>(x + (size_t)n * x_ld + (size_t)v * VN), xf);
#pragma unroll
                for (int r = 0; r < ROWS; r++)
#pragma unroll
                    for (int i = 0; i < VN; i++) acc[r][n] = fmaf(wf[r][i], xf[i], acc[r][n]);
            }
        }
        if (++kb < nkb) return;
        // the rows are complete: warp sums, then a thread a sum adds the eight parts (buffers alternate, so that one barrier is enough)
#pragma unroll
        for (int r = 0; r < ROWS; r++)
            if (row + r < r1) {
#pragma unroll
                for (int n = 0; n < NB; n++) {
                    float t = acc[r][n];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                    if (lane == 0) part[parity][warp][r * NB + n] = t;
                    acc[r][n] = 0.f;
                }
            }
        __syncthreads();
        if (tid < ROWS * NB) {
            const int m = row + tid / NB, n = tid % NB;
            if (m < r1) {
                float t = 0.f;
#pragma unroll
                for (int q = 0; q < 8; q++) t += part[parity][q][tid];
                const float sc = scale ? scale[m] : 1.f, sh = shift ? shift[m] : 0.f;
                const float sl = act.kind == THB_ACT_PRELU ? act.slope[m] : 0.f;
                dt<T>::st(y + (size_t)n * y_ld + m, thb_apply_act(t * sc + sh, act.kind, act.threshold, act.value, act.alpha, sl));
            }
        }
        parity ^= 1;
        kb = 0;
        row += ROWS;
    };

    while (row < r1) {
        consume(buf0);
        load(buf0);
        if (row >= r1) break;
        consume(buf1);
        load(buf1);
    }
}

template <typename T>
int launch_gemv(const void *x, int N, int K, int x_ld, const void *w, int M, const float *scale, const float *shift,
                thb_act a, void *y, int y_ld, cudaStream_t st)
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    const int most = ctas_per_sm(N) * sms, grid = M < most ? M : most;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t le = cudaSuccess;
#define GEMV_CASE(NB)                                                                                                              \
    case NB: {                                                                                                                     \
        const auto kern = M <= grid ? gemv_kernel<T, NB, 1> : M <= 2 * grid ? gemv_kernel<T, NB, 2> : gemv_kernel<T, NB, 4>;       \
        le = cudaLaunchKernelEx(&cfg, kern, (const T *)x, K, x_ld, (const T *)w, M, scale, shift, a, (T *)y, y_ld);                \
        break;                                                                                                                     \
    }
    switch (N) {
        GEMV_CASE(1) GEMV_CASE(2) GEMV_CASE(3) GEMV_CASE(4) GEMV_CASE(5) GEMV_CASE(6) GEMV_CASE(7) GEMV_CASE(8)
    default: return THB_ERR_UNSUPPORTED;
    }
#undef GEMV_CASE
    if (le != cudaSuccess) return thb_note_launch(le, "gemv_kernel");
    return THB_LAUNCH_CHECK("gemv_kernel");
}

}  // namespace

extern "C" int thb_gemv_fwd(int dtype, const void *x, int N, int K, int x_ld, const void *w, int M, const float *scale,
                            const float *shift, const thb_act *act, void *y, int y_ld, thb_stream s)
{
    const int al = thb_channel_align(dtype);
    if (N < 1 || N > 8 || K % al || x_ld % al) return THB_ERR_UNSUPPORTED;
    thb_act a = {THB_ACT_NONE, 0, 0, 0, nullptr};
    if (act) a = *act;
    cudaStream_t st = (cudaStream_t)s;
    switch (dtype) {
    case THB_F32: return launch_gemv<float>(x, N, K, x_ld, w, M, scale, shift, a, y, y_ld, st);
    case THB_F16: return launch_gemv<__half>(x, N, K, x_ld, w, M, scale, shift, a, y, y_ld, st);
    case THB_BF16: return launch_gemv<__nv_bfloat16>(x, N, K, x_ld, w, M, scale, shift, a, y, y_ld, st);
    }
    return THB_ERR_UNSUPPORTED;
}
