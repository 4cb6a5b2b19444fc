// Batch-small Linear (N <= 8 rows of x): y[n][m] = act((sum_k W[m][k] x[n][k]) * scale[m] + shift[m]).
// HBM-bound on the weight matrix: W is streamed once with 16-byte loads (four to eight in flight per thread, marked to leave the
// L2 first: as ordinary lines they push the convolutions' weights out, AlexNet fp32 on one image 120 -> 125 us of kernels), the x
// rows stay in L1/L2, sums are fp32.
// us per chain of launches, weights from HBM, one row of W at a time (a batch four vectors of it) / four rows (a batch a vector of
// each): 9216->4096->4096->1000 fp32, 1 row of x 37.1 / 38.3, 2 rows 45.2 / 41.5, 8 rows 101 / 78; fp16, 1 row 32.5 / 24.0, 4 rows
// 72 / 43, 8 rows 132 / 63; 25088->4096->4096->1000 fp16 54 / 43; 2048->1000 fp16, 8 rows 7.8 / 4.2; 1024->30000 fp32 44 / 21.
// (Four rows: x is read a quarter as often, and a reduction of 4096 halves fills its batches.)  A ring of cp.async in shared memory
// in place of the registers: 23.6 and 3.7 for the fp16 ones, but such copies cannot be marked: 130 us for AlexNet's forward.
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

// A CTA owns a contiguous range of rows and takes them ROWS at a time: a thread owns the vectors tid, tid + 256, ... of each, so a
// batch is a vector of every row and is multiplied by one vector of x per image.  The batch after the one being multiplied is
// already in flight (two register buffers, running on into the CTA's next rows), so the stream of loads never drains.
constexpr int ROWS = 4;
constexpr int ctas_per_sm(int nb) { return nb <= 2 ? 4 : 2; }

template <typename T, int NB>
__global__ void __launch_bounds__(256, ctas_per_sm(NB)) gemv_kernel(const T *x, int K, int x_ld, const T *w, int M, const float *scale,
                                                                    const float *shift, thb_act act, T *y, int y_ld)
{
    constexpr int VN = V16<T>::N;
    __shared__ float part[2][8][ROWS * NB];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nvec = K / VN, nkb = (nvec + 255) / 256;
    const int r0 = (int)((long long)M * blockIdx.x / gridDim.x), r1 = (int)((long long)M * (blockIdx.x + 1) / gridDim.x);
    const uint4 *wv = reinterpret_cast<const uint4 *>(w) + tid;

    int lrow = r0, lkb = 0;  // next batch to load
    auto load = [&](uint4 (&buf)[ROWS]) {
        if (lkb * 256 + tid < nvec) {
#pragma unroll
            for (int r = 0; r < ROWS; r++)
                if (lrow + r < r1) buf[r] = __ldcs(wv + (size_t)(lrow + r) * nvec + lkb * 256);
        }
        if (++lkb == nkb) { lkb = 0; lrow += ROWS; }
    };
    uint4 buf0[ROWS] = {}, buf1[ROWS] = {};
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

    auto consume = [&](const uint4 (&buf)[ROWS]) {
        const int v = kb * 256 + tid;
        if (v < nvec) {
            float wf[ROWS][VN];
#pragma unroll
            for (int r = 0; r < ROWS; r++) V16<T>::unpack(buf[r], wf[r]);
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
#define GEMV_CASE(NB)                                                                                                   \
    case NB:                                                                                                            \
        le = cudaLaunchKernelEx(&cfg, gemv_kernel<T, NB>, (const T *)x, K, x_ld, (const T *)w, M, scale, shift, a, (T *)y, y_ld); \
        break;
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
