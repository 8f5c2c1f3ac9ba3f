// Patches of an image batch (im2col) for NormDistConv, and the sum back onto the image: one launch for the whole
// batch (PyTorch's unfold launches once per image: 128 launches and 0.9 ms for 128 small images), plus the index
// lists of the (channel, position) plane that the mean shift of a spatial layer works on.
#include "common.cuh"
#include "launch.h"

namespace snb {

struct PatchGeo {
    int B, C, H, W, kh, kw, stride, pad, dil, oh, ow;
};

// out [B][C kh kw][oh ow]; consecutive threads take consecutive output positions.
__global__ void __launch_bounds__(256) unfold_kernel(const float* __restrict__ x, float* __restrict__ out, PatchGeo q, long long n) {
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += 256ll * gridDim.x) {
        int t = (int)(i % ((long long)q.oh * q.ow));
        long long r = i / ((long long)q.oh * q.ow);
        const int ox = t % q.ow, oy = t / q.ow;
        const int j = (int)(r % q.kw);
        r /= q.kw;
        const int k = (int)(r % q.kh);
        r /= q.kh;                                           // b * C + c
        const int y = oy * q.stride - q.pad + k * q.dil, xx = ox * q.stride - q.pad + j * q.dil;
        out[i] = (y >= 0 && y < q.H && xx >= 0 && xx < q.W) ? x[(r * q.H + y) * q.W + xx] : 0.f;
    }
}

// gx [B][C][H][W]: every pixel adds up the patches it is part of, in kernel order.
__global__ void __launch_bounds__(256) fold_kernel(const float* __restrict__ g, float* __restrict__ gx, PatchGeo q, long long n) {
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += 256ll * gridDim.x) {
        const int xx = (int)(i % q.W);
        const int y = (int)(i / q.W % q.H);
        const long long bc = i / q.W / q.H;
        float sum = 0.f;
        for (int k = 0; k < q.kh; k++) {
            const int ty = y + q.pad - k * q.dil;
            if (ty < 0 || ty % q.stride || ty / q.stride >= q.oh) continue;
            for (int j = 0; j < q.kw; j++) {
                const int tx = xx + q.pad - j * q.dil;
                if (tx < 0 || tx % q.stride || tx / q.stride >= q.ow) continue;
                sum += g[(((bc * q.kh + k) * q.kw + j) * q.oh + ty / q.stride) * q.ow + tx / q.stride];
            }
        }
        gx[i] = sum;
    }
}

// index [S][G][kept] within-group channels -> [S][G * kept * hw] entries channel * hw + position, still ascending.
__global__ void __launch_bounds__(256) plane_index_kernel(const int* __restrict__ index, int G, int kept, int per_group, int hw,
                                                          int* __restrict__ out, long long n) {
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += 256ll * gridDim.x) {
        const int pos = (int)(i % hw);
        const long long e = i / hw;                          // (s * G + g) * kept + k
        const int g = (int)(e / kept % G);
        out[i] = (index[e] + g * per_group) * hw + pos;
    }
}

static int patch_blocks(long long n) { return (int)((n + 255) / 256 < 2368 ? (n + 255) / 256 : 2368); }

static int make_patch_geo(int B, int C, int H, int W, int kh, int kw, int stride, int pad, int dil, PatchGeo* q) {
    if (B <= 0 || C <= 0 || H <= 0 || W <= 0 || kh <= 0 || kw <= 0 || stride <= 0 || pad < 0 || dil <= 0) return SNB_ERR_BAD_SHAPE;
    const int oh = (H + 2 * pad - dil * (kh - 1) - 1) / stride + 1, ow = (W + 2 * pad - dil * (kw - 1) - 1) / stride + 1;
    if (H + 2 * pad < dil * (kh - 1) + 1 || W + 2 * pad < dil * (kw - 1) + 1) return SNB_ERR_BAD_SHAPE;
    *q = PatchGeo{B, C, H, W, kh, kw, stride, pad, dil, oh, ow};
    return SNB_OK;
}

}  // namespace snb

using namespace snb;

extern "C" int snb_unfold(const float* x, int B, int C, int H, int W, int kh, int kw, int stride, int pad, int dil, float* out,
                          void* stream) {
    if (!x || !out) return SNB_ERR_NULL_POINTER;
    PatchGeo q;
    if (int rc = make_patch_geo(B, C, H, W, kh, kw, stride, pad, dil, &q)) return rc;
    const long long n = (long long)B * C * kh * kw * q.oh * q.ow;
    unfold_kernel<<<patch_blocks(n), 256, 0, (cudaStream_t)stream>>>(x, out, q, n);
    SNB_CUDA(launched());
    return SNB_OK;
}

extern "C" int snb_fold(const float* g, int B, int C, int H, int W, int kh, int kw, int stride, int pad, int dil, float* gx,
                        void* stream) {
    if (!g || !gx) return SNB_ERR_NULL_POINTER;
    PatchGeo q;
    if (int rc = make_patch_geo(B, C, H, W, kh, kw, stride, pad, dil, &q)) return rc;
    const long long n = (long long)B * C * H * W;
    fold_kernel<<<patch_blocks(n), 256, 0, (cudaStream_t)stream>>>(g, gx, q, n);
    SNB_CUDA(launched());
    return SNB_OK;
}

extern "C" int snb_plane_index(const int* index, int S, int G, int kept, int channels, int hw, int* out, void* stream) {
    if (!index || !out) return SNB_ERR_NULL_POINTER;
    if (S <= 0 || G <= 0 || kept <= 0 || hw <= 0 || channels <= 0 || channels % G) return SNB_ERR_BAD_SHAPE;
    const long long n = (long long)S * G * kept * hw;
    plane_index_kernel<<<patch_blocks(n), 256, 0, (cudaStream_t)stream>>>(index, G, kept, channels / G, hw, out, n);
    SNB_CUDA(launched());
    return SNB_OK;
}
