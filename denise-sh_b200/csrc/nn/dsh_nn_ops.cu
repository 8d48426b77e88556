/*
 * dsh_nn_ops.cu — layout, activation, pooling, loss and optimiser kernels of
 * the pseudo-Hessian U-Net (everything except the tensor-core GEMM).  All
 * are bandwidth-bound grid-stride loops over NHWC tensors.
 */
#include "dsh_nn.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

namespace {

typedef __nv_bfloat16 bf16;

inline int grid_for(long long n, int threads = 256)
{
    return (int)std::max<long long>(1, std::min<long long>((n + threads - 1) / threads, 148LL * 16));
}

inline int status() { return cudaGetLastError() == cudaSuccess ? DSH_NN_OK : DSH_NN_ERR_CUDA; }

#define GRID_LOOP(i, n) \
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (long long)gridDim.x * blockDim.x)

/* The vector kernels below move 16 bytes per thread (8 bf16 or 4 floats of
 * one pixel's channels).  They serve channel counts that are a multiple of 8
 * (every layer of the U-Net), 16-byte aligned bases and fewer than 2^31
 * vectors, so that indices fit 32 bits; the scalar kernels serve the rest. */
inline bool al16(const void *p) { return ((uintptr_t)p & 15) == 0; }
inline bool vec_ok(long long nvec, int C) { return C % 8 == 0 && nvec < (1LL << 31) - (1LL << 23); }
inline unsigned vgrid(long long nvec) { return (unsigned)((nvec + 255) / 256); }
#define VEC_INDEX(i, n)                                            \
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;      \
    if (i >= (n)) return

/* one thread per (pixel, tap, channel) column entry */
__global__ void im2col_k(const bf16 *x, int B, int H, int W, int C, bf16 *col, long long ldk)
{
    const long long P = (long long)B * H * W, K = 9LL * C;
    GRID_LOOP(idx, P * K)
    {
        const long long p = idx / K;
        const int k = (int)(idx % K), tap = k / C, c = k % C;
        const int xw = (int)(p % W), yh = (int)((p / W) % H);
        const long long b = p / ((long long)W * H);
        const int yy = yh + tap / 3 - 1, xx = xw + tap % 3 - 1;
        bf16 v = __float2bfloat16_rn(0.0f);
        if (yy >= 0 && yy < H && xx >= 0 && xx < W) v = x[((b * H + yy) * W + xx) * C + c];
        col[p * ldk + k] = v;
    }
}

/* transposed: colT[k][p], consecutive threads along p */
__global__ void im2col_t_k(const bf16 *x, int B, int H, int W, int C, bf16 *colT, long long ldp)
{
    const long long P = (long long)B * H * W, K = 9LL * C;
    GRID_LOOP(idx, P * K)
    {
        const long long k = idx / P, p = idx % P;
        const int tap = (int)(k / C), c = (int)(k % C);
        const int xw = (int)(p % W), yh = (int)((p / W) % H);
        const long long b = p / ((long long)W * H);
        const int yy = yh + tap / 3 - 1, xx = xw + tap % 3 - 1;
        bf16 v = __float2bfloat16_rn(0.0f);
        if (yy >= 0 && yy < H && xx >= 0 && xx < W) v = x[((b * H + yy) * W + xx) * C + c];
        colT[k * ldp + p] = v;
    }
}

/* im2col, 8 channels per thread, threads along the columns of a pixel: every
 * store is a full 16 bytes of a contiguous run.  Bound by the 18 C bytes it
 * writes per pixel; the one-element kernel above spends its time on 64-bit
 * divisions and 2-byte accesses.  33 launches of a training step on two 400 x
 * 1200 maps, when every layer had column matrices: 37.4 ms with it, 3.2 ms with
 * this one; now the first layer and those conv3x3_tc cannot take are left. */
__global__ void im2col_v8(const uint4 *x, int H, int W, unsigned nc, unsigned n, uint4 *col, long long ldk8)
{
    VEC_INDEX(i, n);
    const unsigned per = 9 * nc, p = i / per, k = i - p * per, tap = k / nc, c = k - tap * nc;
    const unsigned row = p / W, xw = p - row * W, yh = row % H;
    const int yy = (int)yh + (int)(tap / 3) - 1, xx = (int)xw + (int)(tap % 3) - 1;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (yy >= 0 && yy < H && xx >= 0 && xx < W) v = __ldg(x + (long long)((long long)p + (yy - (int)yh) * W + xx - (int)xw) * nc + c);
    col[(long long)p * ldk8 + k] = v;
}

/* Transposed columns (TAPS 9) or a plain transpose (TAPS 1) of a tile of 128
 * pixels x 32 channels through shared memory: a thread loads 8 channels of
 * two neighbouring pixels (16 bytes each), stores eight pixel pairs, and
 * writes 16 bytes along the pixels.  Pitch 65 words: the stores of a warp (8
 * pairs x 4 vectors of 8 channels) fall into different banks.  The 17 launches
 * of a training step on two 400 x 1200 maps: 22.5 ms with the one-element
 * kernel, 2.6 ms one pixel per thread, 2.3 ms with this one (6.3 GB written). */
template <int TAPS>
__global__ void __launch_bounds__(256) transpose_v8(const uint4 *x, int H, int W, int C, int P, bf16 *yT, long long ldp)
{
    __shared__ uint32_t t[32 * 65];
    const int tap = TAPS == 9 ? blockIdx.z : 4;
    const int p0 = blockIdx.x * 128, c0 = blockIdx.y * 32;
    {
        const int pair = threadIdx.x >> 2, v8 = threadIdx.x & 3, c = c0 + 8 * v8;
        uint4 v[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int p = p0 + 2 * pair + h;
            v[h] = make_uint4(0, 0, 0, 0);
            bool in = p < P && c < C;
            long long q = p;
            if (TAPS == 9 && in) {
                const int row = p / W, xx = p - row * W + tap % 3 - 1, yy = row % H + tap / 3 - 1;
                in = yy >= 0 && yy < H && xx >= 0 && xx < W;
                q += (tap / 3 - 1) * W + tap % 3 - 1;
            }
            if (in) v[h] = __ldg(x + (q * C + c) / 8);
        }
        const uint32_t a[4] = {v[0].x, v[0].y, v[0].z, v[0].w}, b[4] = {v[1].x, v[1].y, v[1].z, v[1].w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            t[(8 * v8 + 2 * e) * 65 + pair] = __byte_perm(a[e], b[e], 0x5410);
            t[(8 * v8 + 2 * e + 1) * 65 + pair] = __byte_perm(a[e], b[e], 0x7632);
        }
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int k = threadIdx.x + 256 * h, cl = k >> 4, pv = k & 15, c = c0 + cl, p = p0 + 8 * pv;
        if (c >= C || p >= P) continue;
        bf16 *dst = yT + ((TAPS == 9 ? (long long)tap * C : 0) + c) * ldp + p;
        const uint32_t *src = t + cl * 65 + 4 * pv;
        const uint4 w = make_uint4(src[0], src[1], src[2], src[3]);
        if (p + 8 <= P) {
            *reinterpret_cast<uint4 *>(dst) = w;
        } else {
            const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int e = 0; e < 8; e++)
                if (p + e < P) reinterpret_cast<uint16_t *>(dst)[e] = (uint16_t)(u[e >> 1] >> (16 * (e & 1)));
        }
    }
}

/* 32 x 32 tile transpose through shared memory */
__global__ void transpose_k(const bf16 *y, long long P, int C, bf16 *yT, long long ldp)
{
    __shared__ bf16 t[32][33];
    const long long p0 = (long long)blockIdx.x * 32;
    const int c0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const long long p = p0 + r;
        const int c = c0 + threadIdx.x;
        t[r][threadIdx.x] = (p < P && c < C) ? y[p * C + c] : __float2bfloat16_rn(0.0f);
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int c = c0 + r;
        const long long p = p0 + threadIdx.x;
        if (c < C && p < P) yT[(long long)c * ldp + p] = t[threadIdx.x][r];
    }
}

__global__ void prep_weights_k(const float *w, int Cout, int Cin, bf16 *wb, long long ldk, bf16 *wf, long long ldf)
{
    const long long K = 9LL * Cin;
    GRID_LOOP(idx, (long long)Cout * K)
    {
        const int co = (int)(idx / K), k = (int)(idx % K);
        const bf16 v = __float2bfloat16_rn(w[idx]);
        wb[(long long)co * ldk + k] = v;
        const int tap = k / Cin, ci = k % Cin;
        wf[(long long)ci * ldf + (long long)(8 - tap) * Cout + co] = v;
    }
}

__global__ void to_bf16_k(const float *x, bf16 *y, long long n)
{
    GRID_LOOP(i, n) y[i] = __float2bfloat16_rn(x[i]);
}

__global__ void relu_bwd_k(const float *dy, const bf16 *y, bf16 *dx, float *dx32, long long n)
{
    GRID_LOOP(i, n)
    {
        const float d = __bfloat162float(y[i]) > 0.0f ? dy[i] : 0.0f;
        dx[i] = __float2bfloat16_rn(d);
        if (dx32) dx32[i] = d;
    }
}

__device__ __forceinline__ float2 bf2(uint32_t w)
{
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
__device__ __forceinline__ uint32_t pack2(float a, float b)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}

/* relu_bwd, 8 values per thread (dx32 may be dy) */
__global__ void relu_bwd_v8(const float4 *dy, const uint4 *y, uint4 *dx, float4 *dx32, unsigned n)
{
    VEC_INDEX(i, n);
    const uint4 yv = __ldg(y + i);
    float4 a = dy[2 * i], b = dy[2 * i + 1];
    const float2 y0 = bf2(yv.x), y1 = bf2(yv.y), y2 = bf2(yv.z), y3 = bf2(yv.w);
    a.x = y0.x > 0.0f ? a.x : 0.0f; a.y = y0.y > 0.0f ? a.y : 0.0f;
    a.z = y1.x > 0.0f ? a.z : 0.0f; a.w = y1.y > 0.0f ? a.w : 0.0f;
    b.x = y2.x > 0.0f ? b.x : 0.0f; b.y = y2.y > 0.0f ? b.y : 0.0f;
    b.z = y3.x > 0.0f ? b.z : 0.0f; b.w = y3.y > 0.0f ? b.w : 0.0f;
    dx[i] = make_uint4(pack2(a.x, a.y), pack2(a.z, a.w), pack2(b.x, b.y), pack2(b.z, b.w));
    if (dx32) { dx32[2 * i] = a; dx32[2 * i + 1] = b; }
}

__global__ void add_v4(float4 *y, const float4 *x, unsigned n)
{
    VEC_INDEX(i, n);
    float4 a = y[i];
    const float4 b = __ldg(x + i);
    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    y[i] = a;
}

__global__ void add_k(float *y, const float *x, long long n)
{
    GRID_LOOP(i, n) y[i] += x[i];
}

__global__ void maxpool_fwd_k(const bf16 *x, int B, int H, int W, int C, bf16 *y, unsigned char *arg)
{
    const int h = H / 2, w = W / 2;
    GRID_LOOP(idx, (long long)B * h * w * C)
    {
        const int c = (int)(idx % C);
        const long long q = idx / C;
        const int xo = (int)(q % w), yo = (int)((q / w) % h);
        const long long b = q / ((long long)w * h);
        float best = -3.0e38f;
        int a = 0;
        for (int k = 0; k < 4; k++) {
            const float v = __bfloat162float(x[((b * H + 2 * yo + k / 2) * W + 2 * xo + k % 2) * C + c]);
            if (v > best) { best = v; a = k; }
        }
        y[idx] = __float2bfloat16_rn(best);
        arg[idx] = (unsigned char)a;
    }
}

/* 8 channels of one output pixel per thread (nc = C/8) */
__global__ void maxpool_fwd_v8(const uint4 *x, int W, unsigned nc, unsigned n, uint4 *y, uint2 *arg)
{
    VEC_INDEX(i, n);
    const unsigned q = i / nc, c = i - q * nc, w = W / 2, row = q / w, xo = q - row * w;   /* row = b*(H/2) + yo */
    const uint4 *s = x + ((long long)(2 * row) * W + 2 * xo) * nc + c;
    const uint4 v[4] = {__ldg(s), __ldg(s + nc), __ldg(s + (long long)W * nc), __ldg(s + (long long)W * nc + nc)};
    uint32_t out[4], a[8];
#pragma unroll
    for (int h = 0; h < 4; h++) {
        float2 best = make_float2(-3.0e38f, -3.0e38f);
        a[2 * h] = a[2 * h + 1] = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 f = bf2(h == 0 ? v[k].x : h == 1 ? v[k].y : h == 2 ? v[k].z : v[k].w);
            if (f.x > best.x) { best.x = f.x; a[2 * h] = k; }
            if (f.y > best.y) { best.y = f.y; a[2 * h + 1] = k; }
        }
        out[h] = pack2(best.x, best.y);
    }
    y[i] = make_uint4(out[0], out[1], out[2], out[3]);
    arg[i] = make_uint2(a[0] | a[1] << 8 | a[2] << 16 | a[3] << 24, a[4] | a[5] << 8 | a[6] << 16 | a[7] << 24);
}

/* 4 channels of one output pixel per thread (nc = C/4): its four input pixels are written together */
__global__ void maxpool_bwd_v4(const float4 *dy, const uint32_t *arg, int W, unsigned nc, unsigned n, float4 *dx)
{
    VEC_INDEX(i, n);
    const unsigned q = i / nc, c = i - q * nc, w = W / 2, row = q / w, xo = q - row * w;
    const float4 d = __ldg(dy + i);
    const uint32_t a = __ldg(arg + i);
    float4 *o = dx + ((long long)(2 * row) * W + 2 * xo) * nc + c;
#pragma unroll
    for (unsigned k = 0; k < 4; k++)
        o[(k >> 1) * (long long)W * nc + (k & 1) * nc] =
            make_float4((a & 255) == k ? d.x : 0.0f, (a >> 8 & 255) == k ? d.y : 0.0f, (a >> 16 & 255) == k ? d.z : 0.0f,
                        a >> 24 == k ? d.w : 0.0f);
}

/* one input vector of 8 channels to its four output pixels */
__global__ void upsample_fwd_v8(const uint4 *x, int w, unsigned nc, unsigned n, uint4 *y)
{
    VEC_INDEX(i, n);
    const unsigned q = i / nc, c = i - q * nc, row = q / w, xs = q - row * w;
    const uint4 v = __ldg(x + i);
    uint4 *o = y + ((long long)(2 * row) * (2 * w) + 2 * xs) * nc + c;
    o[0] = v;
    o[nc] = v;
    o[2LL * w * nc] = v;
    o[2LL * w * nc + nc] = v;
}

__global__ void upsample_bwd_v4(const float4 *dy, int w, unsigned nc, unsigned n, float4 *dx)
{
    VEC_INDEX(i, n);
    const unsigned q = i / nc, c = i - q * nc, row = q / w, xs = q - row * w;
    const float4 *s = dy + ((long long)(2 * row) * (2 * w) + 2 * xs) * nc + c;
    const float4 a = __ldg(s), b = __ldg(s + nc), e = __ldg(s + 2LL * w * nc), f = __ldg(s + 2LL * w * nc + nc);
    dx[i] = make_float4(a.x + b.x + e.x + f.x, a.y + b.y + e.y + f.y, a.z + b.z + e.z + f.z, a.w + b.w + e.w + f.w);
}

/* vectors of 16 bytes: n1 of a, then n2 of b, per pixel */
__global__ void concat_v(const uint4 *a, unsigned n1, const uint4 *b, unsigned n2, unsigned n, uint4 *y)
{
    VEC_INDEX(i, n);
    const unsigned p = i / (n1 + n2), c = i - p * (n1 + n2);
    y[i] = c < n1 ? __ldg(a + p * n1 + c) : __ldg(b + p * n2 + (c - n1));
}
__global__ void split_v(const uint4 *dy, unsigned n1, unsigned n2, unsigned n, uint4 *a, uint4 *b)
{
    VEC_INDEX(i, n);
    const unsigned p = i / (n1 + n2), c = i - p * (n1 + n2);
    const uint4 v = __ldg(dy + i);
    if (c < n1) a[p * n1 + c] = v;
    else b[p * n2 + (c - n1)] = v;
}

__global__ void maxpool_bwd_k(const float *dy, const unsigned char *arg, int B, int H, int W, int C, float *dx)
{
    GRID_LOOP(idx, (long long)B * H * W * C)
    {
        const int c = (int)(idx % C);
        const long long q = idx / C;
        const int xx = (int)(q % W), yy = (int)((q / W) % H);
        const long long b = q / ((long long)W * H);
        const long long o = ((b * (H / 2) + yy / 2) * (W / 2) + xx / 2) * C + c;
        dx[idx] = (arg[o] == (yy % 2) * 2 + (xx % 2)) ? dy[o] : 0.0f;
    }
}

__global__ void upsample_fwd_k(const bf16 *x, int B, int h, int w, int C, bf16 *y)
{
    const int H = 2 * h, W = 2 * w;
    GRID_LOOP(idx, (long long)B * H * W * C)
    {
        const int c = (int)(idx % C);
        const long long q = idx / C;
        const int xx = (int)(q % W), yy = (int)((q / W) % H);
        const long long b = q / ((long long)W * H);
        y[idx] = x[((b * h + yy / 2) * w + xx / 2) * C + c];
    }
}

__global__ void upsample_bwd_k(const float *dy, int B, int h, int w, int C, float *dx)
{
    const int W = 2 * w;
    GRID_LOOP(idx, (long long)B * h * w * C)
    {
        const int c = (int)(idx % C);
        const long long q = idx / C;
        const int xs = (int)(q % w), ys = (int)((q / w) % h);
        const long long b = q / ((long long)w * h);
        const long long r0 = ((b * 2 * h + 2 * ys) * W + 2 * xs) * C + c;
        dx[idx] = dy[r0] + dy[r0 + C] + dy[r0 + (long long)W * C] + dy[r0 + (long long)W * C + C];
    }
}

__global__ void concat_k(const bf16 *a, int C1, const bf16 *b, int C2, long long P, bf16 *y)
{
    const int C = C1 + C2;
    GRID_LOOP(idx, P * C)
    {
        const long long p = idx / C;
        const int c = (int)(idx % C);
        y[idx] = c < C1 ? a[p * C1 + c] : b[p * C2 + (c - C1)];
    }
}

__global__ void split_k(const float *dy, int C1, int C2, long long P, float *da, float *db)
{
    const int C = C1 + C2;
    GRID_LOOP(idx, P * C)
    {
        const long long p = idx / C;
        const int c = (int)(idx % C);
        if (c < C1) da[p * C1 + c] = dy[idx];
        else db[p * C2 + (c - C1)] = dy[idx];
    }
}

/* one thread per pixel, 16-byte loads, products added in channel order as above (C a multiple of 8) */
__global__ void head_fwd_v8(const uint4 *x, unsigned P, int nc, const float *w, const float *b, float *out)
{
    VEC_INDEX(p, P);
    float s = 0.0f;
    for (int c = 0; c < nc; c++) {
        const uint4 v = __ldg(x + (long long)p * nc + c);
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float2 f = bf2(u[e]);
            s += f.x * __ldg(w + 8 * c + 2 * e);
            s += f.y * __ldg(w + 8 * c + 2 * e + 1);
        }
    }
    out[p] = s + b[0];
}

__global__ void head_fwd_k(const bf16 *x, long long P, int C, const float *w, const float *b, float *out)
{
    GRID_LOOP(p, P)
    {
        float s = 0.0f;
        for (int c = 0; c < C; c++) s += __bfloat162float(x[p * C + c]) * w[c];
        out[p] = s + b[0];
    }
}

/* dx[p][c] = dout[p] w[c], and per block b the partial sums
 * part[b][c] = sum over its rows of dout[p] x[p][c] (c < C) and
 * part[b][C] = sum of dout[p]: thread t of a block owns column t % (C+1) and
 * the rows r = t / (C+1) + k * (256 / (C+1)) of the block's chunk, partials
 * are combined in a fixed order, so the result does not depend on timing. */
__global__ void head_bwd_k(const float *dout, const bf16 *x, long long P, int C, const float *w, float *dx, float *part)
{
    const long long rows = (P + gridDim.x - 1) / gridDim.x;
    const long long r0 = (long long)blockIdx.x * rows, r1 = min(P, r0 + rows);
    if (C % 4 == 0 && (((uintptr_t)dx | (uintptr_t)w) & 15) == 0) {
        const unsigned nv = C / 4, n = (unsigned)max(r1 - r0, 0LL) * nv;
        float4 *o = reinterpret_cast<float4 *>(dx + r0 * C);
        const float4 *wv = reinterpret_cast<const float4 *>(w);
#pragma unroll 4
        for (unsigned i = threadIdx.x; i < n; i += blockDim.x) {
            const unsigned p = i / nv;
            const float d = __ldg(dout + r0 + p);
            const float4 v = __ldg(wv + (i - p * nv));
            o[i] = make_float4(d * v.x, d * v.y, d * v.z, d * v.w);
        }
    } else {
        for (long long idx = r0 * C + threadIdx.x; idx < r1 * C; idx += blockDim.x) {
            const long long p = idx / C;
            dx[idx] = dout[p] * w[idx % C];
        }
    }
    extern __shared__ float acc[];                 /* blockDim.x */
    const int W = C + 1, lanes = blockDim.x / W;
    float s = 0.0f;
    if ((int)threadIdx.x < lanes * W) {
        const int c = threadIdx.x % W, lane = threadIdx.x / W;
#pragma unroll 8
        for (long long p = r0 + lane; p < r1; p += lanes)
            s += c < C ? dout[p] * __bfloat162float(x[p * C + c]) : dout[p];
    }
    acc[threadIdx.x] = s;
    __syncthreads();
    if ((int)threadIdx.x < W) {
        float t = 0.0f;
        for (int lane = 0; lane < lanes; lane++) t += acc[lane * W + threadIdx.x];
        part[(long long)blockIdx.x * W + threadIdx.x] = t;
    }
}

/* per-block partial column sums of dy [P][N] (fixed order, as head_bwd_k) */
__global__ void colsum_k(const float *dy, long long P, int N, float *part)
{
    const long long rows = (P + gridDim.x - 1) / gridDim.x;
    const long long r0 = (long long)blockIdx.x * rows, r1 = min(P, r0 + rows);
    for (int n = threadIdx.x; n < N; n += blockDim.x) {
        float s = 0.0f;
        for (long long p = r0; p < r1; p++) s += dy[p * N + n];
        part[(long long)blockIdx.x * N + n] = s;
    }
}

/* The same sums in the same order (one thread per column, rows in sequence),
 * fed through shared memory: the whole block copies tiles of 4096 floats
 * ahead with cp.async while the first N threads add the current one.  N a
 * multiple of 4, at most 256.  With each column's thread loading its own rows
 * 32 of 256 threads worked when N = 32: 2.45 ms in the 17 launches of a
 * training step on two 400 x 1200 maps; now bound by the chain of additions. */
constexpr int CS_TILE = 4096;
__global__ void __launch_bounds__(256) colsum_tiles(const float *dy, long long P, int N, float *part)
{
    __shared__ __align__(16) float sh[2][CS_TILE];
    const long long rows = (P + gridDim.x - 1) / gridDim.x;
    const long long r0 = (long long)blockIdx.x * rows, r1 = min(P, r0 + rows);
    const int tr = CS_TILE / N;                          /* rows of a tile */
    const long long ntile = r1 > r0 ? (r1 - r0 + tr - 1) / tr : 0;
    auto fetch = [&](long long t) {
        if (t < ntile) {
            const long long p = r0 + t * tr;
            const int n4 = (int)(min((long long)tr, r1 - p) * N / 4);
            const float4 *src = reinterpret_cast<const float4 *>(dy + p * N);
            for (int k = threadIdx.x; k < n4; k += blockDim.x) {
                const uint32_t d = (uint32_t)__cvta_generic_to_shared(&sh[t & 1][4 * k]);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + k) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float s = 0.0f;
    fetch(0);
    for (long long t = 0; t < ntile; t++) {
        fetch(t + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const int n = (int)min((long long)tr, r1 - (r0 + t * tr));
        if ((int)threadIdx.x < N) {
            const float *col = &sh[t & 1][threadIdx.x];
#pragma unroll 16
            for (int p = 0; p < n; p++) s += col[p * N];
        }
        __syncthreads();
    }
    if ((int)threadIdx.x < N) part[(long long)blockIdx.x * N + threadIdx.x] = s;
}

/* g[n] += sum over blocks of part[b*stride + n], blocks in order */
__global__ void sum_parts_k(const float *part, int nblocks, int N, int stride, float *g)
{
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        float s = 0.0f;
        for (int b = 0; b < nblocks; b += 37) {          /* DSH_NN_RED_BLOCKS = 8 x 37: 37 loads in flight */
            float v[37];
#pragma unroll
            for (int k = 0; k < 37; k++) v[k] = part[(long long)(b + k) * stride + n];
#pragma unroll
            for (int k = 0; k < 37; k++) s += v[k];
        }
        g[n] += s;
    }
}

__global__ void mse_k(const float *pred, const float *target, const unsigned char *mask, long long n, float count,
                      float *grad, float *loss)
{
    __shared__ float red[256];
    float s = 0.0f;
    GRID_LOOP(i, n)
    {
        const bool on = !mask || mask[i];
        const float d = on ? pred[i] - target[i] : 0.0f;
        grad[i] = 2.0f * d / count;
        s += d * d;
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, red[0] / count);
}

__global__ void adam_k(float *w, float *m, float *v, const float *g, int rows, int cols, int transposed, float lr,
                       float b1, float b2, float eps, float c1, float c2)
{
    GRID_LOOP(i, (long long)rows * cols)
    {
        const long long r = i / cols, c = i % cols;
        const float gr = transposed ? g[c * rows + r] : g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gr;
        const float vi = b2 * v[i] + (1.0f - b2) * gr * gr;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

}  // namespace

#define ST ((cudaStream_t)stream)

extern "C" int dsh_nn_im2col(const void *x, int B, int H, int W, int C, void *col, long long ldk, void *stream)
{
    if (!x || !col || B <= 0 || H <= 0 || W <= 0 || C <= 0 || ldk < 9LL * C) return DSH_NN_ERR_PARAM;
    const long long n = (long long)B * H * W * 9 * C;
    if (vec_ok(n / 8, C) && ldk % 8 == 0 && al16(x) && al16(col)) {
        im2col_v8<<<vgrid(n / 8), 256, 0, ST>>>((const uint4 *)x, H, W, C / 8, (unsigned)(n / 8), (uint4 *)col, ldk / 8);
        return status();
    }
    im2col_k<<<grid_for(n), 256, 0, ST>>>((const bf16 *)x, B, H, W, C, (bf16 *)col, ldk);
    return status();
}

extern "C" int dsh_nn_im2col_t(const void *x, int B, int H, int W, int C, void *colT, long long ldp, void *stream)
{
    if (!x || !colT || B <= 0 || H <= 0 || W <= 0 || C <= 0 || ldp < (long long)B * H * W) return DSH_NN_ERR_PARAM;
    const long long n = (long long)B * H * W * 9 * C, P = (long long)B * H * W;
    if (vec_ok(P, C) && ldp % 8 == 0 && al16(x) && al16(colT) && C <= 32 * 65535) {
        transpose_v8<9><<<dim3((unsigned)((P + 127) / 128), (unsigned)((C + 31) / 32), 9), 256, 0, ST>>>(
            (const uint4 *)x, H, W, C, (int)P, (bf16 *)colT, ldp);
        return status();
    }
    im2col_t_k<<<grid_for(n), 256, 0, ST>>>((const bf16 *)x, B, H, W, C, (bf16 *)colT, ldp);
    return status();
}

extern "C" int dsh_nn_transpose(const void *y, long long P, int C, void *yT, long long ldp, void *stream)
{
    if (!y || !yT || P <= 0 || C <= 0 || ldp < P) return DSH_NN_ERR_PARAM;
    if (vec_ok(P, C) && ldp % 8 == 0 && al16(y) && al16(yT) && C <= 32 * 65535) {
        transpose_v8<1><<<dim3((unsigned)((P + 127) / 128), (unsigned)((C + 31) / 32), 1), 256, 0, ST>>>(
            (const uint4 *)y, 1, 1, C, (int)P, (bf16 *)yT, ldp);
        return status();
    }
    dim3 grid((unsigned)((P + 31) / 32), (unsigned)((C + 31) / 32));
    transpose_k<<<grid, dim3(32, 8), 0, ST>>>((const bf16 *)y, P, C, (bf16 *)yT, ldp);
    return status();
}

extern "C" int dsh_nn_prep_weights(const float *w, int Cout, int Cin, void *wb, long long ldk, void *wf, long long ldf,
                                   void *stream)
{
    if (!w || !wb || !wf || Cout <= 0 || Cin <= 0 || ldk < 9LL * Cin || ldf < 9LL * Cout) return DSH_NN_ERR_PARAM;
    prep_weights_k<<<grid_for(9LL * Cin * Cout), 256, 0, ST>>>(w, Cout, Cin, (bf16 *)wb, ldk, (bf16 *)wf, ldf);
    return status();
}

extern "C" int dsh_nn_to_bf16(const float *x, void *y, long long n, void *stream)
{
    if (!x || !y || n < 0) return DSH_NN_ERR_PARAM;
    if (n) to_bf16_k<<<grid_for(n), 256, 0, ST>>>(x, (bf16 *)y, n);
    return status();
}

extern "C" int dsh_nn_relu_bwd(const float *dy, const void *y, void *dx, float *dx32, long long n, void *stream)
{
    if (!dy || !y || !dx || n < 0) return DSH_NN_ERR_PARAM;
    if (n && n % 8 == 0 && vec_ok(n / 8, 8) && al16(dy) && al16(y) && al16(dx) && al16(dx32)) {
        relu_bwd_v8<<<vgrid(n / 8), 256, 0, ST>>>((const float4 *)dy, (const uint4 *)y, (uint4 *)dx, (float4 *)dx32,
                                                  (unsigned)(n / 8));
        return status();
    }
    if (n) relu_bwd_k<<<grid_for(n), 256, 0, ST>>>(dy, (const bf16 *)y, (bf16 *)dx, dx32, n);
    return status();
}

extern "C" int dsh_nn_add(float *y, const float *x, long long n, void *stream)
{
    if (!y || !x || n < 0) return DSH_NN_ERR_PARAM;
    if (n && n % 4 == 0 && vec_ok(n / 4, 8) && al16(y) && al16(x)) {
        add_v4<<<vgrid(n / 4), 256, 0, ST>>>((float4 *)y, (const float4 *)x, (unsigned)(n / 4));
        return status();
    }
    if (n) add_k<<<grid_for(n), 256, 0, ST>>>(y, x, n);
    return status();
}

extern "C" int dsh_nn_maxpool_fwd(const void *x, int B, int H, int W, int C, void *y, unsigned char *arg, void *stream)
{
    if (!x || !y || !arg || H % 2 || W % 2 || B <= 0 || C <= 0) return DSH_NN_ERR_PARAM;
    const long long nv = (long long)B * H * W * C / 32;
    if (nv > 0 && vec_ok(nv, C) && al16(x) && al16(y) && ((uintptr_t)arg & 7) == 0) {
        maxpool_fwd_v8<<<vgrid(nv), 256, 0, ST>>>((const uint4 *)x, W, C / 8, (unsigned)nv, (uint4 *)y, (uint2 *)arg);
        return status();
    }
    maxpool_fwd_k<<<grid_for((long long)B * H * W * C / 4), 256, 0, ST>>>((const bf16 *)x, B, H, W, C, (bf16 *)y, arg);
    return status();
}

extern "C" int dsh_nn_maxpool_bwd(const float *dy, const unsigned char *arg, int B, int H, int W, int C, float *dx,
                                  void *stream)
{
    if (!dy || !arg || !dx || H % 2 || W % 2 || B <= 0 || C <= 0) return DSH_NN_ERR_PARAM;
    const long long nv = (long long)B * H * W * C / 16;
    if (nv > 0 && vec_ok(nv, C) && al16(dy) && al16(dx) && ((uintptr_t)arg & 3) == 0) {
        maxpool_bwd_v4<<<vgrid(nv), 256, 0, ST>>>((const float4 *)dy, (const uint32_t *)arg, W, C / 4, (unsigned)nv,
                                                  (float4 *)dx);
        return status();
    }
    maxpool_bwd_k<<<grid_for((long long)B * H * W * C), 256, 0, ST>>>(dy, arg, B, H, W, C, dx);
    return status();
}

extern "C" int dsh_nn_upsample_fwd(const void *x, int B, int h, int w, int C, void *y, void *stream)
{
    if (!x || !y || B <= 0 || h <= 0 || w <= 0 || C <= 0) return DSH_NN_ERR_PARAM;
    const long long nv = (long long)B * h * w * C / 8;
    if (vec_ok(nv, C) && al16(x) && al16(y)) {
        upsample_fwd_v8<<<vgrid(nv), 256, 0, ST>>>((const uint4 *)x, w, C / 8, (unsigned)nv, (uint4 *)y);
        return status();
    }
    upsample_fwd_k<<<grid_for(4LL * B * h * w * C), 256, 0, ST>>>((const bf16 *)x, B, h, w, C, (bf16 *)y);
    return status();
}

extern "C" int dsh_nn_upsample_bwd(const float *dy, int B, int h, int w, int C, float *dx, void *stream)
{
    if (!dy || !dx || B <= 0 || h <= 0 || w <= 0 || C <= 0) return DSH_NN_ERR_PARAM;
    const long long nv = (long long)B * h * w * C / 4;
    if (vec_ok(nv, C) && al16(dy) && al16(dx)) {
        upsample_bwd_v4<<<vgrid(nv), 256, 0, ST>>>((const float4 *)dy, w, C / 4, (unsigned)nv, (float4 *)dx);
        return status();
    }
    upsample_bwd_k<<<grid_for((long long)B * h * w * C), 256, 0, ST>>>(dy, B, h, w, C, dx);
    return status();
}

extern "C" int dsh_nn_concat(const void *a, int C1, const void *b, int C2, long long P, void *y, void *stream)
{
    if (!a || !b || !y || C1 <= 0 || C2 <= 0 || P <= 0) return DSH_NN_ERR_PARAM;
    const long long nv = P * (C1 + C2) / 8;
    if (vec_ok(nv, C1) && C2 % 8 == 0 && al16(a) && al16(b) && al16(y)) {
        concat_v<<<vgrid(nv), 256, 0, ST>>>((const uint4 *)a, C1 / 8, (const uint4 *)b, C2 / 8, (unsigned)nv, (uint4 *)y);
        return status();
    }
    concat_k<<<grid_for(P * (C1 + C2)), 256, 0, ST>>>((const bf16 *)a, C1, (const bf16 *)b, C2, P, (bf16 *)y);
    return status();
}

extern "C" int dsh_nn_split(const float *dy, int C1, int C2, long long P, float *da, float *db, void *stream)
{
    if (!dy || !da || !db || C1 <= 0 || C2 <= 0 || P <= 0) return DSH_NN_ERR_PARAM;
    const long long nv = P * (C1 + C2) / 4;
    if (vec_ok(nv, C1) && C2 % 8 == 0 && al16(dy) && al16(da) && al16(db)) {
        split_v<<<vgrid(nv), 256, 0, ST>>>((const uint4 *)dy, C1 / 4, C2 / 4, (unsigned)nv, (uint4 *)da, (uint4 *)db);
        return status();
    }
    split_k<<<grid_for(P * (C1 + C2)), 256, 0, ST>>>(dy, C1, C2, P, da, db);
    return status();
}

extern "C" int dsh_nn_head_fwd(const void *x, long long P, int C, const float *w, const float *b, float *out,
                               void *stream)
{
    if (!x || !w || !b || !out || P <= 0 || C <= 0) return DSH_NN_ERR_PARAM;
    if (vec_ok(P, C) && al16(x)) {
        head_fwd_v8<<<vgrid(P), 256, 0, ST>>>((const uint4 *)x, (unsigned)P, C / 8, w, b, out);
        return status();
    }
    head_fwd_k<<<grid_for(P), 256, 0, ST>>>((const bf16 *)x, P, C, w, b, out);
    return status();
}

constexpr int RED_BLOCKS = DSH_NN_RED_BLOCKS;
static_assert(RED_BLOCKS % 37 == 0, "sum_parts_k");

extern "C" int dsh_nn_head_bwd(const float *dout, const void *x, long long P, int C, const float *w, float *dx,
                               float *gw, float *gb, float *part, void *stream)
{
    if (!dout || !x || !w || !dx || !gw || !gb || !part || P <= 0 || C <= 0 || C + 1 > 256) return DSH_NN_ERR_PARAM;
    head_bwd_k<<<RED_BLOCKS, 256, 256 * sizeof(float), ST>>>(dout, (const bf16 *)x, P, C, w, dx, part);
    sum_parts_k<<<1, 256, 0, ST>>>(part, RED_BLOCKS, C, C + 1, gw);
    sum_parts_k<<<1, 32, 0, ST>>>(part + C, RED_BLOCKS, 1, C + 1, gb);   /* column C of the (C+1)-wide table */
    return status();
}

extern "C" int dsh_nn_colsum(const float *dy, long long P, int N, float *g, float *part, void *stream)
{
    if (!dy || !g || !part || P <= 0 || N <= 0) return DSH_NN_ERR_PARAM;
    if (N % 4 == 0 && N <= 256 && al16(dy))
        colsum_tiles<<<RED_BLOCKS, 256, 0, ST>>>(dy, P, N, part);
    else
        colsum_k<<<RED_BLOCKS, 256, 0, ST>>>(dy, P, N, part);
    sum_parts_k<<<(N + 255) / 256, 256, 0, ST>>>(part, RED_BLOCKS, N, N, g);
    return status();
}

extern "C" int dsh_nn_mse(const float *pred, const float *target, const unsigned char *mask, long long n, float count,
                          float *grad, float *loss, void *stream)
{
    if (!pred || !target || !grad || !loss || n <= 0 || !(count > 0)) return DSH_NN_ERR_PARAM;
    mse_k<<<grid_for(n), 256, 0, ST>>>(pred, target, mask, n, count, grad, loss);
    return status();
}

extern "C" int dsh_nn_adam(float *w, float *m, float *v, const float *g, int rows, int cols, int transposed, float lr,
                           float beta1, float beta2, float eps, int step, void *stream)
{
    if (!w || !m || !v || !g || rows <= 0 || cols <= 0 || step < 1) return DSH_NN_ERR_PARAM;
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    adam_k<<<grid_for((long long)rows * cols), 256, 0, ST>>>(w, m, v, g, rows, cols, transposed, lr, beta1, beta2, eps,
                                                             c1, c2);
    return status();
}
