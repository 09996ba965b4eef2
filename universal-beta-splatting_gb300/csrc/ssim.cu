// ssim.cu -- the training loss (1 - l) L1 + l (1 - SSIM) and its gradient.
//
// SSIM as the reference defines it (utils/loss_utils.py:26-80, the function
// the fused_ssim package used by train.py:117-121 evaluates): an 11 x 11
// Gaussian window (sigma 1.5) applied with zero padding ("same" output size)
// to x, y, x^2, y^2 and x y; C1 = 0.01^2, C2 = 0.03^2;
//   map = (2 mx my + C1)(2 sxy + C2) / ((mx^2 + my^2 + C1)(sxx + syy + C2))
// with sxx = E[x^2] - mx^2, sxy = E[xy] - mx my, and the loss reads the mean
// of the map (optionally cropped by the window radius, fused_ssim's "valid").
//
// Two kernels.  A warp owns a strip of 64 columns and some rows of one (image,
// channel) and goes down it row by row, two columns per lane: a row (with the
// halo columns) comes through a ring of shared rows that only this warp uses,
// the horizontal 11 taps are formed from it in registers, and the vertical ones
// by ten running sums per quantity, acc[k] = g[9 - k] h + acc[k + 1], of which
// the last is complete.  No barriers and no pass over shared memory for the
// vertical window; quantities that are filtered with the same window travel in
// pairs through Blackwell's packed FP32x2 FMA ((x, y), (x^2, y^2), (D1, D2)):
//  * ssim_map_kernel: the five windowed moments, the map, the loss partials and
//    -- for the gradient -- the map's derivatives with the E[.] moments as the
//    free variables, D0 = d map / d mx, D1 = d map / d E[x^2],
//    D2 = d map / d E[xy], stored as a D0 plane and a (D1, D2) plane (12 B
//    per pixel-channel, mostly L2-resident between the two launches);
//  * ssim_grad_kernel: d loss / d x_p = gb sum_q w(q - p) (D0 + 2 x_p D1 +
//    y_p D2) + ga sign(x_p - y_p): the window over the three planes and the
//    combination with the image and target.
// Loss sums: one partial per CTA, reduced in a fixed order by the last CTA to
// finish (a ticket counter that the last CTA resets), so the result is
// deterministic and the launches can be replayed from a CUDA graph.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "ubs_common.cuh"

namespace ubs {
namespace {

constexpr int SS_R = 5;                 // window radius (11 taps)
constexpr int SS_W = 2 * SS_R + 1;
constexpr int SS_C = 64;                // columns of a strip (two per lane)
constexpr int SS_IN = SS_C + 2 * SS_R;  // 74: with the halo
constexpr int SS_IP = SS_IN + 2;        // row pitch of the ring (16-byte rows of pairs)
constexpr int SS_RING = 8;              // rows in flight or in use
constexpr int SS_WARPS = 4;             // strips of a CTA
constexpr int SS_THREADS = 32 * SS_WARPS;
constexpr int SS_CTAS = 4;              // CTAs per SM (map kernel: 80 running sums per lane)

struct SsimArgs {
    const float *img;
    const float *gt;
    float *grad;                 // null: loss only
    int64_t is[4], gs[4], ds[4]; // element strides (image, channel, row, column)
    int32_t n, c, h, w;
    int32_t strips_x, strips_y, rows; // strips of `rows` rows
    int32_t pitch;                    // of the derivative planes (even)
    int32_t valid;               // count only map points >= SS_R from every edge
    float c1, c2;
    float ga, gb;                // d loss / d |x - y| (per pixel), d loss / d map (per point)
    double inv_px, inv_map;      // 1 / pixels, 1 / counted map points
    double wl1, wssim, wconst;   // loss = wl1 mean|x-y| + wssim mean(map) + wconst
    float g[SS_R + 1];           // normalised 1-D window, first half and centre
    float *dmap0;                // [n c][h][pitch] D0 plane (gradient only)
    float2 *dmap12;              // [n c][h][pitch] (D1, D2) plane
    double *partials;            // [n_ctas][2]
    unsigned *counter;
    float *out;                  // [3]: mean(map), mean|x-y|, loss
};

__device__ __forceinline__ float block_sum(float v, float *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    float s = 0.f;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += red[i];
    return s; // valid in thread 0
}

// The 11-tap window over 11 consecutive values: scalar, and two streams at
// once with the packed FP32x2 FMA (same rounding per component).
__device__ __forceinline__ float tap(const float (&g)[SS_R + 1], int t) {
    return g[t <= SS_R ? t : SS_W - 1 - t];
}
__device__ __forceinline__ float2 fma_g(float g, float2 v, float2 c) {
    return __ffma2_rn(make_float2(g, g), v, c);
}
__device__ __forceinline__ float fma_g(float g, float v, float c) { return fmaf(g, v, c); }
template <class T> __device__ __forceinline__ T zero_of();
template <> __device__ __forceinline__ float zero_of<float>() { return 0.f; }
template <> __device__ __forceinline__ float2 zero_of<float2>() { return make_float2(0.f, 0.f); }

__device__ __forceinline__ float2 add_g(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float add_g(float a, float b) { return a + b; }
// From both ends to the centre: two short chains, whose partial sums stay small
// until the last two additions.
template <class T>
__device__ __forceinline__ T taps(const float (&g)[SS_R + 1], const T *v) {
    T lo = zero_of<T>(), hi = lo;
#pragma unroll
    for (int t = 0; t < SS_R; ++t) {
        lo = fma_g(g[t], v[t], lo);
        hi = fma_g(g[t], v[SS_W - 1 - t], hi);
    }
    return add_g(fma_g(g[SS_R], v[SS_R], lo), hi);
}
// The vertical window: the running sums take the row's value h, and the one
// that has now seen its eleven rows (taps in ascending order) is returned.
template <class T>
__device__ __forceinline__ T roll(const float (&g)[SS_R + 1], T (&acc)[SS_W - 1], T h) {
    const T out = fma_g(tap(g, SS_W - 1), h, acc[0]);
#pragma unroll
    for (int k = 0; k < SS_W - 2; ++k) acc[k] = fma_g(tap(g, SS_W - 2 - k), h, acc[k + 1]);
    acc[SS_W - 2] = fma_g(tap(g, 0), h, zero_of<T>());
    return out;
}

// A warp's strip: plane, first column, first row, rows.
struct Strip {
    int plane, x0, y0, rows;
};
__device__ __forceinline__ Strip strip_of(const SsimArgs &a) {
    const int64_t id = (int64_t)blockIdx.x * SS_WARPS + (threadIdx.x >> 5);
    const int per = a.strips_x * a.strips_y;
    Strip s;
    s.plane = (int)(id / per);
    const int r = (int)(id - (int64_t)s.plane * per), sy = r / a.strips_x;
    s.x0 = (r - sy * a.strips_x) * SS_C;
    s.y0 = sy * a.rows;
    s.rows = s.plane < a.n * a.c ? min(a.rows, a.h - s.y0) : 0; // past the last strip: none
    return s;
}
// Which of the three columns of a lane's copies of a row (x0 - SS_R + lane + 32 k)
// lie in the image; the others stay zero in the ring.
struct Columns {
    bool in[3];
    __device__ __forceinline__ Columns(int x0, int w) {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int gx = x0 - SS_R + lane + 32 * k;
            in[k] = gx >= 0 && gx < w && lane + 32 * k < SS_IN;
        }
    }
};

// Asynchronous global -> shared copies of 4 or 8 bytes (no register staging,
// so several rows of a strip are in flight at once).
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst), "l"(src), "n"(BYTES)
                 : "memory");
}
__device__ __forceinline__ void lds(uint32_t at, float2 &u, float2 &v) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                 : "=f"(u.x), "=f"(u.y), "=f"(v.x), "=f"(v.y)
                 : "r"(at));
}
__device__ __forceinline__ void lds(uint32_t at, float &u, float &v) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];\n" : "=f"(u), "=f"(v) : "r"(at));
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
// this warp's row `SS_RING - 1` commits ago has arrived, for every lane
__device__ __forceinline__ void ring_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(SS_RING - 2) : "memory");
    __syncwarp();
}

// the CTA's partials -> the last CTA reduces all of them in a fixed order
__device__ void finish_loss(const SsimArgs &a, double s, double l) {
    __shared__ bool last;
    __shared__ double dred[2][SS_WARPS];
    auto all = [&](double &s, double &l) { // -> sums over the CTA in thread 0
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            l += __shfl_xor_sync(0xffffffffu, l, o);
        }
        __syncthreads();
        if ((threadIdx.x & 31) == 0) {
            dred[0][threadIdx.x >> 5] = s;
            dred[1][threadIdx.x >> 5] = l;
        }
        __syncthreads();
        s = l = 0.0;
        for (int i = 0; i < SS_WARPS; ++i) {
            s += dred[0][i];
            l += dred[1][i];
        }
    };
    all(s, l);
    if (threadIdx.x == 0) {
        a.partials[2 * blockIdx.x] = s;
        a.partials[2 * blockIdx.x + 1] = l;
        __threadfence();
        last = atomicAdd(a.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = l = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += SS_THREADS) {
        s += __ldcg(a.partials + 2 * i);
        l += __ldcg(a.partials + 2 * i + 1);
    }
    all(s, l);
    if (threadIdx.x == 0) {
        const double ms = s * a.inv_map, ml = l * a.inv_px;
        a.out[0] = (float)ms;
        a.out[1] = (float)ml;
        a.out[2] = (float)(a.wl1 * ml + a.wssim * ms + a.wconst);
        *a.counter = 0u;
    }
}

template <bool GRAD>
__global__ void __launch_bounds__(SS_THREADS, SS_CTAS) ssim_map_kernel(const SsimArgs a) {
    __shared__ __align__(16) float2 ring_[SS_WARPS][SS_RING][SS_IP]; // (x, y)
    constexpr int ROW = SS_IP * sizeof(float2);
    float2(*ring)[SS_IP] = ring_[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const Strip st = strip_of(a);
    float ssim_sum = 0.f, l1_sum = 0.f; // of sums of 8 rows
    if (st.rows > 0) {
        const int img = st.plane / a.c, ch = st.plane % a.c;
        const Columns col(st.x0, a.w);
        const int n_in = st.rows + 2 * SS_R;
        // this lane's first column of the next row to fetch
        const int y_first = max(st.y0 - SS_R, 0);
        const float *X = a.img + img * a.is[0] + ch * a.is[1] + y_first * a.is[2] +
                         (st.x0 - SS_R + lane) * a.is[3];
        const float *Y = a.gt + img * a.gs[0] + ch * a.gs[1] + y_first * a.gs[2] +
                         (st.x0 - SS_R + lane) * a.gs[3];
        const int64_t x32 = 32 * a.is[3], y32 = 32 * a.gs[3];
        const uint32_t slot0 = (uint32_t)__cvta_generic_to_shared(ring[0] + lane);
        for (int e = lane; e < SS_RING * SS_IP; e += 32) ring[0][e] = make_float2(0.f, 0.f);
        __syncwarp();
        // row y0 - SS_R + i of both images (zero outside) into its slot
        auto fetch = [&](int i) {
            const int gy = st.y0 - SS_R + i;
            if (i < n_in && gy >= 0) {
                const uint32_t d = slot0 + i % SS_RING * ROW;
                if (gy < a.h) {
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (col.in[k]) {
                            cp_async<4>(d + 256 * k, X + k * x32);
                            cp_async<4>(d + 256 * k + 4, Y + k * y32);
                        }
                    X += a.is[2];
                    Y += a.gs[2];
                } else {
                    for (int e = lane; e < SS_IP; e += 32)
                        ring[i % SS_RING][e] = make_float2(0.f, 0.f);
                }
            }
            cp_async_commit();
        };
        float g[SS_R + 1];
#pragma unroll
        for (int t = 0; t <= SS_R; ++t) g[t] = a.g[t];
        float2 A[2][SS_W - 1], B[2][SS_W - 1]; // running sums of (x, y), (x^2 + y^2, x y)
#pragma unroll
        for (int k = 0; k < SS_W - 1; ++k)
            A[0][k] = A[1][k] = B[0][k] = B[1][k] = make_float2(0.f, 0.f);
        const int gx = st.x0 + 2 * lane;
        const bool col0 = gx < a.w;
        bool cnt[2]; // columns that count for the mean
#pragma unroll
        for (int c = 0; c < 2; ++c)
            cnt[c] = a.valid ? gx + c >= SS_R && gx + c < a.w - SS_R : gx + c < a.w;
        int64_t at = ((int64_t)st.plane * a.h + st.y0) * a.pitch + gx;
        float s_run = 0.f, l_run = 0.f; // of up to 8 rows
        float2 mA[2], mB[2];
        const uint32_t read0 = (uint32_t)__cvta_generic_to_shared(ring[0]) + 16 * lane;
        // takes row i; what it completes is in mA and mB
        auto step = [&](int i) {
            ring_wait();
            fetch(i + SS_RING - 1); // into the slot that row i - 1 left
            float2 v[12];
            const uint32_t row = read0 + i % SS_RING * ROW;
#pragma unroll
            for (int j = 0; j < 6; ++j) lds(row + 16 * j, v[2 * j], v[2 * j + 1]);
            if (i >= SS_R && i < SS_R + st.rows)
                l_run += fabsf(v[SS_R].x - v[SS_R].y) + fabsf(v[SS_R + 1].x - v[SS_R + 1].y);
#pragma unroll
            for (int c = 0; c < 2; ++c) mA[c] = roll(g, A[c], taps(g, v + c));
#pragma unroll
            for (int j = 0; j < 12; ++j)
                v[j] = make_float2(fmaf(v[j].x, v[j].x, v[j].y * v[j].y), v[j].x * v[j].y);
#pragma unroll
            for (int c = 0; c < 2; ++c) mB[c] = roll(g, B[c], taps(g, v + c));
            if (i % 8 == 7) {
                ssim_sum += s_run;
                l1_sum += l_run;
                s_run = l_run = 0.f;
            }
        };
        for (int i = 0; i < SS_RING - 1; ++i) fetch(i);
        for (int i = 0; i < 2 * SS_R; ++i) step(i);
        for (int i = 2 * SS_R; i < n_in; ++i) {
            step(i);
            const int gy = st.y0 + i - 2 * SS_R;
            const bool row_counts = !a.valid || (gy >= SS_R && gy < a.h - SS_R);
            float d0[2], d1[2], d2[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const bool counted = row_counts && cnt[c];
                const float mx = mA[c].x, my = mA[c].y;
                const float mxx = mx * mx, myy = my * my, mxy = mx * my;
                const float vxy = (mB[c].x - mxx) - myy, cxy = mB[c].y - mxy;
                const float A1 = 2.f * mxy + a.c1, A2 = 2.f * cxy + a.c2;
                const float B1 = mxx + myy + a.c1, B2 = vxy + a.c2;
                const float s = (A1 * A2) / (B1 * B2);
                s_run += counted ? s : 0.f;
                if (GRAD) {
                    const float iB1 = 1.f / B1, iB2 = 1.f / B2, iBB = iB1 * iB2;
                    d0[c] = counted ? 2.f * my * (A2 - A1) * iBB - 2.f * mx * s * (iB1 - iB2) : 0.f;
                    d1[c] = counted ? -s * iB2 : 0.f;
                    d2[c] = counted ? 2.f * A1 * iBB : 0.f;
                }
            }
            if (GRAD && col0) { // the pitch is even: a pair fits
                *reinterpret_cast<float2 *>(a.dmap0 + at) = make_float2(d0[0], d0[1]);
                *reinterpret_cast<float4 *>(a.dmap12 + at) = make_float4(d1[0], d2[0], d1[1], d2[1]);
            }
            at += a.pitch;
        }
        ssim_sum += s_run;
        l1_sum += l_run;
    }
    finish_loss(a, ssim_sum, l1_sum);
}

__global__ void __launch_bounds__(SS_THREADS, SS_CTAS) ssim_grad_kernel(const SsimArgs a) {
    __shared__ __align__(16) float2 r12_[SS_WARPS][SS_RING][SS_IP]; // (D1, D2)
    __shared__ __align__(16) float r0_[SS_WARPS][SS_RING][SS_IP];   // D0
    __shared__ float px_[SS_WARPS][SS_RING][4][32]; // a lane's pixels: x, x, y, y
    constexpr int ROW12 = SS_IP * sizeof(float2), ROW0 = SS_IP * sizeof(float);
    float2(*r12)[SS_IP] = r12_[threadIdx.x >> 5];
    float(*r0)[SS_IP] = r0_[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const float *px = px_[threadIdx.x >> 5][0][0] + lane;
    const Strip st = strip_of(a);
    if (st.rows <= 0) return;
    const int img = st.plane / a.c, ch = st.plane % a.c;
    const Columns col(st.x0, a.w);
    const int n_in = st.rows + 2 * SS_R;
    const int gx = st.x0 + 2 * lane;
    const bool col0 = gx < a.w, col1 = gx + 1 < a.w;
    // the next row to fetch: this lane's first column of the derivative
    // planes, its two columns of the image and the target
    const int64_t first = ((int64_t)st.plane * a.h + max(st.y0 - SS_R, 0)) * a.pitch + st.x0 - SS_R + lane;
    const float *D0 = a.dmap0 + first;
    const float2 *D12 = a.dmap12 + first;
    const float *X = a.img + img * a.is[0] + ch * a.is[1] + gx * a.is[3] + st.y0 * a.is[2];
    const float *Y = a.gt + img * a.gs[0] + ch * a.gs[1] + gx * a.gs[3] + st.y0 * a.gs[2];
    float *Gd = a.grad + img * a.ds[0] + ch * a.ds[1] + gx * a.ds[3] + st.y0 * a.ds[2];
    const uint32_t slot12 = (uint32_t)__cvta_generic_to_shared(r12[0] + lane);
    const uint32_t slot0 = (uint32_t)__cvta_generic_to_shared(r0[0] + lane);
    const uint32_t slot_px = (uint32_t)__cvta_generic_to_shared(px);
    for (int e = lane; e < SS_RING * SS_IP; e += 32) {
        r12[0][e] = make_float2(0.f, 0.f);
        r0[0][e] = 0.f;
    }
    __syncwarp();
    // row y0 - SS_R + i of the planes (zero outside) into its slot, with the
    // pixels of the row that it completes
    auto fetch = [&](int i) {
        const int gy = st.y0 - SS_R + i;
        const int slot = i % SS_RING;
        if (i < n_in && gy >= 0) {
            if (gy < a.h) {
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (col.in[k]) {
                        cp_async<8>(slot12 + slot * ROW12 + 256 * k, D12 + 32 * k);
                        cp_async<4>(slot0 + slot * ROW0 + 128 * k, D0 + 32 * k);
                    }
                D12 += a.pitch;
                D0 += a.pitch;
            } else {
                for (int e = lane; e < SS_IP; e += 32) {
                    r12[slot][e] = make_float2(0.f, 0.f);
                    r0[slot][e] = 0.f;
                }
            }
        }
        if (i >= 2 * SS_R && i < n_in) {
            const uint32_t d = slot_px + slot * 512;
            if (col0) {
                cp_async<4>(d, X);
                cp_async<4>(d + 256, Y);
            }
            if (col1) {
                cp_async<4>(d + 128, X + a.is[3]);
                cp_async<4>(d + 384, Y + a.gs[3]);
            }
            X += a.is[2];
            Y += a.gs[2];
        }
        cp_async_commit();
    };
    float g[SS_R + 1];
#pragma unroll
    for (int t = 0; t <= SS_R; ++t) g[t] = a.g[t];
    float2 S12[2][SS_W - 1], G12[2];
    float S0[2][SS_W - 1], G0[2];
#pragma unroll
    for (int k = 0; k < SS_W - 1; ++k)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            S12[c][k] = make_float2(0.f, 0.f);
            S0[c][k] = 0.f;
        }
    const uint32_t read12 = (uint32_t)__cvta_generic_to_shared(r12[0]) + 16 * lane;
    const uint32_t read0 = (uint32_t)__cvta_generic_to_shared(r0[0]) + 8 * lane;
    auto step = [&](int i) {
        ring_wait();
        fetch(i + SS_RING - 1);
        {
            float2 v[12];
#pragma unroll
            for (int j = 0; j < 6; ++j)
                lds(read12 + i % SS_RING * ROW12 + 16 * j, v[2 * j], v[2 * j + 1]);
#pragma unroll
            for (int c = 0; c < 2; ++c) G12[c] = roll(g, S12[c], taps(g, v + c));
        }
        {
            float v[12];
#pragma unroll
            for (int j = 0; j < 6; ++j)
                lds(read0 + i % SS_RING * ROW0 + 8 * j, v[2 * j], v[2 * j + 1]);
#pragma unroll
            for (int c = 0; c < 2; ++c) G0[c] = roll(g, S0[c], taps(g, v + c));
        }
    };
    for (int i = 0; i < SS_RING - 1; ++i) fetch(i);
    for (int i = 0; i < 2 * SS_R; ++i) step(i);
    for (int i = 2 * SS_R; i < n_in; ++i) {
        step(i);
        const float *q = px + i % SS_RING * 128;
        auto grad_of = [&](float x, float y, float2 d12, float d0) {
            const float d = x - y;
            const float sg = d > 0.f ? 1.f : (d < 0.f ? -1.f : 0.f);
            return fmaf(a.gb, fmaf(2.f * x, d12.x, fmaf(y, d12.y, d0)), a.ga * sg);
        };
        if (col0) Gd[0] = grad_of(q[0], q[64], G12[0], G0[0]);
        if (col1) Gd[a.ds[3]] = grad_of(q[32], q[96], G12[1], G0[1]);
        Gd += a.ds[2];
    }
}

// ---- L1 alone (train.py's l1_loss, utils/loss_utils.py:18-19): mean |x - y|
// over contiguous arrays and its gradient sign(x - y) w / n, one pass; the
// sums reduced like the SSIM partials (fixed order, last CTA).
constexpr int L1_THREADS = 256;
constexpr int L1_PER = 8; // float4 per thread per pass

__global__ void __launch_bounds__(L1_THREADS) l1_kernel(const float *__restrict__ x,
                                                        const float *__restrict__ y,
                                                        float *__restrict__ grad, int64_t n,
                                                        float gscale, double inv_n, double w,
                                                        float *partials, unsigned *counter,
                                                        float *out) {
    float acc = 0.f;
    const int64_t n4 = n >> 2;
    const bool vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) |
                       reinterpret_cast<uintptr_t>(grad)) & 15) == 0;
    const int64_t stride = (int64_t)gridDim.x * L1_THREADS;
    if (vec) {
        // two quads per step, both loads issued before either is used
        auto quad = [&](const float4 &a, const float4 &b, int64_t i) {
            const float d0 = a.x - b.x, d1 = a.y - b.y, d2 = a.z - b.z, d3 = a.w - b.w;
            acc += fabsf(d0) + fabsf(d1) + fabsf(d2) + fabsf(d3);
            if (grad) {
                auto sg = [](float d) { return d > 0.f ? 1.f : (d < 0.f ? -1.f : 0.f); };
                reinterpret_cast<float4 *>(grad)[i] = make_float4(
                    gscale * sg(d0), gscale * sg(d1), gscale * sg(d2), gscale * sg(d3));
            }
        };
        for (int64_t i = (int64_t)blockIdx.x * L1_THREADS + threadIdx.x; i < n4; i += 2 * stride) {
            const int64_t j = i + stride;
            const float4 a = reinterpret_cast<const float4 *>(x)[i];
            const float4 b = reinterpret_cast<const float4 *>(y)[i];
            float4 a2 = make_float4(0.f, 0.f, 0.f, 0.f), b2 = a2;
            if (j < n4) {
                a2 = reinterpret_cast<const float4 *>(x)[j];
                b2 = reinterpret_cast<const float4 *>(y)[j];
            }
            quad(a, b, i);
            if (j < n4) quad(a2, b2, j);
        }
    }
    for (int64_t i = (vec ? n4 * 4 : 0) + (int64_t)blockIdx.x * L1_THREADS + threadIdx.x; i < n;
         i += stride) {
        const float d = x[i] - y[i];
        acc += fabsf(d);
        if (grad) grad[i] = gscale * (d > 0.f ? 1.f : (d < 0.f ? -1.f : 0.f));
    }
    __shared__ float red[L1_THREADS / 32];
    __shared__ bool last;
    __shared__ double dred[L1_THREADS / 32];
    const float bs = block_sum(acc, red);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = bs;
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double s = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += L1_THREADS) s += (double)__ldcg(partials + i);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) dred[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < L1_THREADS / 32; ++i) t += dred[i];
        out[0] = (float)(t * inv_n);
        out[1] = (float)(w * t * inv_n);
        *counter = 0u;
    }
}

// out = x times a device scalar (the stored gradient of a loss times the incoming
// one): four 16-byte accesses per thread in flight.  Bound by memory; 8 views of
// 1352x1014 (33M floats): 40 us, against 81 of the general broadcast product.
constexpr int SCALE_THREADS = 256, SCALE_UNROLL = 4;
__global__ void __launch_bounds__(SCALE_THREADS) scale_kernel(const float *__restrict__ x,
                                                              const float *__restrict__ by,
                                                              float *__restrict__ out, int64_t n) {
    const float f = *by;
    const int64_t i0 = (int64_t)blockIdx.x * (SCALE_THREADS * SCALE_UNROLL) + threadIdx.x;
    int64_t done = 0;
    if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
        const int64_t n4 = n >> 2;
        float4 v[SCALE_UNROLL];
#pragma unroll
        for (int k = 0; k < SCALE_UNROLL; ++k)
            if (i0 + k * SCALE_THREADS < n4)
                v[k] = reinterpret_cast<const float4 *>(x)[i0 + k * SCALE_THREADS];
#pragma unroll
        for (int k = 0; k < SCALE_UNROLL; ++k)
            if (i0 + k * SCALE_THREADS < n4)
                reinterpret_cast<float4 *>(out)[i0 + k * SCALE_THREADS] =
                    make_float4(v[k].x * f, v[k].y * f, v[k].z * f, v[k].w * f);
        done = n4 << 2;
    }
    // what is left: everything, or up to three floats
    for (int64_t i = done + (int64_t)blockIdx.x * SCALE_THREADS + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * SCALE_THREADS)
        out[i] = x[i] * f;
}

int l1_grid(int64_t n) {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t want = (n / 4 + (int64_t)L1_THREADS * L1_PER - 1) / ((int64_t)L1_THREADS * L1_PER);
    const int64_t cap = (int64_t)sms * 8;
    return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}

size_t ws_header() { return 256; }

// Rows per strip.  A strip's time is its rows plus the ten halo rows, times a
// row's time with the warps that share its SM (measured: 0.4 us with 4 warps or
// fewer, 0.58, 0.76 and 0.94 with 8, 12 and 16), so the strips either fill the
// SMs evenly -- whole CTAs per SM, a few turns of four where an image is large
// -- or stay few and long.  Of those the split with the smallest product.  Both
// kernels, RGB, us (rows: time): 640x480 12: 36, 6: 42, 64: 69; 979x547 24: 47,
// 10: 58, 108: 103; 1080p 54: 101, 40: 101, 108: 127; 2400x1600 80: 171, 32: 189,
// 270: 279.
struct SsimSplit {
    int32_t strips_x, strips_y, rows;
    int64_t ctas;
    int32_t pitch;
};
SsimSplit ssim_split(int64_t planes, int32_t h, int32_t w) {
    constexpr int64_t SMS = 152;
    constexpr double ROW_US[SS_CTAS + 1] = {0.0, 0.40, 0.58, 0.76, 0.94};
    SsimSplit s;
    s.strips_x = (w + SS_C - 1) / SS_C;
    const int64_t per_row = planes * s.strips_x;
    double best = 1e300;
    s.rows = h;
    for (int64_t per_sm = 1; per_sm <= 64; ++per_sm) {
        const int64_t fit = std::max<int64_t>(1, SMS * SS_WARPS * per_sm / per_row);
        const int64_t rows = (h + fit - 1) / fit;
        const int64_t ctas = (per_row * ((h + rows - 1) / rows) + SS_WARPS - 1) / SS_WARPS;
        const int64_t used = (ctas + SMS - 1) / SMS;
        const double cost = (double)(rows + 2 * SS_R) *
                            ((double)(used / SS_CTAS) * ROW_US[SS_CTAS] + ROW_US[used % SS_CTAS]);
        if (cost < best) {
            best = cost;
            s.rows = (int32_t)rows;
        }
    }
    s.strips_y = (h + s.rows - 1) / s.rows;
    s.ctas = (per_row * s.strips_y + SS_WARPS - 1) / SS_WARPS;
    s.pitch = (w + 1) & ~1;
    return s;
}
size_t ssim_partials_bytes(const SsimSplit &s) {
    return ((size_t)s.ctas * 2 * sizeof(double) + 255) & ~(size_t)255;
}

} // namespace
} // namespace ubs

using namespace ubs;

extern "C" {

size_t ubs_ssim_workspace_bytes(int32_t n_images, int32_t channels, int32_t height,
                                int32_t width) {
    if (n_images <= 0 || channels <= 0 || height <= 0 || width <= 0) return ws_header();
    const SsimSplit sp = ssim_split((int64_t)n_images * channels, height, width);
    const size_t maps = (size_t)3 * n_images * channels * height * sp.pitch * sizeof(float);
    return ws_header() + 16 + ssim_partials_bytes(sp) + maps;
}

int ubs_ssim_loss(const float *img, const int64_t *img_strides, const float *gt,
                  const int64_t *gt_strides, float *grad, const int64_t *grad_strides,
                  int32_t n_images, int32_t channels, int32_t height, int32_t width,
                  int32_t valid_padding, double weight_l1, double weight_ssim,
                  double weight_const, float *out, void *workspace, size_t workspace_bytes,
                  void *stream) {
    UBS_REQUIRE(n_images > 0 && channels > 0 && height > 0 && width > 0,
                "ssim_loss: empty image batch");
    UBS_REQUIRE((int64_t)n_images * channels <= 65535, "ssim_loss: too many image channels");
    UBS_REQUIRE(!valid_padding || (height > 2 * SS_R && width > 2 * SS_R),
                "ssim_loss: 'valid' padding needs images larger than the window");
    UBS_REQUIRE(img && gt && out && img_strides && gt_strides, "ssim_loss: null pointer");
    UBS_REQUIRE(!grad || grad_strides, "ssim_loss: gradient strides missing");
    UBS_REQUIRE(workspace && workspace_bytes >= ubs_ssim_workspace_bytes(n_images, channels,
                                                                         height, width),
                "ssim_loss: workspace too small");
    SsimArgs a;
    a.img = img;
    a.gt = gt;
    a.grad = grad;
    for (int i = 0; i < 4; ++i) {
        a.is[i] = img_strides[i];
        a.gs[i] = gt_strides[i];
        a.ds[i] = grad ? grad_strides[i] : 0;
    }
    a.n = n_images;
    a.c = channels;
    a.h = height;
    a.w = width;
    const SsimSplit sp = ssim_split((int64_t)n_images * channels, height, width);
    a.strips_x = sp.strips_x;
    a.strips_y = sp.strips_y;
    a.rows = sp.rows;
    a.pitch = sp.pitch;
    a.valid = valid_padding ? 1 : 0;
    a.c1 = (float)(0.01 * 0.01);
    a.c2 = (float)(0.03 * 0.03);
    const double px = (double)n_images * channels * height * width;
    const double pts = valid_padding
                           ? (double)n_images * channels * (height - 2 * SS_R) * (width - 2 * SS_R)
                           : px;
    a.inv_px = 1.0 / px;
    a.inv_map = 1.0 / pts;
    a.wl1 = weight_l1;
    a.wssim = weight_ssim;
    a.wconst = weight_const;
    a.ga = (float)(weight_l1 / px);
    a.gb = (float)(weight_ssim / pts);
    // normalised Gaussian of sigma 1.5 over the 11 taps
    double gs[SS_W], tot = 0.0;
    for (int i = 0; i < SS_W; ++i) {
        const double d = i - SS_R;
        gs[i] = std::exp(-d * d / (2.0 * 1.5 * 1.5));
        tot += gs[i];
    }
    for (int i = 0; i <= SS_R; ++i) a.g[i] = (float)(gs[i] / tot); // symmetric
    a.counter = static_cast<unsigned *>(workspace);
    // 16-byte stores of derivative pairs: aligned here, whatever the caller's
    // workspace is aligned to
    char *part = reinterpret_cast<char *>(
        (reinterpret_cast<uintptr_t>(workspace) + ws_header() + 15) & ~(uintptr_t)15);
    a.partials = reinterpret_cast<double *>(part);
    char *maps = part + ssim_partials_bytes(sp);
    const size_t px_all = (size_t)n_images * channels * height * sp.pitch;
    a.dmap12 = reinterpret_cast<float2 *>(maps);
    a.dmap0 = reinterpret_cast<float *>(maps + px_all * sizeof(float2));
    a.out = out;
    const unsigned grid = (unsigned)sp.ctas;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (grad) {
        UBS_TIMED("ssim_map", st, ssim_map_kernel<true><<<grid, SS_THREADS, 0, st>>>(a));
        UBS_TIMED("ssim_grad", st, ssim_grad_kernel<<<grid, SS_THREADS, 0, st>>>(a));
        note_launch(2);
    } else {
        UBS_TIMED("ssim_map", st, ssim_map_kernel<false><<<grid, SS_THREADS, 0, st>>>(a));
        note_launch();
    }
    return check_launch("ssim_loss");
}

int ubs_scale(const float *x, const float *by, float *out, int64_t n, void *stream) {
    UBS_REQUIRE(n >= 0 && (n == 0 || (x && by && out)), "scale: bad arguments");
    if (n == 0) return UBS_OK;
    constexpr int64_t per = 4LL * SCALE_THREADS * SCALE_UNROLL;
    UBS_REQUIRE((n + per - 1) / per < (1LL << 31), "scale: too many values");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    UBS_TIMED("loss_scale", st,
              scale_kernel<<<(unsigned)((n + per - 1) / per), SCALE_THREADS, 0, st>>>(x, by, out, n));
    note_launch();
    return check_launch("scale");
}

size_t ubs_l1_loss_workspace_bytes(int64_t n) {
    return ws_header() + (((size_t)l1_grid(n < 1 ? 1 : n) * sizeof(float) + 255) & ~(size_t)255);
}

int ubs_l1_loss(const float *x, const float *y, float *grad, int64_t n, double weight,
                float *out, void *workspace, size_t workspace_bytes, void *stream) {
    UBS_REQUIRE(n > 0 && x && y && out, "l1_loss: bad arguments");
    UBS_REQUIRE(workspace && workspace_bytes >= ubs_l1_loss_workspace_bytes(n),
                "l1_loss: workspace too small");
    const int grid = l1_grid(n);
    unsigned *counter = static_cast<unsigned *>(workspace);
    float *partials = reinterpret_cast<float *>(static_cast<char *>(workspace) + ws_header());
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // d mean / d x as torch forms it: the mean's 1/n in float, times the weight
    const float gscale = (float)weight * (float)(1.0 / (double)n);
    UBS_TIMED("l1_loss", st,
              l1_kernel<<<grid, L1_THREADS, 0, st>>>(x, y, grad, n, gscale, 1.0 / (double)n,
                                                     weight, partials, counter, out));
    note_launch();
    return check_launch("l1_loss");
}

} // extern "C"
