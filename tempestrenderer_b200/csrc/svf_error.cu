// svf_error.cu - the error of fitted SVBRDF maps against a BTF, per texel
// (svbrdf-error-tool, tools/svbrdf-error-tool/svbrdf-error-tool.cc:88-250),
// and the rendered BTF of SVBRDF maps (the same BRDF written out).
//
// For texel t the map values give the material (diffuse and specular RGB, the
// SGGX scales, the basis quaternion; Fresnel 1) and the SGGX surface BRDF is
// evaluated at every (light, view) pair of the BTF's directions (the factored
// form of svf_model.cuh); the residual is BTF - BRDF per channel (color) or of
// the luminance.  Pair-wise: MSE over all L^2 pairs and the peak BTF value;
// max-view: the view whose sum over the lights is largest (per channel), its
// sum / L and its peak.  RMSE = sqrt(MSE), PSNR = 20 log10(peak / RMSE).
//
// One CTA per texel, sums in FP64 reduced in a fixed order (deterministic).  The
// pair-wise error and the renderer keep a light in each thread's registers and take the
// views two at a time, in paired FP32 instructions, from shared memory, where all lanes
// read the same entry; max-view takes warps over views and lanes over lights, a table of
// directions in shared memory.  Both pair kernels are bound by instruction issue (78 %).
// Measured, ring-81: pair-wise error of 128 x 128 texels 0.45 ms (0.63 with a pair a
// thread, both its directions' entries read from tables of 12-word entries), 200 x 200
// texels rendered 0.76 ms (0.96; 0.91 where the samples leave a value to a store).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "svf_internal.h"
#include "svf_model.cuh"

namespace svf
{

namespace
{

constexpr int kThreads = 256, kWarps = kThreads / 32, kPairThreads = 384;

__device__ __forceinline__ void load_rgb(const ErrorArgs& a, uint64_t s, uint32_t lv, float* v)
{
    const uint64_t i = (s * a.N + lv) * 3;
    if(a.sample_type == SVF_SAMPLES_F16)
    {
        const __half* p = static_cast<const __half*>(a.samples) + i;
        v[0] = __half2float(p[0]);
        v[1] = __half2float(p[1]);
        v[2] = __half2float(p[2]);
    }
    else
    {
        const float* p = static_cast<const float*>(a.samples) + i;
        v[0] = p[0];
        v[1] = p[1];
        v[2] = p[2];
    }
}

// RGBToLuminance (spectrum.hh:328-331), products and sums rounded in order
__device__ __forceinline__ float lum(const float* c)
{
    return __fadd_rn(__fadd_rn(__fmul_rn(0.2126f, c[0]), __fmul_rn(0.7152f, c[1])), __fmul_rn(0.0722f, c[2]));
}

// A texel's material: the channels' colours and (thread 0 of the CTA) the parameter set.
template <typename Args>
__device__ __forceinline__ void load_material(const Args& a, uint64_t t, float* kd, float* ks, ParamSet& ps)
{
    for(int c = 0; c < 3; ++c)
    {
        kd[c] = a.diffuse[3 * t + c];
        ks[c] = a.specular[3 * t + c];
    }
    if(threadIdx.x == 0)
    {
        float p[12];
        float sx = a.sigma[a.sigma_channels * t], sy = a.sigma[a.sigma_channels * t + 1];
        if(a.sigma_channels == 3)
        {
            const float sz = a.sigma[3 * t + 2];
            sx = sx / sz;
            sy = sy / sz;
        }
        p[6] = sx;
        p[7] = sy;
        for(int k = 0; k < 4; ++k)
            p[8 + k] = a.basis[4 * t + k];
        make_param_set_rgb(p, ps);
    }
    __syncthreads();
}

// What a pair takes from its two views (2p, 2p + 1), side by side: the direction, its
// place in the surface's frame, sigma over the cosine, kspec over the cosine and the
// hemisphere.
struct alignas(16) ViewPair
{
    float2 w[3], a[3], sp, kv, up, pad;
};

// What it takes from its light, in registers.
struct Light
{
    float w[3], a[3], sp, kdc, up;
};

__device__ __forceinline__ DirEntry direction_entry(const float* geo, uint32_t L, uint32_t d, const ParamSet& ps, float* w)
{
    DirEntry e;
    for(int k = 0; k < 3; ++k)
        w[k] = geo[k * L + d];
    make_dir_entry(ps, w[0], w[1], w[2], e);
    return e;
}

__device__ __forceinline__ void fill_views(const float* geo, uint32_t L, const ParamSet& ps, ViewPair* views)
{
    for(uint32_t d = threadIdx.x; d < ((L + 1) & ~1u); d += blockDim.x)
    {
        float w[3];
        const DirEntry e = direction_entry(geo, L, d < L ? d : L - 1, ps, w);   // (an odd L's last view stands twice)
        float* v = reinterpret_cast<float*>(views + d / 2) + (d & 1);
        for(int k = 0; k < 3; ++k)
        {
            v[2 * k] = w[k];
            v[6 + 2 * k] = e.a[k];
        }
        v[12] = e.sp;
        v[14] = ps.kspec * e.kv;
        v[16] = e.up;
    }
    __syncthreads();
}

__device__ __forceinline__ Light load_light(const float* geo, uint32_t L, uint32_t d, const ParamSet& ps)
{
    Light l;
    const DirEntry e = direction_entry(geo, L, d, ps, l.w);
    for(int k = 0; k < 3; ++k)
        l.a[k] = e.a[k];
    l.sp = e.sp;
    l.kdc = e.kdc;
    l.up = e.up;
    return l;
}

__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }

// The BRDF of a light and two views, per channel.
__device__ __forceinline__ void eval_views(const Light& li, const ViewPair& vo, float u, float v, float fresnel,
                                           const float* kd, const float* ks, float2* f)
{
    const float2 W0 = __fadd2_rn(both(li.w[0]), vo.w[0]), W1 = __fadd2_rn(both(li.w[1]), vo.w[1]),
                 W2 = __fadd2_rn(both(li.w[2]), vo.w[2]);
    const float2 g = __ffma2_rn(W2, W2, __ffma2_rn(W0, W0, __fmul2_rn(W1, W1)));
    const float2 s0 = __fadd2_rn(both(li.a[0]), vo.a[0]), s1 = __fadd2_rn(both(li.a[1]), vo.a[1]),
                 s2 = __fadd2_rn(both(li.a[2]), vo.a[2]);
    const float2 Q = __ffma2_rn(s2, s2, __ffma2_rn(__fmul2_rn(both(u), s0), s0,
                                                   __fmul2_rn(__fmul2_rn(both(v), s1), s1)));
    const float2 S = __fadd2_rn(both(li.sp), vo.sp);
    const float2 QQS = __fmul2_rn(__fmul2_rn(Q, Q), S);
    float2 k = __fmul2_rn(vo.kv, both(li.up));
    if(fresnel != 1.0f)
    {
        const float w0[3] = { vo.w[0].x, vo.w[1].x, vo.w[2].x }, w1[3] = { vo.w[0].y, vo.w[1].y, vo.w[2].y };
        k.x *= fresnel_factor(fresnel, li.w, w0);
        k.y *= fresnel_factor(fresnel, li.w, w1);
    }
    const float2 num = __fmul2_rn(__fmul2_rn(k, g), g);
    const float2 spec = make_float2(QQS.x > 0.0f ? num.x / QQS.x : 0.0f, QQS.y > 0.0f ? num.y / QQS.y : 0.0f);
    const float2 diff = __fmul2_rn(vo.up, both(li.kdc));
#pragma unroll
    for(int c = 0; c < 3; ++c)
        f[c] = __ffma2_rn(both(kd[c]), diff, __fmul2_rn(both(ks[c]), spec));
}

// The pair kernels' CTA: groups of L threads; a thread keeps a light and its group goes
// through every groups-th two views.  As many groups, in at most 384 threads, as leave
// the fewest threads idle (81 lights: three, 243 threads of 256 and 41 of 42 rounds).
__host__ __device__ __forceinline__ unsigned group_threads(uint32_t groups, uint32_t L) { return (groups * L + 31) / 32 * 32; }
uint32_t pair_groups(uint32_t L)
{
    const uint32_t pairs = (L + 1) / 2;
    uint32_t best = 1;
    double use = 0.0;
    for(uint32_t groups = 1; groups <= pairs && group_threads(groups, L) <= kPairThreads; ++groups)
    {
        const double x = (double)L * pairs / ((double)group_threads(groups, L) * ((pairs + groups - 1) / groups));
        if(x >= use)
        {
            use = x;
            best = groups;
        }
    }
    return best;
}

__device__ __forceinline__ uint64_t sample_row(const ErrorArgs& a, uint64_t t)
{
    const uint64_t ry = t / a.region_w, rx = t - ry * a.region_w;
    return ry * a.row_texels + a.x0 + rx;
}

__device__ __forceinline__ void store_error(const ErrorArgs& a, uint64_t o, double mse, float peak)
{
    const float rmse = (float)sqrt(mse);
    a.rmse[o] = rmse;
    a.psnr[o] = 20.0f * log10f(peak / rmse);
}

// Pair-wise error.
template <bool kColor>
__global__ void __launch_bounds__(kPairThreads) error_pairs_kernel(ErrorArgs a, uint32_t groups)
{
    extern __shared__ ViewPair views[];
    constexpr int C = kColor ? 3 : 1, kWarpsMax = kPairThreads / 32;
    __shared__ double red_sq[kWarpsMax][C];
    __shared__ float red_mx[kWarpsMax][C];
    __shared__ ParamSet ps;
    const uint32_t L = a.L;
    const uint64_t t = blockIdx.x, s = sample_row(a, t);
    float kd[3], ks[3];
    load_material(a, t, kd, ks, ps);
    fill_views(a.geo, L, ps, views);
    double sq[C] = {};
    float mx[C] = {};
    const uint32_t group = threadIdx.x / L, light = threadIdx.x - group * L;
    if(group < groups)
    {
        const Light li = load_light(a.geo, L, light, ps);
        for(uint32_t p = group; 2 * p < L; p += groups)
        {
            const bool two = 2 * p + 1 < L;
            float v[2][3] = {};
            load_rgb(a, s, 2 * p * L + light, v[0]);
            if(two)
                load_rgb(a, s, (2 * p + 1) * L + light, v[1]);
            float2 f[3];
            eval_views(li, views[p], ps.u, ps.v, 1.0f, kd, ks, f);
#pragma unroll
            for(int h = 0; h < 2; ++h)
            {
                const float fh[3] = { h ? f[0].y : f[0].x, h ? f[1].y : f[1].x, h ? f[2].y : f[2].x };
#pragma unroll
                for(int c = 0; c < C; ++c)
                {
                    const float b = kColor ? v[h][c] : lum(v[h]);
                    const float r = h && !two ? 0.0f : b - (kColor ? fh[c] : lum(fh));
                    sq[c] += (double)r * r;
                    mx[c] = fmaxf(mx[c], b);
                }
            }
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for(int c = 0; c < C; ++c)
    {
        for(int o = 16; o > 0; o >>= 1)
        {
            sq[c] += __shfl_xor_sync(0xffffffffu, sq[c], o);
            mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], o));
        }
        if(lane == 0)
        {
            red_sq[warp][c] = sq[c];
            red_mx[warp][c] = mx[c];
        }
    }
    __syncthreads();
    if(threadIdx.x < C)
    {
        const int c = threadIdx.x;
        double tot = red_sq[0][c];
        float peak = red_mx[0][c];
        for(int w = 1; w < (int)(blockDim.x >> 5); ++w)
        {
            tot += red_sq[w][c];
            peak = fmaxf(peak, red_mx[w][c]);
        }
        store_error(a, C * t + c, tot / ((double)L * L), peak);
    }
}

// Max-view error.
__global__ void __launch_bounds__(kThreads) error_views_kernel(ErrorArgs a)
{
    extern __shared__ float smem[];
    const uint32_t L = a.L;
    DirEntry* tab = reinterpret_cast<DirEntry*>(smem);
    float* dirs = reinterpret_cast<float*>(tab + L);                    // [L][3]
    __shared__ double red_sq[kWarps][3];
    __shared__ float red_mx[kWarps][3];
    __shared__ ParamSet ps;
    const uint64_t t = blockIdx.x, s = sample_row(a, t);
    const uint32_t nch = a.color ? 3 : 1;
    float kd[3], ks[3];
    load_material(a, t, kd, ks, ps);
    for(uint32_t d = threadIdx.x; d < L; d += kThreads)
    {
        const float wx = a.geo[d], wy = a.geo[L + d], wz = a.geo[2 * L + d];
        make_dir_entry(ps, wx, wy, wz, tab[d]);
        dirs[3 * d] = wx;
        dirs[3 * d + 1] = wy;
        dirs[3 * d + 2] = wz;
    }
    __syncthreads();

    // the residuals of pair (light, view): r[c] and the BTF value b[c]
    auto pair = [&](uint32_t light, uint32_t view, float* r, float* b) {
        float v[3];
        load_rgb(a, s, view * L + light, v);
        const DirEntry& li = tab[light];
        const DirEntry& vo = tab[view];
        const float* wi = dirs + 3 * light;
        const float* wo = dirs + 3 * view;
        const float W0 = wi[0] + wo[0], W1 = wi[1] + wo[1], W2 = wi[2] + wo[2];
        const float g = W0 * W0 + W1 * W1 + W2 * W2;
        const float s0 = li.a[0] + vo.a[0], s1 = li.a[1] + vo.a[1], s2 = li.a[2] + vo.a[2];
        const float Q = ps.u * s0 * s0 + ps.v * s1 * s1 + s2 * s2;
        const float S = li.sp + vo.sp;
        const float QQS = Q * Q * S;
        const float spec = QQS > 0.0f ? ps.kspec * vo.kv * li.up * g * g / QQS : 0.0f;
        const float diff = vo.up * li.kdc;
        float f[3];
        for(int c = 0; c < 3; ++c)
            f[c] = kd[c] * diff + ks[c] * spec;
        if(a.color)
            for(int c = 0; c < 3; ++c)
            {
                b[c] = v[c];
                r[c] = v[c] - f[c];
            }
        else
        {
            b[0] = lum(v);
            r[0] = b[0] - lum(f);
        }
    };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // warps over views; a warp keeps, per channel, its largest view sum
    double best[3] = { -1.0, -1.0, -1.0 };
    float best_mx[3] = { 0.0f, 0.0f, 0.0f };
    for(uint32_t view = warp; view < L; view += kWarps)
    {
        double vs[3] = { 0.0, 0.0, 0.0 };
        float vm[3] = { 0.0f, 0.0f, 0.0f };
        for(uint32_t light = lane; light < L; light += 32)
        {
            float r[3], b[3];
            pair(light, view, r, b);
            for(uint32_t c = 0; c < nch; ++c)
            {
                vs[c] += (double)r[c] * r[c];
                vm[c] = fmaxf(vm[c], b[c]);
            }
        }
        for(uint32_t c = 0; c < nch; ++c)
        {
            for(int o = 16; o > 0; o >>= 1)
            {
                vs[c] += __shfl_xor_sync(0xffffffffu, vs[c], o);
                vm[c] = fmaxf(vm[c], __shfl_xor_sync(0xffffffffu, vm[c], o));
            }
            if(vs[c] > best[c])
            {
                best[c] = vs[c];
                best_mx[c] = vm[c];
            }
        }
    }
    if(lane == 0)
        for(uint32_t c = 0; c < nch; ++c)
        {
            red_sq[warp][c] = best[c];
            red_mx[warp][c] = best_mx[c];
        }
    __syncthreads();
    if(threadIdx.x == 0)
        for(uint32_t c = 0; c < nch; ++c)
        {
            double tot = red_sq[0][c];
            float peak = red_mx[0][c];
            for(int w = 1; w < kWarps; ++w)
                if(red_sq[w][c] > tot)
                {
                    // views were dealt round robin: warp w held views w, w+8, ...;
                    // equal sums keep the warp seen first
                    tot = red_sq[w][c];
                    peak = red_mx[w][c];
                }
            store_error(a, nch * t + c, tot < 0.0 ? 0.0 : tot / L, peak);
        }
}

// Four consecutive samples' values, 4 elements aligned.
__device__ __forceinline__ void store4(float* o, float4 v) { *reinterpret_cast<float4*>(o) = v; }
__device__ __forceinline__ void store4(__half* o, float4 v)
{
    __half2 h[2] = { __floats2half2_rn(v.x, v.y), __floats2half2_rn(v.z, v.w) };
    *reinterpret_cast<uint2*>(o) = *reinterpret_cast<const uint2*>(h);
}
__device__ __forceinline__ void store1(float* o, float v) { *o = v; }
__device__ __forceinline__ void store1(__half* o, float v) { *o = __float2half_rn(v); }

// Floats of a stage buffer: two views of each group, shifted by up to 3.
__host__ __device__ __forceinline__ uint32_t stage_floats(uint32_t groups, uint32_t L)
{
    return (2 * groups * 3 * L + 3 + 3) / 4 * 4;
}

// Rendered BTF: texel t's samples [L^2][3] from its map values, lv = view * L + light.
// The groups' views are consecutive, so their samples are one run of memory; they leave
// through shared memory, two buffers in turn, four values to a store: a buffer begins
// as many values past 16 bytes as its run of memory does past four values.
template <typename T>
__global__ void __launch_bounds__(kPairThreads) render_kernel(RenderArgs a, uint32_t groups)
{
    extern __shared__ ViewPair views[];
    __shared__ ParamSet ps;
    const uint32_t L = a.L, pairs = (L + 1) / 2;
    const uint64_t t = blockIdx.x;
    const uint32_t group = threadIdx.x / L, light = threadIdx.x - group * L, row = 3 * L;   // values of a view
    float* stage = reinterpret_cast<float*>(views + pairs);
    float kd[3], ks[3];
    load_material(a, t, kd, ks, ps);
    fill_views(a.geo, L, ps, views);
    const Light li = load_light(a.geo, L, light, ps);
    const float u = ps.u, v = ps.v;
    T* to = static_cast<T*>(a.out) + t * L * row;
    const uint32_t mine = 2 * group * row + 3 * light;
    for(uint32_t p0 = 0; p0 < pairs; p0 += groups, to += 2 * groups * row)
    {
        const uint32_t p = p0 + group, shift = (uint32_t)((uintptr_t)to / sizeof(T)) & 3;
        if(group < groups && p < pairs)
        {
            float2 f[3];
            eval_views(li, views[p], u, v, a.fresnel, kd, ks, f);
            float* o = stage + shift + mine;
#pragma unroll
            for(int c = 0; c < 3; ++c)
            {
                o[c] = f[c].x;
                o[row + c] = f[c].y;
            }
        }
        __syncthreads();   // (the buffer is written again past the next barrier)
        const uint32_t end = shift + (2 * (p0 + groups) < L ? 2 * groups : L - 2 * p0) * row;
        for(uint32_t e = 4 * threadIdx.x; e < end; e += 4 * blockDim.x)
        {
            const float4 x = *reinterpret_cast<const float4*>(stage + e);
            if(e >= shift && e + 4 <= end)
                store4(to + e - shift, x);
            else
            {
                const float y[4] = { x.x, x.y, x.z, x.w };
#pragma unroll
                for(uint32_t k = 0; k < 4; ++k)
                    if(e + k >= shift && e + k < end)
                        store1(to + (e + k - shift), y[k]);
            }
        }
        stage = reinterpret_cast<float*>(views + pairs) + (stage == reinterpret_cast<float*>(views + pairs)
                                                               ? stage_floats(groups, L) : 0);
    }
}

} // namespace

cudaError_t launch_render(const RenderArgs& a, cudaStream_t stream)
{
    if(a.count == 0)
        return cudaSuccess;
    if(a.count > 0x7fffffffull)
        return cudaErrorInvalidValue;
    const uint32_t groups = pair_groups(a.L);
    const size_t smem = sizeof(ViewPair) * ((a.L + 1) / 2) + sizeof(float) * 2 * stage_floats(groups, a.L);
    if(a.sample_type == SVF_SAMPLES_F16)
        render_kernel<__half><<<(unsigned)a.count, group_threads(groups, a.L), smem, stream>>>(a, groups);
    else
        render_kernel<float><<<(unsigned)a.count, group_threads(groups, a.L), smem, stream>>>(a, groups);
    return cudaGetLastError();
}

cudaError_t launch_error(const ErrorArgs& a, cudaStream_t stream)
{
    if(a.count == 0)
        return cudaSuccess;
    if(a.count > 0x7fffffffull)
        return cudaErrorInvalidValue;
    if(a.method == SVF_ERROR_PAIRWISE)
    {
        const uint32_t groups = pair_groups(a.L);
        const unsigned threads = group_threads(groups, a.L);
        const size_t smem = sizeof(ViewPair) * ((a.L + 1) / 2);
        if(a.color)
            error_pairs_kernel<true><<<(unsigned)a.count, threads, smem, stream>>>(a, groups);
        else
            error_pairs_kernel<false><<<(unsigned)a.count, threads, smem, stream>>>(a, groups);
        return cudaGetLastError();
    }
    const size_t smem = (sizeof(DirEntry) + 3 * sizeof(float)) * a.L;
    error_views_kernel<<<(unsigned)a.count, kThreads, smem, stream>>>(a);
    return cudaGetLastError();
}

} // namespace svf
