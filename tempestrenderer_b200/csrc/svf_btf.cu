// svf_btf.cu - decode of a factored BTF (DFMF / FMF planes resident in HBM)
// into RGB samples [texels][L*L][3], texel-major, as svf_fit_texels reads them.
//
// Reference: BTFEvaluateMatrix (include/tempest/image/btf.hh:608-634) and
// BTFFetchSpectrum (btf.hh:498-556).  Channel c of sample (lv, texel) is
// sum_k U_c[lv][k] * SxV_c[col][k], summed in order k = 0, 1, ... in the
// accumulator type of the plane elements (float for half and float planes,
// double for double planes) with every product rounded before it is added, as
// the reference's x86-64 build evaluates it; then colour model 11 (log-YUV ->
// RGB) and the dynamic range reduction exp(x) - 1e-5.  col is the file column
// of texel y*W + x: LoadBTF flips rows (btf.cc:1000-1022), so it is
// (H - 1 - y)*W + x.
//
// The sums are bit-identical to the reference's; with colour model 11 or DRR
// the exponentials are CUDA's expf (within 2 ulp of libm's), so those samples
// agree to a few ulp.
//
// Half and float planes (btf_decode_tile_kernel): a CTA of 256 threads decodes 128
// pairs x 64 texels, a thread 8 x 4 of them in all three channels: 96 sums, so that
// its samples leave with their channels together and two CTAs share an SM (one
// stores while the other multiplies).  What bounds it is the 32 words a clock that
// shared memory returns to registers, whether or not lanes ask for the same word: 12
// words for 32 products, 82 % of that rate against 51 % of the FP32 pipe's.  8 x 8 a
// thread (16 words for 64 products) needs 192 sums and leaves one CTA: 9.25 ms where
// this takes 8.45.  Half planes accumulate with FMAs (a product of two halves is exact
// in float, so the FMA rounds as the reference's separate multiply and add do), two
// pairs to an instruction; float planes multiply, then add; each sum keeps its order.
// Measured, 81 directions, half planes of 48 components: 400 x 400 texels 8.6 ms
// (17.2 with a thread to one pair x 16 texels and 128 threads), 64 x 64 0.25 (0.48),
// one texel 35 us (38); float planes, 400 x 400: 13.9 ms (24.7).
// Double planes (btf_decode_kernel): a thread takes one pair, a CTA 128 pairs and
// 16 texels.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "svf_internal.h"

namespace svf
{

namespace
{

constexpr int kThreads = 128, kChunk = 32;

__device__ __forceinline__ float elem(const __half* p, uint64_t i) { return __half2float(p[i]); }
__device__ __forceinline__ float elem(const float* p, uint64_t i) { return p[i]; }
__device__ __forceinline__ double elem(const double* p, uint64_t i) { return p[i]; }

// sum + u * v with the product rounded first (no contraction into an FMA,
// which would round once).
__device__ __forceinline__ double madd(double sum, double u, double v) { return __dadd_rn(sum, __dmul_rn(u, v)); }

// Colour model 11 (log-YUV) and DRR on a sample's three decoded values.
__device__ __forceinline__ void to_sample(const BtfDecodeArgs& a, float* v)
{
    const float eps = 1e-5f;
    if(a.color_model == 11)
    {
        // btf.hh:522-531 and YUVToRGB (spectrum.hh:344-350): dot products
        // with the conversion's columns, left to right, then a clamp to [0, 1]
        const float Y = __fsub_rn(expf(v[0]), eps);
        const float U = __fadd_rn(__fmul_rn(v[1], Y), eps);
        const float V = __fadd_rn(__fmul_rn(v[2], Y), eps);
        v[0] = __fadd_rn(__fadd_rn(__fmul_rn(Y, 1.0f), __fmul_rn(U, 0.0f)), __fmul_rn(V, 1.13983f));
        v[1] = __fadd_rn(__fadd_rn(__fmul_rn(Y, 1.0f), __fmul_rn(U, -0.39465f)), __fmul_rn(V, -0.5806f));
        v[2] = __fadd_rn(__fadd_rn(__fmul_rn(Y, 1.0f), __fmul_rn(U, 2.03211f)), __fmul_rn(V, 0.0f));
        // Clamp (functions.hh:156-159)
#pragma unroll
        for(int i = 0; i < 3; ++i)
            v[i] = v[i] <= 0.0f ? 0.0f : (v[i] >= 1.0f ? 1.0f : v[i]);
    }
    if(a.drr)
#pragma unroll
        for(int i = 0; i < 3; ++i)
            v[i] = __fsub_rn(expf(v[i]), eps);
}

// The epilogue of a CTA of btf_decode_kernel: the TX texels' samples of its 128
// pairs, a warp storing 32 consecutive pairs x RGB of one texel at a time.
template <typename Acc, int TX>
__device__ __forceinline__ void store_texels(const BtfDecodeArgs& a, const Acc (&acc)[3][TX], uint64_t t0,
                                             uint32_t lv0)
{
    __shared__ float s_out[kThreads / 32][96];   // one texel's 32 pairs x RGB per warp
    const uint64_t t_end = a.first + a.count;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lv_w = lv0 + warp * 32;   // the warp's first pair
    const uint32_t nvalid = lv_w >= a.N ? 0u : (a.N - lv_w < 32u ? a.N - lv_w : 32u);
#pragma unroll
    for(int j = 0; j < TX; ++j)
    {
        const uint64_t t = t0 + j;
        if(t >= t_end)
            break;   // (the same for the whole CTA)
        float v[3] = { (float)acc[0][j], (float)acc[1][j], (float)acc[2][j] };
        to_sample(a, v);
        // the warp's 32 samples are 96 consecutive values: stage them and store
        // them lane-consecutive (each store instruction covers 32 neighbours)
        s_out[warp][3 * lane] = v[0];
        s_out[warp][3 * lane + 1] = v[1];
        s_out[warp][3 * lane + 2] = v[2];
        __syncwarp();
        const uint64_t o = ((t - a.first) * a.N + lv_w) * 3;
        if(a.out_type == SVF_SAMPLES_F16)
        {
            __half* out = static_cast<__half*>(a.out) + o;
            for(uint32_t e = lane; e < 3 * nvalid; e += 32)
                out[e] = __float2half_rn(s_out[warp][e]);
        }
        else
        {
            float* out = static_cast<float*>(a.out) + o;
            for(uint32_t e = lane; e < 3 * nvalid; e += 32)
                out[e] = s_out[warp][e];
        }
        __syncwarp();
    }
}

template <typename T, typename Acc, int TX>
__global__ void __launch_bounds__(kThreads) btf_decode_kernel(BtfDecodeArgs a, uint64_t t_begin)
{
    // rows padded by 4: the staging writes of one warp (32 components of one
    // texel) spread over 8 banks, and rows stay 16-byte aligned for the
    // vector broadcasts of the inner loop
    __shared__ __align__(16) Acc s_sxv[kChunk][TX + 4];
    __shared__ Acc s_u[kChunk][kThreads + 1];
    __shared__ uint64_t s_col[TX];   // file column of each texel (after the row flip)
    const uint32_t lv0 = blockIdx.x * kThreads;
    const uint64_t t0 = t_begin + (uint64_t)blockIdx.y * TX;
    const uint64_t t_end = a.first + a.count;
    if(threadIdx.x < TX)
    {
        const uint64_t t = t0 + threadIdx.x;
        const uint64_t y = t / a.width, x = t - y * a.width;
        s_col[threadIdx.x] = t < t_end ? (a.height - 1 - y) * a.width + x : ~0ull;
    }
    Acc acc[3][TX];
#pragma unroll
    for(int c = 0; c < 3; ++c)
#pragma unroll
        for(int j = 0; j < TX; ++j)
            acc[c][j] = Acc(0);

#pragma unroll
    for(int c = 0; c < 3; ++c)
    {
        const T* U = static_cast<const T*>(a.u[c]);
        const T* S = static_cast<const T*>(a.sxv[c]);
        const uint32_t K = a.k[c];
        for(uint32_t k0 = 0; k0 < K; k0 += kChunk)
        {
            __syncthreads();
            // a warp reads 32 consecutive components of one row per step
            const int kk = threadIdx.x % kChunk, r0 = threadIdx.x / kChunk;
            const bool k_ok = k0 + kk < K;
            for(int j = r0; j < TX; j += kThreads / kChunk)
            {
                const uint64_t col = s_col[j];
                s_sxv[kk][j] = (col != ~0ull && k_ok) ? elem(S, col * a.sxv_row[c] + k0 + kk) : Acc(0);
            }
            {
                const T* up = U + (uint64_t)(lv0 + r0) * a.u_row[c] + k0 + kk;
                const uint64_t step = (uint64_t)(kThreads / kChunk) * a.u_row[c];
                for(int row = r0; row < kThreads; row += kThreads / kChunk, up += step)
                    s_u[kk][row] = (lv0 + row < a.N && k_ok) ? elem(up, 0) : Acc(0);
            }
            __syncthreads();
            const uint32_t n = K - k0 < (uint32_t)kChunk ? K - k0 : (uint32_t)kChunk;
            for(uint32_t kk = 0; kk < n; ++kk)
            {
                const Acc u = s_u[kk][threadIdx.x];
#pragma unroll
                for(int j = 0; j < TX; ++j)
                    acc[c][j] = madd(acc[c][j], u, s_sxv[kk][j]);
            }
        }
    }
    store_texels<Acc, TX>(a, acc, t0, lv0);
}

constexpr int kTilePairs = 128, kTileTexels = 64, kTileThreads = 256, kTileK = 16;

__device__ __forceinline__ float2 pair_madd(float2 sum, float2 u, float v, const __half*)
{
    return __ffma2_rn(u, make_float2(v, v), sum);
}
// (the paired multiply and add would be contracted)
__device__ __forceinline__ float2 pair_madd(float2 sum, float2 u, float v, const float*)
{
    return make_float2(__fadd_rn(sum.x, __fmul_rn(u.x, v)), __fadd_rn(sum.y, __fmul_rn(u.y, v)));
}

// kE consecutive elements of a row, as they lie in the file.
template <typename T, int kE>
struct alignas(sizeof(T) * kE < 16 ? sizeof(T) * kE : 16) Elems { T v[kE]; };

// Elements k0 .. k0 + kE - 1 of a row of K, 0 past K.  kWide: the row is aligned to
// Elems<T, kE> at k0 and K is a multiple of kE.
template <bool kWide, typename T, int kE>
__device__ __forceinline__ void load_elems(const T* row, uint32_t k0, uint32_t K, bool ok, Elems<T, kE>& e)
{
    if constexpr(kWide)
    {
        if(ok && k0 < K)
            e = *reinterpret_cast<const Elems<T, kE>*>(row + k0);
        else
#pragma unroll
            for(int i = 0; i < kE; ++i)
                e.v[i] = T(0.0f);
    }
    else
#pragma unroll
        for(int i = 0; i < kE; ++i)
            e.v[i] = ok && k0 + i < K ? row[k0 + i] : T(0.0f);
}

// Column swaps of the staged operands' upper 8 rows, so that the lanes that stage
// consecutive pieces of one row do not meet in a bank.
__device__ __forceinline__ int swap_u(int kk) { return kk >= 8 ? 16 : 0; }
__device__ __forceinline__ int swap_s(int kk) { return kk >= 8 ? 8 : 0; }

// Thread (tl, tx): pairs tl * 4 + {0..3} and 64 + tl * 4 + {0..3}, texels tx * 4 +
// {0..3}; a warp is 8 tl x 4 tx.  The components go by in tiles of 16 through two
// shared buffers, the next tile's elements in registers during this one's products.
template <typename T, bool kWide>
__global__ void __launch_bounds__(kTileThreads, 2) btf_decode_tile_kernel(BtfDecodeArgs a, uint64_t t_begin)
{
    constexpr int TX = 4, kTexels = kTileTexels;
    constexpr int kS = kTexels * kTileK / kTileThreads;   // elements of SxV a thread stages of a tile
    struct Operands
    {
        float u[2][kTileK][kTilePairs + 4];
        float s[2][kTileK][kTexels + 4];
    };
    union Shared   // the samples leave through the operands' memory
    {
        Operands op;
        float out[kTileThreads / 32][4][2][96];
    };
    __shared__ __align__(16) unsigned char s_mem[sizeof(Shared)];
    Shared& sh = *reinterpret_cast<Shared*>(s_mem);
    const uint32_t lv0 = blockIdx.x * kTilePairs;
    const uint64_t t0 = t_begin + (uint64_t)blockIdx.y * kTexels;
    const uint64_t t_end = a.first + a.count;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tl = (lane & 7) + 8 * (warp & 1), tx = (lane >> 3) + 4 * (warp >> 1);
    // staging: U elements 8 pu .. of pair lu; SxV elements kS ps .. of texel ls, whose
    // file column is row H - 1 - y
    const int lu = threadIdx.x / 2, pu = threadIdx.x % 2;
    const int ls = threadIdx.x / (kTileK / kS), ps = threadIdx.x % (kTileK / kS);
    const bool u_ok = lv0 + lu < a.N, s_ok = t0 + ls < t_end;
    uint64_t col = 0;
    if(s_ok)
    {
        const uint64_t t = t0 + ls, y = t / a.width;
        col = (a.height - 1 - y) * a.width + (t - y * a.width);
    }
    float2 acc[3][4][TX];
#pragma unroll
    for(int c = 0; c < 3; ++c)
#pragma unroll
        for(int i = 0; i < 4; ++i)
#pragma unroll
            for(int j = 0; j < TX; ++j)
                acc[c][i][j] = make_float2(0.0f, 0.0f);
    int buf = 0;
#pragma unroll
    for(int c = 0; c < 3; ++c)
    {
        const T* U = static_cast<const T*>(a.u[c]) + (uint64_t)(u_ok ? lv0 + lu : 0) * a.u_row[c] + 8 * pu;
        const T* S = static_cast<const T*>(a.sxv[c]) + col * a.sxv_row[c] + kS * ps;
        const uint32_t K = a.k[c], Ku = K > 8u * pu ? K - 8 * pu : 0, Ks = K > (uint32_t)(kS * ps) ? K - kS * ps : 0;
        Elems<T, 8> ru;
        Elems<T, kS> rs;
        load_elems<kWide>(U, 0, Ku, u_ok, ru);
        load_elems<kWide>(S, 0, Ks, s_ok, rs);
        for(uint32_t k0 = 0; k0 < K; k0 += kTileK)
        {
#pragma unroll
            for(int i = 0; i < 8; ++i)
                sh.op.u[buf][8 * pu + i][lu ^ swap_u(8 * pu)] = elem(ru.v, i);
#pragma unroll
            for(int i = 0; i < kS; ++i)
                sh.op.s[buf][kS * ps + i][ls ^ swap_s(kS * ps)] = elem(rs.v, i);
            __syncthreads();   // (a buffer is written again two tiles on, past the next barrier)
            if(k0 + kTileK < K)
            {
                load_elems<kWide>(U, k0 + kTileK, Ku, u_ok, ru);
                load_elems<kWide>(S, k0 + kTileK, Ks, s_ok, rs);
            }
            const uint32_t n = K - k0 < (uint32_t)kTileK ? K - k0 : (uint32_t)kTileK;
            auto step = [&](uint32_t kk) {
                const float4 u0 = *reinterpret_cast<const float4*>(&sh.op.u[buf][kk][(4 * tl) ^ swap_u(kk)]);
                const float4 u1 = *reinterpret_cast<const float4*>(&sh.op.u[buf][kk][64 + ((4 * tl) ^ swap_u(kk))]);
                const float2 u[4] = { make_float2(u0.x, u0.y), make_float2(u0.z, u0.w), make_float2(u1.x, u1.y),
                                      make_float2(u1.z, u1.w) };
                const float4 s0 = *reinterpret_cast<const float4*>(&sh.op.s[buf][kk][(4 * tx) ^ swap_s(kk)]);
                const float v[TX] = { s0.x, s0.y, s0.z, s0.w };
#pragma unroll
                for(int j = 0; j < TX; ++j)
#pragma unroll
                    for(int i = 0; i < 4; ++i)
                        acc[c][i][j] = pair_madd(acc[c][i][j], u[i], v[j], static_cast<const T*>(nullptr));
            };
            if(n == (uint32_t)kTileK)
            {
#pragma unroll 8
                for(uint32_t kk = 0; kk < (uint32_t)kTileK; ++kk)
                    step(kk);
            }
            else
                for(uint32_t kk = 0; kk < n; ++kk)
                    step(kk);
            buf ^= 1;
        }
    }
    // samples out: two of a warp's texels at a time through shared memory, so that its
    // stores are consecutive
    __syncthreads();
    float(*out)[2][96] = sh.out[warp];
#pragma unroll
    for(int j = 0; j < TX; ++j)
    {
#pragma unroll
        for(int g = 0; g < 2; ++g)
        {
            float v[12];   // the group's four pairs
#pragma unroll
            for(int i = 0; i < 2; ++i)
#pragma unroll
                for(int c = 0; c < 3; ++c)
                {
                    v[6 * i + c] = acc[c][2 * g + i][j].x;
                    v[6 * i + 3 + c] = acc[c][2 * g + i][j].y;
                }
#pragma unroll
            for(int p = 0; p < 4; ++p)
                to_sample(a, v + 3 * p);
#pragma unroll
            for(int w = 0; w < 3; ++w)
                *reinterpret_cast<float4*>(&out[lane >> 3][g][12 * (lane & 7) + 4 * w]) =
                    make_float4(v[4 * w], v[4 * w + 1], v[4 * w + 2], v[4 * w + 3]);
        }
        __syncwarp();
#pragma unroll
        for(int r = 0; r < 4; ++r)
        {
            const uint64_t t = t0 + (uint64_t)(4 * (warp >> 1) + r) * TX + j;
            if(t >= t_end)
                continue;
#pragma unroll
            for(int g = 0; g < 2; ++g)
            {
                const uint32_t lv = lv0 + 64 * g + 32 * (warp & 1);
                const uint32_t values = lv >= a.N ? 0 : a.N - lv < 32 ? 3 * (a.N - lv) : 96;
                const uint64_t o = ((t - a.first) * a.N + lv) * 3;
                if(a.out_type == SVF_SAMPLES_F16)
                {
#pragma unroll
                    for(uint32_t e = lane; e < 96; e += 32)
                        if(e < values)
                            static_cast<__half*>(a.out)[o + e] = __float2half_rn(out[r][g][e]);
                }
                else
#pragma unroll
                    for(uint32_t e = lane; e < 96; e += 32)
                        if(e < values)
                            static_cast<float*>(a.out)[o + e] = out[r][g][e];
            }
        }
        __syncwarp();
    }
}

template <typename T, bool kWide>
cudaError_t launch_tiles_of(const BtfDecodeArgs& a, cudaStream_t stream)
{
    constexpr uint64_t texels = kTileTexels, per_launch = 65535ull * texels;   // grid.y limit
    for(uint64_t t = a.first; t < a.first + a.count; t += per_launch)
    {
        const uint64_t n = a.first + a.count - t < per_launch ? a.first + a.count - t : per_launch;
        const dim3 grid((a.N + kTilePairs - 1) / kTilePairs, (unsigned)((n + texels - 1) / texels));
        btf_decode_tile_kernel<T, kWide><<<grid, kTileThreads, 0, stream>>>(a, t);
        const cudaError_t e = cudaGetLastError();
        if(e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

template <typename T>
cudaError_t launch_tiles(const BtfDecodeArgs& a, cudaStream_t stream)
{
    // Elems loads of 8 components want aligned rows of whole groups; 47 components, an
    // element at a time, take 10.1 ms where 48 take 8.6
    bool wide = true;
    for(int c = 0; c < 3; ++c)
        wide = wide && a.k[c] % 8 == 0 && a.u_row[c] * sizeof(T) % 16 == 0 && a.sxv_row[c] * sizeof(T) % 16 == 0 &&
               (uintptr_t)a.u[c] % 16 == 0 && (uintptr_t)a.sxv[c] % 16 == 0;
    return wide ? launch_tiles_of<T, true>(a, stream) : launch_tiles_of<T, false>(a, stream);
}

template <typename T, typename Acc, int TX>
cudaError_t launch_typed(const BtfDecodeArgs& a, cudaStream_t stream)
{
    const uint64_t per_launch = 65535ull * TX;   // grid.y limit
    for(uint64_t t = a.first; t < a.first + a.count; t += per_launch)
    {
        const uint64_t n = a.first + a.count - t < per_launch ? a.first + a.count - t : per_launch;
        dim3 grid((a.N + kThreads - 1) / kThreads, (unsigned)((n + TX - 1) / TX));
        btf_decode_kernel<T, Acc, TX><<<grid, kThreads, 0, stream>>>(a, t);
        const cudaError_t e = cudaGetLastError();
        if(e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

} // namespace

cudaError_t launch_btf_decode(const BtfDecodeArgs& a, cudaStream_t stream)
{
    if(a.count == 0)
        return cudaSuccess;
    switch(a.data_size)
    {
    case 2: return launch_tiles<__half>(a, stream);
    case 4: return launch_tiles<float>(a, stream);
    case 8: return launch_typed<double, double, 16>(a, stream);
    default: return cudaErrorInvalidValue;
    }
}

} // namespace svf
