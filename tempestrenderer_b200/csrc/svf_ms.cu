// svf_ms.cu - the pseudo-volume multi-scattering BRDF (svbrdffit -m).
//
// SGGXMicroFlakePseudoVolumeBRDF (ggx-models-impl.hh:621-758): a single-
// scattering term plus `samples` random walks of at most `depth` scattering
// events inside a pseudo volume of SGGX micro-flakes, the walks of one
// evaluation drawing from one LCG sequence (FastFloatRand, functions.hh:214-
// 252) in order.  Because a walk's start state depends on how many numbers the
// walks before it drew, the walks of an evaluation run in order on one thread;
// the parallelism is over texels, direction pairs and (for the Jacobian) the
// 14 perturbed parameter vectors of a pair.
//
//   ms_render_kernel    the BTF of SVBRDF maps with this BRDF (RGB); of many pairs
//                       ms_walk_kernel, ms_lookup_kernel and ms_rest_kernel
//   ms_eval_kernel      residuals of the luminance fit, or the 14 central-
//                       difference evaluations of a pair's Jacobian row
//   ms_reduce_kernel    a texel's residual sum, or J^T J and J^T r (FP64, fixed order)
//   ms_control_kernel   the LM step logic of LevenbergMarquardtCurveFit
//                       (fitting.hh:457-678), one thread per texel, FP64
//
// This file is compiled with -fmad=false: every float operation rounds as in
// the reference's x86-64 build (no fused multiply-adds), so an evaluation
// differs from the reference's only through the last bits of logf, expf and
// tanf (and, rarely, a walk that those bits send across one of its break tests).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/svf.h"
#include "svf_internal.h"

namespace svf
{
namespace
{

constexpr float kPi = 3.141592f;   // functions.hh:55

struct V3
{
    float x, y, z;
};
__device__ __forceinline__ V3 v3(float x, float y, float z) { return V3{ x, y, z }; }
__device__ __forceinline__ V3 add(V3 a, V3 b) { return v3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ V3 sub(V3 a, V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ V3 mul(V3 a, V3 b) { return v3(a.x * b.x, a.y * b.y, a.z * b.z); }
// Vector3 * float (vector3.hh:159,163)
__device__ __forceinline__ V3 scale(V3 a, float s) { return v3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float len(V3 a) { return sqrtf(a.x * a.x + a.y * a.y + a.z * a.z); }
// Vector3 / float multiplies by the reciprocal (vector3.hh:185-190)
__device__ __forceinline__ V3 divs(V3 a, float s)
{
    const float r = 1.0f / s;
    return scale(a, r);
}
__device__ __forceinline__ V3 normalize(V3 a)
{
    const float l = len(a);
    return l != 0.0f ? divs(a, l) : a;
}
__device__ __forceinline__ V3 cross(V3 a, V3 b)
{
    return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
// Reflect (vector3.hh:420): 2 (n . i) n - i
__device__ __forceinline__ V3 reflect(V3 i, V3 n) { return sub(scale(n, 2.0f * dot(n, i)), i); }

// A 3x3 matrix by columns, as Matrix3::Columns (matrix3.hh:40-56).
struct M3
{
    V3 c[3];
};

// Matrix3 * Matrix3 (matrix3.hh:355-360)
__device__ __forceinline__ M3 mmul(const M3& l, const M3& r)
{
    M3 o;
#pragma unroll
    for(int j = 0; j < 3; ++j)
        o.c[j] = add(add(scale(l.c[0], r.c[j].x), scale(l.c[1], r.c[j].y)), scale(l.c[2], r.c[j].z));
    return o;
}

__device__ __forceinline__ M3 transpose(const M3& m)
{
    M3 o;
    o.c[0] = v3(m.c[0].x, m.c[1].x, m.c[2].x);
    o.c[1] = v3(m.c[0].y, m.c[1].y, m.c[2].y);
    o.c[2] = v3(m.c[0].z, m.c[1].z, m.c[2].z);
    return o;
}

// Matrix3::transformCovariance (matrix3.hh:151-158): B diag(var) B^T
__device__ __forceinline__ M3 covariance(const M3& b, V3 var)
{
    M3 o;
    o.c[0] = add(add(scale(scale(b.c[0], var.x), b.c[0].x), scale(scale(b.c[1], var.y), b.c[1].x)),
                 scale(scale(b.c[2], var.z), b.c[2].x));
    o.c[1] = add(add(scale(scale(b.c[0], var.x), b.c[0].y), scale(scale(b.c[1], var.y), b.c[1].y)),
                 scale(scale(b.c[2], var.z), b.c[2].y));
    o.c[2] = add(add(scale(scale(b.c[0], var.x), b.c[0].z), scale(scale(b.c[1], var.y), b.c[1].z)),
                 scale(scale(b.c[2], var.z), b.c[2].z));
    return o;
}

__device__ __forceinline__ V3 transform(const M3& m, V3 v)
{
    return add(add(scale(m.c[0], v.x), scale(m.c[1], v.y)), scale(m.c[2], v.z));
}

// Matrix3::transformRotationInverse (matrix3.hh:139-142): B^T v
__device__ __forceinline__ V3 rot_inverse(const M3& m, V3 v) { return v3(dot(v, m.c[0]), dot(v, m.c[1]), dot(v, m.c[2])); }

// Matrix3::makeBasis (matrix3.hh:99-108): a frame whose third column is n
__device__ __forceinline__ M3 basis_of(V3 n)
{
    const V3 d0 = cross(v3(1.0f, 0.0f, 0.0f), n), d1 = cross(v3(0.0f, 1.0f, 0.0f), n);
    const float l0 = dot(d0, d0), l1 = dot(d1, d1);
    M3 o;
    o.c[0] = l0 > l1 ? divs(d0, sqrtf(l0)) : divs(d1, sqrtf(l1));
    o.c[1] = cross(n, o.c[0]);
    o.c[2] = n;
    return o;
}

// Matrix3::choleskyDecomposition (matrix3.hh:173-191)
__device__ __forceinline__ M3 cholesky(const M3& m)
{
    const float l00 = sqrtf(m.c[0].x);
    const float r00 = 1.0f / l00;
    const float l10 = r00 * m.c[0].y;
    const float l20 = r00 * m.c[0].z;
    const float l11 = sqrtf(m.c[1].y - l10 * l10);
    const float r11 = 1.0f / l11;
    const float l21 = r11 * (m.c[1].z - l20 * l10);
    const float l22 = sqrtf(m.c[2].z - l21 * l21 - l20 * l20);
    M3 o;
    o.c[0] = v3(l00, l10, l20);
    o.c[1] = v3(0.0f, l11, l21);
    o.c[2] = v3(0.0f, 0.0f, l22);
    return o;
}

// FloatIntelFastRand (functions.hh:214-218,249-252)
__device__ __forceinline__ float lcg_value(unsigned s) { return (float)((s >> 16) & 0x7FFFu) / 32767.0f; }
__device__ __forceinline__ float lcg(unsigned& s)
{
    s = 214013u * s + 2531011u;
    return lcg_value(s);
}

// SinCos_Tan (functions.hh:322-329), the reference's FastSinCos on the CPU
__device__ __forceinline__ void sincos_tan(float w, float* s, float* c)
{
    const float t = tanf(w * 0.5f);
    const float t2 = t * t;
    const float d = 1.0f / (1.0f + t2);
    *s = 2.0f * t * d;
    *c = (1.0f - t2) * d;
}

// SGGXProjectedArea (ggx-models-impl.hh:102-105)
__device__ __forceinline__ float projected_area(V3 sd, const M3& b, V3 w) { return len(mul(rot_inverse(b, w), sd)); }

// SGGXMicroFlakeNDF(stddev, basis, normal) (ggx-models-impl.hh:49-57), split
// into what one evaluation's parameters fix (the inverse covariance, its
// determinant test and the numerator 0.5 sqrt(det)) and the per-normal rest;
// the same operations in the same order as the reference's single function.
struct NdfConst
{
    M3 ic;
    float num;   // 0.5 sqrt(det); 0 where det < 1e-6 (the reference returns 0)
};

__device__ __forceinline__ NdfConst ndf_const(V3 sd, const M3& b)
{
    const V3 sq = mul(sd, sd);
    NdfConst k;
    k.ic = covariance(b, v3(1.0f / sq.x, 1.0f / sq.y, 1.0f / sq.z));
    const M3& ic = k.ic;
    // Matrix3::determinant (matrix3.hh:193-201), Elements[i][j] = column i, row j
    const float det = ic.c[0].x * (ic.c[1].y * ic.c[2].z - ic.c[1].z * ic.c[2].y) -
                      ic.c[1].x * (ic.c[0].y * ic.c[2].z - ic.c[0].z * ic.c[2].y) +
                      ic.c[2].x * (ic.c[0].y * ic.c[1].z - ic.c[0].z * ic.c[1].y);
    k.num = det < 1e-6f ? 0.0f : 0.5f * sqrtf(det);
    return k;
}

__device__ __forceinline__ float sggx_ndf(const NdfConst& k, V3 n)
{
    if(k.num == 0.0f)
        return 0.0f;
    const float den = dot(n, transform(k.ic, n));
    return k.num / (kPi * den * den);
}

// UniformSampleSphere (sampling3.hh:106-116) of the walk's next two numbers: the
// reference's GCC build evaluates its two FastFloatRand arguments right to left, so
// rb is the first drawn.
__device__ __forceinline__ V3 sample_sphere(float rb, float ra)
{
    float s, c;
    sincos_tan(2.0f * kPi * ra, &s, &c);
    const float ct = 2.0f * rb - 1.0f;
    const float st = sqrtf(1.0f - ct * ct);
    return v3(c * st, s * st, ct);
}

// The numbers of an evaluation's walks.  Every evaluation of a launch draws from one
// sequence (the seed is the launch's), so what the walks make of the numbers at a
// position is the same in all of them: entry j of the table holds the sphere sample
// of draws j and j + 1 and -log of draw j + 2, by the same operations as without it.
// An event is then one 16-byte load, in place of three LCG steps and divisions, a
// tangent, a square root and a logarithm.
__device__ __forceinline__ void fill_walk_table(float4* tab, uint32_t entries, unsigned seed)
{
    for(uint32_t j = threadIdx.x; j < entries; j += blockDim.x)
    {
        unsigned mul_n = 1u, add_n = 0u, mul_1 = 214013u, add_1 = 2531011u;   // the LCG's j-th power
        for(uint32_t n = j; n; n >>= 1)
        {
            if(n & 1)
            {
                add_n = add_n * mul_1 + add_1;
                mul_n *= mul_1;
            }
            add_1 *= mul_1 + 1u;
            mul_1 *= mul_1;
        }
        unsigned st = mul_n * seed + add_n;
        const float rb = lcg_value(st);
        const float ra = lcg(st);
        const V3 u = sample_sphere(rb, ra);
        tab[j] = make_float4(u.x, u.y, u.z, -logf(lcg(st)));
    }
    __syncthreads();
}

// The draws of `samples` walks of `depth` events, and so the table's entries.
__host__ __device__ __forceinline__ uint64_t walk_draws(uint32_t samples, uint32_t depth)
{
    return 1 + (uint64_t)samples * (1 + 3 * (uint64_t)depth);
}

template <bool kTable>
struct Draws
{
    const float4* tab;
    uint32_t pos;     // draws so far (kTable)
    unsigned state;   // the LCG's state (!kTable)

    __device__ __forceinline__ float walk_log()
    {
        if constexpr(kTable)
            return tab[pos++ - 1].w;
        else
            return -logf(lcg(state));
    }
    // an event's sphere sample and the -log of the number after it
    __device__ __forceinline__ V3 event(float* log_next)
    {
        if constexpr(kTable)
        {
            const float4 e = tab[pos + 1];
            pos += 3;
            *log_next = e.w;
            return v3(e.x, e.y, e.z);
        }
        else
        {
            const float rb = lcg(state);
            const float ra = lcg(state);
            const V3 u = sample_sphere(rb, ra);
            *log_next = -logf(lcg(state));
            return u;
        }
    }
};

// What SGGXMicroFlakeSampleIncidentLight (ggx-models-impl.hh:554-570) makes of its
// direction alone: the frame and the Cholesky factor of the covariance seen in it.
// cov: Matrix3::transformCovariance of the basis by stddev^2, fixed per evaluation.
struct Seen
{
    M3 ob, chol;
};
__device__ __forceinline__ Seen seen_from(V3 wo, const M3& cov)
{
    Seen v;
    v.ob = basis_of(wo);
    v.chol = cholesky(mmul(mmul(v.ob, cov), transpose(v.ob)));
    return v;
}

// The rest of it: a visible normal of the distribution seen from `wo`, and wo
// reflected about it.
__device__ __forceinline__ V3 sample_incident(V3 wo, const Seen& v, V3 u)
{
    const V3 vn = transform(v.ob, normalize(rot_inverse(v.chol, u)));
    return reflect(wo, vn);
}

// The next scattering event of a walk that looks along out_l at depth_in: the
// direction it leaves in, the projected area along it and the depth where the next
// event lies.
template <bool kTable>
__device__ __forceinline__ void scatter(Draws<kTable>& draws, const Seen& seen, V3 sd, const M3& b, V3& out_l,
                                        float& depth_in, float& dd)
{
    float log_next;
    const V3 u = draws.event(&log_next);
    const V3 inc_l = sample_incident(out_l, seen, u);
    dd = projected_area(sd, b, inc_l);
    out_l = v3(-inc_l.x, -inc_l.y, -inc_l.z);
    depth_in += (log_next / dd) * out_l.z;
}

// SGGXMicroFlakePseudoVolumeBRDF in the fitting frame (tangent x, binormal y,
// normal z) for C spectrum channels; a walk continues while every channel's
// throughput is above 1e-3.  The reference's Fresnel branch is compiled out
// (USE_PSEUDO_VOLUME_FRESNEL is not defined).  One (light, view) pair's evaluation:
template <int C>
struct PairEval
{
    V3 wi, wo;
    float in_density, rad[C];
    NdfConst nk;

    // false: the BRDF is zero
    __device__ __forceinline__ static bool lit(V3 sd, V3 wi, V3 wo)
    {
        return !(wo.z < 0.0f || wi.z < 0.0f) && !(sd.x < 1e-6f || sd.y < 1e-6f);
    }
    // the single-scattering term
    __device__ __forceinline__ void start(const float* spec, V3 sd, const M3& b, float out_density, V3 wi_, V3 wo_,
                                          uint32_t samples)
    {
        wi = wi_;
        wo = wo_;
        const float dot_inc = wi.z, dot_out = wo.z;
        in_density = projected_area(sd, b, wi);
        const V3 h = normalize(add(wo, wi));
        const float contrib = (float)samples / (out_density + in_density * dot_out / dot_inc);
        // what the evaluation's parameters fix, computed once (the reference recomputes it per call)
        nk = ndf_const(sd, b);
        const float ndf = sggx_ndf(nk, h);
#pragma unroll
        for(int c = 0; c < C; ++c)
            rad[c] = spec[c] * contrib * ndf * 2.0f * 0.25f;
    }
    // the light from wi that an event at depth_in sends along the walk; dd4: 4 times
    // the projected area along it.  Whether it is visible there (the walk ends else).
    __device__ __forceinline__ bool event(const float* spec, V3 out_l, float depth_in, float dd4, float* thr)
    {
        const float ext = expf(-in_density * (depth_in / wi.z));
        if(ext < 1e-9f)
            return false;
        const float f = sggx_ndf(nk, normalize(add(out_l, wi))) * 2.0f / dd4;
#pragma unroll
        for(int c = 0; c < C; ++c)
        {
            thr[c] *= spec[c];
            rad[c] += ext * thr[c] * f;
        }
        return true;
    }
    __device__ __forceinline__ static bool alive(const float* thr)
    {
        bool on = true;
#pragma unroll
        for(int c = 0; c < C; ++c)
            on = on && thr[c] > 1e-3f;
        return on;
    }
    // walks first .. samples - 1
    template <bool kTable>
    __device__ __forceinline__ void walks(const float* spec, V3 sd, const M3& b, float out_density, uint32_t depth,
                                          uint32_t first, uint32_t samples, Draws<kTable> draws)
    {
        if(depth == 0 || !alive(spec))
            return;
        const M3 cov = covariance(b, mul(sd, sd));
        // every walk starts along wo; without the table of draws the frame's registers
        // cost more than it (24 texels of 40 directions at depth 9: 221 ms a fit against
        // 206), and so does one loop for both (221 against 216)
        Seen seen0;
        if constexpr(kTable)
            seen0 = seen_from(wo, cov);
        float thr[C];
        for(uint32_t s = first; s < samples; ++s)
        {
#pragma unroll
            for(int c = 0; c < C; ++c)
                thr[c] = spec[c];
            V3 out_l = wo;
            float depth_in = (draws.walk_log() / out_density) * wo.z, dd;
            if constexpr(kTable)
            {
                scatter(draws, seen0, sd, b, out_l, depth_in, dd);
                for(uint32_t it = 1;; ++it)
                {
                    if(depth_in < 0.0f || !event(spec, out_l, depth_in, 4.0f * dd, thr) || it == depth || !alive(thr))
                        break;
                    scatter(draws, seen_from(out_l, cov), sd, b, out_l, depth_in, dd);
                }
            }
            else
                for(uint32_t it = 0; it < depth && alive(thr); ++it)
                {
                    scatter(draws, seen_from(out_l, cov), sd, b, out_l, depth_in, dd);
                    if(depth_in < 0.0f || !event(spec, out_l, depth_in, 4.0f * dd, thr))
                        break;
                }
        }
    }
    __device__ __forceinline__ void finish(const float* diff, uint32_t samples, float* out) const
    {
        const float rcp = 1.0f / (float)samples;
#pragma unroll
        for(int c = 0; c < C; ++c)
            out[c] = rad[c] * rcp + diff[c] * wi.z * (1.0f / kPi);
    }
};

// The sequence's first draw is dropped.
template <bool kTable>
__device__ __forceinline__ Draws<kTable> first_draws(unsigned seed, const float4* tab)
{
    (void)lcg(seed);
    return Draws<kTable>{ tab, 1u, seed };
}

template <int C, bool kTable>
__device__ __forceinline__ void pseudo_volume(const float* spec, const float* diff, V3 sd, const M3& b,
                                              float out_density, V3 wi, V3 wo, uint32_t depth, uint32_t samples,
                                              unsigned seed, const float4* tab, float* out)
{
#pragma unroll
    for(int c = 0; c < C; ++c)
        out[c] = 0.0f;
    if(!PairEval<C>::lit(sd, wi, wo))
        return;
    PairEval<C> e;
    e.start(spec, sd, b, out_density, wi, wo, samples);
    e.walks(spec, sd, b, out_density, depth, 0, samples, first_draws<kTable>(seed, tab));
    e.finish(diff, samples, out);
}

// ToQuaternion(euler) (quaternion.hh:82-94) with the reference's FastSinCos,
// then ToMatrix3 (quaternion.hh:122-139) of the unnormalised quaternion, as
// the pseudo-volume BRDF takes it (ggx-models-impl.hh:660).
__device__ __forceinline__ M3 quat_matrix(const float* r)
{
    const float xx = r[0] * r[0], xy = r[0] * r[1], xz = r[0] * r[2], xw = r[0] * r[3];
    const float yy = r[1] * r[1], yz = r[1] * r[2], yw = r[1] * r[3];
    const float zz = r[2] * r[2], zw = r[2] * r[3];
    M3 m;
    m.c[0] = v3(1.0f - 2.0f * (yy + zz), 2.0f * (xy + zw), 2.0f * (xz - yw));
    m.c[1] = v3(2.0f * (xy - zw), 1.0f - 2.0f * (xx + zz), 2.0f * (yz + xw));
    m.c[2] = v3(2.0f * (xz + yw), 2.0f * (yz - xw), 1.0f - 2.0f * (xx + yy));
    return m;
}

__device__ __forceinline__ M3 euler_matrix(const float* e)
{
    float s1, c1, s2, c2, s3, c3;
    sincos_tan(0.5f * e[0], &s1, &c1);
    sincos_tan(0.5f * e[1], &s2, &c2);
    sincos_tan(0.5f * e[2], &s3, &c3);
    const float q[4] = { s1 * c2 * c3 + c1 * s2 * s3, -s1 * c2 * s3 + c1 * s2 * c3, c1 * c2 * s3 + s1 * s2 * c3,
                         c1 * c2 * c3 - s1 * s2 * s3 };
    return quat_matrix(q);
}

constexpr uint32_t kFitWalks = 256;

// BRDFEvaluator::operator() with BounceCount = depth (svbrdf-lsq-fitting-
// internal.hh:91-153): parameters handed over as doubles and rounded to float,
// 256 walks from LCG seed 0 (the evaluator's texture coordinate is 0).
template <bool kTable>
__device__ float evaluator_ms(const double* pd, V3 wi, V3 wo, uint32_t depth, const float4* tab)
{
    float p[7];
#pragma unroll
    for(int k = 0; k < 7; ++k)
        p[k] = (float)pd[k];
    const V3 sd = v3(p[0] > 0.0f ? p[0] : 0.0f, p[1] > 0.0f ? p[1] : 0.0f, 1.0f);
    const M3 b = euler_matrix(p + 4);
    const float ks = p[2] > 0.0f ? p[2] : 0.0f;
    const float kd = p[3] > 0.0f ? p[3] : 0.0f;
    float r;
    pseudo_volume<1, kTable>(&ks, &kd, sd, b, projected_area(sd, b, wo), wi, wo, depth, kFitWalks, 0u, tab, &r);
    return r;
}

__device__ __forceinline__ V3 direction(const float* geo, uint32_t L, uint32_t d)
{
    return v3(geo[d], geo[L + d], geo[2 * L + d]);
}

constexpr int kMsThreads = 256, kWalkThreads = 64;
// The kernels that walk pair by pair: blocks that share a table of draws are larger.
// 24 warps an SM (80 registers), 16 where the table leaves room for two blocks (6 and 7
// events: a fit of 24 texels of 40 directions takes 150 and 172 ms with it, 174 and 199
// without).
__host__ __device__ constexpr int ms_threads(bool table) { return table ? kMsThreads : 128; }
__host__ __device__ constexpr int ms_blocks(bool table) { return table ? 3 : 6; }

// Shared memory of the walk table; 0 where there is none: up to 96 KB (256 walks of 7
// events take 90 KB), twice of which fits on an SM.
size_t walk_table_bytes(uint32_t samples, uint32_t depth)
{
    const uint64_t bytes = sizeof(float4) * walk_draws(samples, depth);
    return bytes <= 96 * 1024 ? (size_t)bytes : 0;
}

template <typename Kernel>
cudaError_t allow_smem(Kernel* kernel, size_t bytes)
{
    if(bytes <= 48 * 1024)
        return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(96 * 1024));
}

} // namespace

// ---- rendering ----------------------------------------------------------------------

namespace
{

// A texel's material from the maps.
struct MsMaterial
{
    V3 sd;
    float kd[3], ks[3];
    M3 b;
};
__device__ __forceinline__ MsMaterial ms_material(const MsRenderArgs& a, uint64_t t)
{
    MsMaterial m;
    float sx = a.sigma[a.sigma_channels * t], sy = a.sigma[a.sigma_channels * t + 1];
    if(a.sigma_channels == 3)
    {
        const float sz = a.sigma[3 * t + 2];
        sx = sx / sz;
        sy = sy / sz;
    }
    m.sd = v3(sx > 0.0f ? sx : 0.0f, sy > 0.0f ? sy : 0.0f, 1.0f);
    float q[4];
#pragma unroll
    for(int k = 0; k < 4; ++k)
        q[k] = a.basis[4 * t + k];
#pragma unroll
    for(int c = 0; c < 3; ++c)
    {
        m.kd[c] = fmaxf(a.diffuse[3 * t + c], 0.0f);
        m.ks[c] = fmaxf(a.specular[3 * t + c], 0.0f);
    }
    m.b = quat_matrix(q);
    return m;
}

// A pair's three values in the output's sample type.
__device__ __forceinline__ void store_pair(const MsRenderArgs& a, uint64_t i, const float* f)
{
    const uint64_t o = i * 3;
#pragma unroll
    for(int c = 0; c < 3; ++c)
    {
        if(a.sample_type == SVF_SAMPLES_F16)
            static_cast<__half*>(a.out)[o + c] = __float2half_rn(f[c]);
        else
            static_cast<float*>(a.out)[o + c] = f[c];
    }
}

} // namespace

// The walks of an evaluation are those of its view: the light enters only in what an
// event sends along and in the test whether it still sees it (the walk ends there, and
// the evaluation's later numbers are others than its view's).  So the views' walks are
// worked out once (ms_walk_kernel) and the pairs look their events up
// (ms_lookup_kernel); a pair that loses sight of an event that its view's walk goes on
// from leaves its sums in a list, and the rest of its walks are its own
// (ms_rest_kernel).  16 x 16 texels of ring-81, 256 walks of two events: 0.31 + 4.0 +
// 1.1 to 1.4 ms (by the maps), where every pair walking by itself (ms_render_kernel)
// takes 10.0, and 16.0 without the table of draws.  Finishing the lost pairs in the lookup takes 9.9: a few
// lanes of a warp then walk for all, on half as many warps.
struct MsRest
{
    uint64_t i;        // the pair
    uint32_t s, pos;   // its next walk, the draws before it
    float rad[3];
};

struct MsWalks
{
    float4* ev;      // [texel][view][walk][event]: direction, depth
    float* dd4;      // 4 times the projected area along it
    MsRest* rest;    // room for every pair
    uint32_t* lost;  // their number
};

// One thread per (texel, view): the walks as they go on while no light loses sight of
// an event; one that leaves the volume ends with a record of negative depth.
__global__ void __launch_bounds__(kWalkThreads) ms_walk_kernel(MsRenderArgs a, MsWalks w)
{
    extern __shared__ float4 walk_table[];
    fill_walk_table(walk_table, (uint32_t)walk_draws(a.samples, a.bounces), a.seed);
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i == 0)
        *w.lost = 0;
    if(i >= a.count * a.L)
        return;
    const MsMaterial m = ms_material(a, i / a.L);
    const V3 wo = direction(a.geo, a.L, (uint32_t)(i % a.L));
    if(!PairEval<3>::lit(m.sd, wo, wo) || !PairEval<3>::alive(m.ks))
        return;
    const float out_density = projected_area(m.sd, m.b, wo);
    const M3 cov = covariance(m.b, mul(m.sd, m.sd));
    const Seen seen0 = seen_from(wo, cov);
    Draws<true> draws = first_draws<true>(a.seed, walk_table);
    for(uint32_t s = 0; s < a.samples; ++s)
    {
        float thr[3] = { m.ks[0], m.ks[1], m.ks[2] };
        V3 out_l = wo;
        float depth_in = (draws.walk_log() / out_density) * wo.z, dd;
        scatter(draws, seen0, m.sd, m.b, out_l, depth_in, dd);
        for(uint32_t e = 0;;)
        {
            const uint64_t r = (i * a.samples + s) * a.bounces + e;
            w.ev[r] = make_float4(out_l.x, out_l.y, out_l.z, depth_in);
            w.dd4[r] = 4.0f * dd;
#pragma unroll
            for(int c = 0; c < 3; ++c)
                thr[c] *= m.ks[c];
            if(depth_in < 0.0f || ++e == a.bounces || !PairEval<3>::alive(thr))
                break;
            scatter(draws, seen_from(out_l, cov), m.sd, m.b, out_l, depth_in, dd);
        }
    }
}

// One thread per (texel, view, light), bound by the issue of the events' arithmetic
// (three divisions, a reciprocal, a square root and an exponential, correctly rounded).
__global__ void __launch_bounds__(kMsThreads, 4) ms_lookup_kernel(MsRenderArgs a, MsWalks w)
{
    const uint64_t N = (uint64_t)a.L * a.L;
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= a.count * N)
        return;
    const uint64_t t = i / N;
    const uint32_t lv = (uint32_t)(i % N);
    const uint32_t view = lv / a.L, light = lv % a.L;
    const MsMaterial m = ms_material(a, t);
    const V3 wi = direction(a.geo, a.L, light), wo = direction(a.geo, a.L, view);
    float f[3] = { 0.0f, 0.0f, 0.0f };
    if(PairEval<3>::lit(m.sd, wi, wo))
    {
        PairEval<3> p;
        p.start(m.ks, m.sd, m.b, projected_area(m.sd, m.b, wo), wi, wo, a.samples);
        const uint64_t first = (t * a.L + view) * a.samples * a.bounces;
        const float4* ev = w.ev + first;
        const float* dd4 = w.dd4 + first;
        uint32_t pos = 1;
        if(PairEval<3>::alive(m.ks))
            for(uint32_t s = 0; s < a.samples; ++s, ev += a.bounces, dd4 += a.bounces)
            {
                float thr[3] = { m.ks[0], m.ks[1], m.ks[2] };
                ++pos;
                bool lost = false;
                for(uint32_t e = 0;;)
                {
                    const float4 x = ev[e];
                    pos += 3;
                    if(x.w < 0.0f)
                        break;
                    const bool seen = p.event(m.ks, v3(x.x, x.y, x.z), x.w, dd4[e], thr);
                    if(!seen)   // (the view's throughput after the event)
#pragma unroll
                        for(int c = 0; c < 3; ++c)
                            thr[c] *= m.ks[c];
                    if(++e == a.bounces || !PairEval<3>::alive(thr))
                        break;
                    if(!seen)
                    {
                        lost = true;
                        break;
                    }
                }
                if(lost && s + 1 < a.samples)
                {
                    w.rest[atomicAdd(w.lost, 1u)] = MsRest{ i, s + 1, pos, { p.rad[0], p.rad[1], p.rad[2] } };
                    return;
                }
            }
        p.finish(m.kd, a.samples, f);
    }
    store_pair(a, i, f);
}

// Blocks of 128 threads (105 registers) where more than two of them have room for the
// table; else of 384 at 80 registers, so that two keep the SM busy: 256 texels of ring-81
// with orientations all over the sphere, 6 and 7 events, take 30.3 and 33.7 ms in all, 39.6
// and 44.8 in blocks of 128 (32.6 and 34.6 where every pair walks by itself without the
// table), with orientations near the normal 19.6 and 22.4 (23.0 and 27.4); at 4 events
// 64 texels take 3.65 ms, 3.94 in blocks of 384.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, kThreads > 128 ? 2 : 1) ms_rest_kernel(MsRenderArgs a, MsWalks w)
{
    extern __shared__ float4 walk_table[];
    const uint32_t lost = *w.lost;
    if((uint64_t)blockIdx.x * blockDim.x >= lost)
        return;
    fill_walk_table(walk_table, (uint32_t)walk_draws(a.samples, a.bounces), a.seed);
    const uint64_t N = (uint64_t)a.L * a.L;
    for(uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < lost; k += (uint64_t)gridDim.x * blockDim.x)
    {
        const MsRest r = w.rest[k];
        const uint32_t lv = (uint32_t)(r.i % N);
        const MsMaterial m = ms_material(a, r.i / N);
        const V3 wi = direction(a.geo, a.L, lv % a.L), wo = direction(a.geo, a.L, lv / a.L);
        PairEval<3> p;
        const float out_density = projected_area(m.sd, m.b, wo);
        p.start(m.ks, m.sd, m.b, out_density, wi, wo, a.samples);
#pragma unroll
        for(int c = 0; c < 3; ++c)
            p.rad[c] = r.rad[c];
        p.walks(m.ks, m.sd, m.b, out_density, a.bounces, r.s, a.samples, Draws<true>{ walk_table, r.pos, 0u });
        float f[3];
        p.finish(m.kd, a.samples, f);
        store_pair(a, r.i, f);
    }
}

// One thread per (texel, view, light), every pair with walks of its own: of few pairs,
// and where the views' walks have no room.
template <bool kTable>
__global__ void __launch_bounds__(ms_threads(kTable), ms_blocks(kTable)) ms_render_kernel(MsRenderArgs a)
{
    extern __shared__ float4 walk_table[];
    if constexpr(kTable)
        fill_walk_table(walk_table, (uint32_t)walk_draws(a.samples, a.bounces), a.seed);
    const uint64_t N = (uint64_t)a.L * a.L;
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= a.count * N)
        return;
    const uint32_t lv = (uint32_t)(i % N);
    const MsMaterial m = ms_material(a, i / N);
    const V3 wi = direction(a.geo, a.L, lv % a.L), wo = direction(a.geo, a.L, lv / a.L);
    float f[3];
    pseudo_volume<3, kTable>(m.ks, m.kd, m.sd, m.b, projected_area(m.sd, m.b, wo), wi, wo, a.bounces, a.samples, a.seed,
                             walk_table, f);
    store_pair(a, i, f);
}

uint64_t ms_walk_bytes(uint32_t L, uint32_t samples, uint32_t bounces)
{
    if(bounces == 0 || walk_table_bytes(samples, bounces) == 0)
        return 0;
    return (uint64_t)L * samples * bounces * (sizeof(float4) + sizeof(float)) + (uint64_t)L * L * sizeof(MsRest);
}

cudaError_t launch_ms_render(const MsRenderArgs& all, void* walks, uint64_t walk_texels, int sms, cudaStream_t stream)
{
    const uint64_t N = (uint64_t)all.L * all.L;
    if(all.count * N == 0)
        return cudaSuccess;
    const size_t smem = walk_table_bytes(all.samples, all.bounces);
    cudaError_t e = cudaSuccess;
    auto blocks_of = [](uint64_t n, int threads) { return (n + threads - 1) / threads; };
    if(!walks)
    {
        const uint64_t blocks = blocks_of(all.count * N, ms_threads(smem != 0));
        if(blocks > 0x7fffffffull)
            return cudaErrorInvalidValue;
        if(smem == 0)
            ms_render_kernel<false><<<(unsigned)blocks, ms_threads(false), 0, stream>>>(all);
        else if((e = allow_smem(ms_render_kernel<true>, smem)) != cudaSuccess)
            return e;
        else
            ms_render_kernel<true><<<(unsigned)blocks, kMsThreads, smem, stream>>>(all);
        return cudaGetLastError();
    }
    auto rest_kernel = ms_rest_kernel<128>;
    int rest_threads = 128, resident = 0;
    if((e = allow_smem(ms_walk_kernel, smem)) != cudaSuccess || (e = allow_smem(rest_kernel, smem)) != cudaSuccess ||
       (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, rest_kernel, rest_threads, smem)) != cudaSuccess)
        return e;
    if(resident <= 2)
    {
        rest_kernel = ms_rest_kernel<384>;
        rest_threads = 384;
        if((e = allow_smem(rest_kernel, smem)) != cudaSuccess ||
           (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, rest_kernel, rest_threads, smem)) != cudaSuccess)
            return e;
    }
    const uint64_t rest_blocks = (uint64_t)std::max(resident, 1) * sms;   // one wave
    MsWalks w;
    const uint64_t events = walk_texels * all.L * all.samples * all.bounces;
    w.lost = static_cast<uint32_t*>(walks);
    w.ev = reinterpret_cast<float4*>(w.lost + kMsWalkHeader / sizeof(uint32_t));
    w.rest = reinterpret_cast<MsRest*>(w.ev + events);
    w.dd4 = reinterpret_cast<float*>(w.rest + walk_texels * N);
    for(uint64_t t0 = 0; t0 < all.count; t0 += walk_texels)
    {
        MsRenderArgs a = all;
        a.count = all.count - t0 < walk_texels ? all.count - t0 : walk_texels;
        a.diffuse += 3 * t0;
        a.specular += 3 * t0;
        a.sigma += a.sigma_channels * t0;
        a.basis += 4 * t0;
        a.out = static_cast<char*>(a.out) + t0 * N * 3 * (a.sample_type == SVF_SAMPLES_F16 ? 2 : 4);
        const uint64_t pairs = blocks_of(a.count * N, kMsThreads), views = blocks_of(a.count * a.L, kWalkThreads);
        if(pairs > 0x7fffffffull || views > 0x7fffffffull || a.count * N > 0xffffffffull)
            return cudaErrorInvalidValue;
        ms_walk_kernel<<<(unsigned)views, kWalkThreads, smem, stream>>>(a, w);
        ms_lookup_kernel<<<(unsigned)pairs, kMsThreads, 0, stream>>>(a, w);
        const uint64_t rest = std::min(blocks_of(a.count * N, rest_threads), rest_blocks);
        rest_kernel<<<(unsigned)rest, rest_threads, smem, stream>>>(a, w);
        if((e = cudaGetLastError()) != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

// ---- the multi-scattering LM fit ------------------------------------------------------
//
// LevenbergMarquardtCurveFit (fitting.hh:457-678) with the central-difference
// Jacobian ParallelFDComputeResidualJacobianCenterPoint (fitting.hh:883-908,
// step (|p| + 1e-4) 1e-4) over the evaluator above, for a batch of texels.
// Each texel's LM state lives in MsTexel; the host runs the LM's iterations
// in lock step (every texel one iteration per round) as a sequence of
// launches: control (the step) -> residuals of the trial points -> control
// (gain, accept) -> Jacobians of the accepted points -> J^T J, J^T r ->
// control (damping).  The control stages append the texels that need the
// next evaluation to a list, whose length the host reads to size that launch.

namespace
{

constexpr int kMsEvals = 14;   // two evaluations per parameter

// The texel's parameters with parameter k moved by +-its finite-difference step.
__device__ __forceinline__ void fd_params(const MsTexel& s, int e, double* p)
{
#pragma unroll
    for(int i = 0; i < 7; ++i)
        p[i] = s.p[i];
    const int k = e >> 1;
    const double h = (double)1e-4f;
    const double step = (fabs(s.p[k]) + h) * h;
    p[k] = (e & 1) ? s.p[k] - step : s.p[k] + step;
}

} // namespace

// count: the list's length, or (dcount non-null) at most this many, *dcount
template <bool kTable>
__global__ void __launch_bounds__(ms_threads(kTable), ms_blocks(kTable)) ms_eval_kernel(MsFitArgs a, uint32_t mode, uint32_t count,
                                                             const uint32_t* dcount)
{
    extern __shared__ float4 walk_table[];
    if(dcount)
        count = min(count, *dcount);
    const uint64_t N = (uint64_t)a.L * a.L;
    const uint64_t per = mode == kMsEvalJacobian ? N * kMsEvals : N;
    if((uint64_t)blockIdx.x * blockDim.x >= (uint64_t)count * per)
        return;
    if constexpr(kTable)
        fill_walk_table(walk_table, (uint32_t)walk_draws(kFitWalks, a.bounces), 0u);
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= (uint64_t)count * per)
        return;
    const uint32_t t = a.list[i / per];
    const uint64_t r = i % per;
    const MsTexel& s = a.st[t];
    const uint32_t idx = (uint32_t)(mode == kMsEvalJacobian ? r / kMsEvals : r);
    const V3 wi = direction(a.geo, a.L, idx % a.L), wo = direction(a.geo, a.L, idx / a.L);
    if(mode == kMsEvalJacobian)
    {
        double p[7];
        fd_params(s, (int)(r % kMsEvals), p);
        a.fev[(uint64_t)t * N * kMsEvals + r] = -evaluator_ms<kTable>(p, wi, wo, a.bounces, walk_table);
        return;
    }
    const float f = evaluator_ms<kTable>(mode == kMsEvalTrial ? s.tmp : s.p, wi, wo, a.bounces, walk_table);
    a.res[(uint64_t)t * N + idx] = a.lum[t * a.lum_stride + idx] - f;
}

// Per listed texel: the sum of squared residuals (residual modes) or J^T J and
// J^T r (Jacobian mode), in FP64 with a fixed reduction order.
__global__ void __launch_bounds__(256) ms_reduce_kernel(MsFitArgs a, uint32_t mode, const uint32_t* dcount)
{
    constexpr int kV = 35;   // J^T r (7) + the upper triangle of J^T J (28)
    __shared__ double part[8][kV];
    if(dcount && blockIdx.x >= *dcount)
        return;
    const uint32_t t = a.list[blockIdx.x];
    MsTexel& s = a.st[t];
    const uint32_t N = a.L * a.L;
    const float* res = a.res + (uint64_t)t * N;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if(mode != kMsEvalJacobian)
    {
        double sum = 0.0;
        for(uint32_t idx = threadIdx.x; idx < N; idx += blockDim.x)
        {
            const float r = res[idx];
            sum += (double)(r * r);
        }
        for(int o = 16; o > 0; o >>= 1)
            sum += __shfl_down_sync(0xffffffffu, sum, o);
        if(lane == 0)
            part[warp][0] = sum;
        __syncthreads();
        if(threadIdx.x == 0)
        {
            double tot = 0.0;
            for(int w = 0; w < (int)(blockDim.x >> 5); ++w)
                tot += part[w][0];
            if(mode == kMsEvalTrial)
                s.trial = tot;
            else
                s.last = tot;
            ++s.residuals;
        }
        return;
    }
    double step2[7];
    const double h = (double)1e-4f;
#pragma unroll
    for(int k = 0; k < 7; ++k)
        step2[k] = 2.0f * ((fabs(s.p[k]) + h) * h);
    double v[kV];
#pragma unroll
    for(int k = 0; k < kV; ++k)
        v[k] = 0.0;
    const float* fev = a.fev + (uint64_t)t * N * kMsEvals;
    for(uint32_t idx = threadIdx.x; idx < N; idx += blockDim.x)
    {
        double J[7];
#pragma unroll
        for(int k = 0; k < 7; ++k)
            J[k] = (double)(fev[(uint64_t)idx * kMsEvals + 2 * k] - fev[(uint64_t)idx * kMsEvals + 2 * k + 1]) /
                   step2[k];
        const double r = (double)res[idx];
        int o = 7;
#pragma unroll
        for(int i = 0; i < 7; ++i)
        {
            v[i] += J[i] * r;
#pragma unroll
            for(int j = i; j < 7; ++j)
                v[o++] += J[i] * J[j];
        }
    }
#pragma unroll
    for(int k = 0; k < kV; ++k)
    {
        double x = v[k];
        for(int o = 16; o > 0; o >>= 1)
            x += __shfl_down_sync(0xffffffffu, x, o);
        if(lane == 0)
            part[warp][k] = x;
    }
    __syncthreads();
    if(threadIdx.x < kV)
    {
        double tot = 0.0;
        for(int w = 0; w < (int)(blockDim.x >> 5); ++w)
            tot += part[w][threadIdx.x];
        const int k = threadIdx.x;
        if(k < 7)
            s.grad[k] = tot;
        else
        {
            int o = 7;
            for(int i = 0; i < 7; ++i)
                for(int j = i; j < 7; ++j, ++o)
                    if(o == k)
                    {
                        s.hess[7 * i + j] = tot;
                        s.hess[7 * j + i] = tot;
                    }
        }
    }
    if(threadIdx.x == 0)
        ++s.jacobians;
}

namespace
{

// Inverse by Gauss-Jordan elimination with partial pivoting (FP64), as the
// oracle restates the reference's Eigen PartialPivLU inverse.
__device__ void invert7(const double* a, double* inv)
{
    double m[7][14];
    for(int i = 0; i < 7; ++i)
        for(int j = 0; j < 14; ++j)
            m[i][j] = j < 7 ? a[7 * i + j] : (j - 7 == i ? 1.0 : 0.0);
    for(int col = 0; col < 7; ++col)
    {
        int piv = col;
        for(int r = col + 1; r < 7; ++r)
            if(fabs(m[r][col]) > fabs(m[piv][col]))
                piv = r;
        if(piv != col)
            for(int j = 0; j < 14; ++j)
            {
                const double t = m[col][j];
                m[col][j] = m[piv][j];
                m[piv][j] = t;
            }
        const double d = m[col][col];
        for(int j = 0; j < 14; ++j)
            m[col][j] /= d;
        for(int r = 0; r < 7; ++r)
        {
            if(r == col)
                continue;
            const double f = m[r][col];
            for(int j = 0; j < 14; ++j)
                m[r][j] -= f * m[col][j];
        }
    }
    for(int i = 0; i < 7; ++i)
        for(int j = 0; j < 7; ++j)
            inv[7 * i + j] = m[i][7 + j];
}

// The step stage of one texel (phase kMsStep): the damped solve, the small-step
// and constraint tests, and the trial point (listed for its residuals).
__device__ void ms_step(const MsFitArgs& a, MsTexel& s, uint32_t t)
{
    const double N = (double)a.L * a.L;
    const double eps = a.eps;
    if(!(s.iter < a.max_iter && a.mse_target < s.last / N))
    {
        s.phase = kMsDone;
        return;
    }
    double damp[49], inv[49];
    for(int i = 0; i < 49; ++i)
        damp[i] = s.hess[i];
    for(int i = 0; i < 7; ++i)
        damp[8 * i] += s.damping;
    invert7(damp, inv);
    if(!isfinite(inv[0]))
    {
        s.damping *= s.mult;
        s.mult *= s.mult;
        ++s.iter;
        return;
    }
    double step_len = 0.0, pmag = 0.0;
    for(int i = 0; i < 7; ++i)
    {
        double v = 0.0;
        for(int j = 0; j < 7; ++j)
            v += inv[7 * i + j] * s.grad[j];
        s.step[i] = v;
        step_len += v * v;
        const double q = s.p[i] + eps;
        pmag += q * q;
    }
    if(sqrt(step_len) <= eps * (sqrt(pmag) + eps))
    {
        s.phase = kMsDone;
        return;
    }
    // AcceptStepConstraints (svbrdf-lsq-fitting-internal.hh:67-77)
    bool accept = true;
    for(int i = 0; i < 4; ++i)
        if(s.p[i] - s.step[i] < 0.0f)
            accept = false;
    if(!accept)
    {
        s.damping *= s.mult;
        s.mult *= s.mult;
        ++s.iter;
        return;
    }
    for(int i = 0; i < 7; ++i)
        s.tmp[i] = s.p[i] - s.step[i];
    s.phase = kMsTrial;
    a.list[atomicAdd(&a.counts[0], 1u)] = t;
}

} // namespace

// One thread per texel of the batch.  stage: kMsStageStart (after the first
// residual and Jacobian), kMsStageStep, kMsStageGain, kMsStageDamping.
__global__ void ms_control_kernel(MsFitArgs a, uint32_t stage)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if(t >= a.texels)
        return;
    MsTexel& s = a.st[t];
    const double N = (double)a.L * a.L;
    const double eps = a.eps;
    if(stage == kMsStageStart)
    {
        double d = 1.0;
        for(int i = 0; i < 7; ++i)
            d = fmax(d, s.hess[8 * i]);
        s.damping = d * (double)0.75f;
        s.mult = 2.0;
        s.phase = kMsStep;
        return;
    }
    if(stage == kMsStageStep)
    {
        if(s.phase == kMsStep)
            ms_step(a, s, t);
        if(s.phase != kMsDone)
            atomicAdd(&a.counts[2], 1u);
        return;
    }
    if(stage == kMsStageGain)
    {
        if(s.phase != kMsTrial)
            return;
        double pred = 0.0;
        for(int i = 0; i < 7; ++i)
            pred += s.step[i] * (s.step[i] * s.damping + s.grad[i]);
        pred *= 0.5f;
        const double gain = 0.5f * (s.last - s.trial) / pred;
        if(gain > 0.0f)
        {
            ++s.effective;
            for(int i = 0; i < 7; ++i)
                s.p[i] = s.tmp[i];
            s.last = s.trial;
            if(s.last / N <= a.mse_target)
            {
                s.phase = kMsDone;
                return;
            }
            s.gain = gain;
            s.phase = kMsJacobian;
            a.list[atomicAdd(&a.counts[1], 1u)] = t;
        }
        else
        {
            s.damping *= s.mult;
            s.mult *= s.mult;
            ++s.iter;
            s.phase = kMsStep;
        }
        return;
    }
    // kMsStageDamping: after the accepted point's J^T J and J^T r
    if(s.phase != kMsJacobian)
        return;
    double glen = 0.0;
    for(int i = 0; i < 7; ++i)
        glen += s.grad[i] * s.grad[i];
    if(glen <= eps * eps)
    {
        s.phase = kMsDone;
        return;
    }
    const double min_mul = 1.0f / 3.0f;
    s.damping *= fmax(min_mul, 1.0f - pow(2.0f * s.gain - 1.0f, 3.0f));
    s.mult = 2.0f;
    ++s.iter;
    s.phase = kMsStep;
}

// The batch's state from the initial guesses; every texel listed.
__global__ void ms_setup_kernel(MsFitArgs a, const float* init)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if(t >= a.texels)
        return;
    MsTexel& s = a.st[t];
    for(int i = 0; i < 7; ++i)
        s.p[i] = init[7 * (uint64_t)t + i];
    s.iter = s.effective = s.jacobians = s.residuals = 0;
    s.phase = kMsStep;
    a.list[t] = t;
}

// The fitted parameters, RMSE and statistics; a texel whose fit is not finite
// gets its initial guess back and SVF_TEXEL_NONFINITE.
__global__ void ms_finish_kernel(MsFitArgs a, const float* init, float* out, float* rmse, svf_texel_stats* stats)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if(t >= a.texels)
        return;
    const MsTexel& s = a.st[t];
    bool finite = true;
    float v[7];
    for(int i = 0; i < 7; ++i)
    {
        v[i] = (float)s.p[i];
        finite = finite && isfinite(v[i]);
    }
    const float r = (float)sqrt(s.last / ((double)a.L * a.L));
    finite = finite && isfinite(r);
    for(int i = 0; i < 7; ++i)
        out[7 * (uint64_t)t + i] = finite ? v[i] : init[7 * (uint64_t)t + i];
    if(rmse)
        rmse[t] = r;
    if(stats)
    {
        svf_texel_stats st;
        st.iterations = s.iter;
        st.effective = s.effective;
        st.jacobians = s.jacobians;
        st.residuals = s.residuals;
        st.status = (finite ? 0u : SVF_TEXEL_NONFINITE) | (s.iter >= a.max_iter ? SVF_TEXEL_MAX_ITER : 0u);
        stats[t] = st;
    }
}

cudaError_t launch_ms_setup(const MsFitArgs& a, const float* init, cudaStream_t stream)
{
    ms_setup_kernel<<<(unsigned)((a.texels + 127) / 128), 128, 0, stream>>>(a, init);
    return cudaGetLastError();
}

cudaError_t launch_ms_eval(const MsFitArgs& a, uint32_t mode, uint32_t count, const uint32_t* dcount,
                           cudaStream_t stream)
{
    if(count == 0)
        return cudaSuccess;
    const uint64_t N = (uint64_t)a.L * a.L;
    const uint64_t n = (uint64_t)count * N * (mode == kMsEvalJacobian ? kMsEvals : 1);
    const size_t smem = walk_table_bytes(kFitWalks, a.bounces);
    const unsigned threads = ms_threads(smem != 0);
    const uint64_t blocks = (n + threads - 1) / threads;
    if(blocks > 0x7fffffffull)
        return cudaErrorInvalidValue;
    cudaError_t e = cudaSuccess;
    if(smem == 0)
        ms_eval_kernel<false><<<(unsigned)blocks, threads, 0, stream>>>(a, mode, count, dcount);
    else
    {
        e = allow_smem(ms_eval_kernel<true>, smem);
        if(e != cudaSuccess)
            return e;
        ms_eval_kernel<true><<<(unsigned)blocks, threads, smem, stream>>>(a, mode, count, dcount);
    }
    e = cudaGetLastError();
    if(e != cudaSuccess)
        return e;
    ms_reduce_kernel<<<count, 256, 0, stream>>>(a, mode, dcount);
    return cudaGetLastError();
}

cudaError_t launch_ms_control(const MsFitArgs& a, uint32_t stage, cudaStream_t stream)
{
    ms_control_kernel<<<(unsigned)((a.texels + 127) / 128), 128, 0, stream>>>(a, stage);
    return cudaGetLastError();
}

cudaError_t launch_ms_finish(const MsFitArgs& a, const float* init, float* out, float* rmse, svf_texel_stats* stats,
                             cudaStream_t stream)
{
    ms_finish_kernel<<<(unsigned)((a.texels + 127) / 128), 128, 0, stream>>>(a, init, out, rmse, stats);
    return cudaGetLastError();
}

} // namespace svf
