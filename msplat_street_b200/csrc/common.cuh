// Shared device helpers for the msplat B200 kernels.
//
// Parity contract. The splatting kernels reproduce the reference backend's float32
// results (core/cpu/msplat_cpu.cpp, itself a port of core/metal/msplat_metal.metal)
// bit for bit wherever an integer decision depends on them: tile rectangles, radii,
// depth keys and the alpha / transmittance cut-offs. To that end
//  * the translation units that compute them are compiled with -fmad=false, so every
//    a*b+c stays two rounded operations, in the reference's order;
//  * exponentials are evaluated in double and rounded once to float: exp_ref(), which
//    agrees with a correctly rounded expf except in rare near-halfway cases, and the
//    table methods below, which are correctly rounded;
//  * division and square root are IEEE (nvcc's default -prec-div / -prec-sqrt).
// Matrices are column-major (c[col] is a column) because the reference's helper
// types follow MSL conventions (core/cpu/cpu_math.hpp:1-4).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace msplat {

constexpr int TILE = 16;            // core/cpu/msplat_cpu.cpp:27
constexpr int TILE_PIX = TILE * TILE;

// Real SH basis constants (core/cpu/msplat_cpu.cpp:29-38).
constexpr float SH_C0 = 0.28209479177387814f;
constexpr float SH_C1 = 0.4886025119029199f;
constexpr float SH_C2_0 = 1.0925484305920792f, SH_C2_1 = -1.0925484305920792f, SH_C2_2 = 0.31539156525252005f,
                SH_C2_3 = -1.0925484305920792f, SH_C2_4 = 0.5462742152960396f;
constexpr float SH_C3_0 = -0.5900435899266435f, SH_C3_1 = 2.890611442640554f, SH_C3_2 = -0.4570457994644658f,
                SH_C3_3 = 0.3731763325901154f, SH_C3_4 = -0.4570457994644658f, SH_C3_5 = 1.445305721320277f,
                SH_C3_6 = -0.5900435899266435f;
constexpr float SH_C4_0 = 2.5033429417967046f, SH_C4_1 = -1.7701307697799304f, SH_C4_2 = 0.9461746957575601f,
                SH_C4_3 = -0.6690465435572892f, SH_C4_4 = 0.10578554691520431f, SH_C4_5 = -0.6690465435572892f,
                SH_C4_6 = 0.47308734787878004f, SH_C4_7 = -1.7701307697799304f, SH_C4_8 = 0.6258357354491761f;

__host__ __device__ inline uint32_t num_sh_bases(uint32_t degree) {
    return degree == 0 ? 1 : degree == 1 ? 4 : degree == 2 ? 9 : degree == 3 ? 16 : 25;
}

// exp in double, rounded once to float
__device__ __forceinline__ float exp_ref(float x) { return (float)exp((double)x); }

// The rasterizers' exponential, exp(x) rounded once to float for x = -sigma in
// [-5.55, 0]: Tang's table-driven method (P. T. P. Tang, ACM TOMS 15(2), 1989) in
// double precision. x = (128 m + j) ln2 / 128 + r with |r| <= ln2 / 256, so
// exp(x) = 2^m 2^(j/128) exp(r); exp(r) is a polynomial of degree 4 (1 + r s(r), s the
// cubic through (exp(r) - 1) / r at the Chebyshev nodes of the interval: off by at most
// 1.6e-16), and 2^m 2^(j/128) comes from a table over the range that the block fills
// once (exp_span_init_a, a barrier, exp_span_init_b). The reduction is one fused step:
// k times the rounding of ln2 / 128 stays below 4.5e-16 for |k| <= 1026. The double
// result is within about 1e-15 of exp(x); no float of [-5.55, 0] has its exponential that
// close to a float rounding boundary: evaluated for all of them, the float is the
// correctly rounded one, as that of a degree 5 with two reduction steps over 64 entries
// is (two operations more of fifteen). A change to any constant here needs that check.
constexpr double EXP_INV_LN2_T = 0x1.71547652b82fep+7;    // 128 / ln 2
constexpr double EXP_LN2_T = 0x1.62e42fefa39efp-8;     // ln 2 / 128
constexpr double EXP_LN2_T_HI = 0x1.62e42fefa2000p-8;  // its upper 40 bits: k * HI is exact
constexpr double EXP_LN2_T_LO = 0x1.9ef35793c7673p-48;  // ln 2 / 128 - HI
constexpr int EXP_TABLE = 128, EXP_BITS = 7;
constexpr int EXP_SPAN = 1040;  // covers k down to -1039 (x >= -5.62)

// exp(r), |r| <= ln2 / 256
__device__ __forceinline__ double exp_poly(double r) {
    double p = fma(r, 0x1.55555acd08c2ep-5, 0x1.55555d88e27efp-3);
    p = fma(p, r, 0x1.fffffffffff58p-2);
    p = fma(p, r, 0x1.ffffffffffe08p-1);
    return fma(p, r, 1.0);
}

// k = round(x 128 / ln 2): adding 1.5 * 2^52 leaves the rounded integer in the low word
// of the sum (exact for |k| < 2^31)
__device__ __forceinline__ int exp_index(double x, double &k) {
    const double shifted = fma(x, EXP_INV_LN2_T, 0x1.8p52);
    k = shifted - 0x1.8p52;
    return __double2loint(shifted);
}

// v 2^m, exactly, where v and the result are normal: the exponent field moved
__device__ __forceinline__ double exp_scale(double v, int m) {
    return __hiloint2double(__double2hiint(v) + m * (1 << 20), __double2loint(v));
}

// 2^(j/128), rounded to double
static __device__ const double EXP2_TABLE[EXP_TABLE] = {
    0x1.0000000000000p+0, 0x1.0163da9fb3335p+0, 0x1.02c9a3e778061p+0, 0x1.04315e86e7f85p+0,
    0x1.059b0d3158574p+0, 0x1.0706b29ddf6dep+0, 0x1.0874518759bc8p+0, 0x1.09e3ecac6f383p+0,
    0x1.0b5586cf9890fp+0, 0x1.0cc922b7247f7p+0, 0x1.0e3ec32d3d1a2p+0, 0x1.0fb66affed31bp+0,
    0x1.11301d0125b51p+0, 0x1.12abdc06c31ccp+0, 0x1.1429aaea92de0p+0, 0x1.15a98c8a58e51p+0,
    0x1.172b83c7d517bp+0, 0x1.18af9388c8deap+0, 0x1.1a35beb6fcb75p+0, 0x1.1bbe084045cd4p+0,
    0x1.1d4873168b9aap+0, 0x1.1ed5022fcd91dp+0, 0x1.2063b88628cd6p+0, 0x1.21f49917ddc96p+0,
    0x1.2387a6e756238p+0, 0x1.251ce4fb2a63fp+0, 0x1.26b4565e27cddp+0, 0x1.284dfe1f56381p+0,
    0x1.29e9df51fdee1p+0, 0x1.2b87fd0dad990p+0, 0x1.2d285a6e4030bp+0, 0x1.2ecafa93e2f56p+0,
    0x1.306fe0a31b715p+0, 0x1.32170fc4cd831p+0, 0x1.33c08b26416ffp+0, 0x1.356c55f929ff1p+0,
    0x1.371a7373aa9cbp+0, 0x1.38cae6d05d866p+0, 0x1.3a7db34e59ff7p+0, 0x1.3c32dc313a8e5p+0,
    0x1.3dea64c123422p+0, 0x1.3fa4504ac801cp+0, 0x1.4160a21f72e2ap+0, 0x1.431f5d950a897p+0,
    0x1.44e086061892dp+0, 0x1.46a41ed1d0057p+0, 0x1.486a2b5c13cd0p+0, 0x1.4a32af0d7d3dep+0,
    0x1.4bfdad5362a27p+0, 0x1.4dcb299fddd0dp+0, 0x1.4f9b2769d2ca7p+0, 0x1.516daa2cf6642p+0,
    0x1.5342b569d4f82p+0, 0x1.551a4ca5d920fp+0, 0x1.56f4736b527dap+0, 0x1.58d12d497c7fdp+0,
    0x1.5ab07dd485429p+0, 0x1.5c9268a5946b7p+0, 0x1.5e76f15ad2148p+0, 0x1.605e1b976dc09p+0,
    0x1.6247eb03a5585p+0, 0x1.6434634ccc320p+0, 0x1.6623882552225p+0, 0x1.68155d44ca973p+0,
    0x1.6a09e667f3bcdp+0, 0x1.6c012750bdabfp+0, 0x1.6dfb23c651a2fp+0, 0x1.6ff7df9519484p+0,
    0x1.71f75e8ec5f74p+0, 0x1.73f9a48a58174p+0, 0x1.75feb564267c9p+0, 0x1.780694fde5d3fp+0,
    0x1.7a11473eb0187p+0, 0x1.7c1ed0130c132p+0, 0x1.7e2f336cf4e62p+0, 0x1.80427543e1a12p+0,
    0x1.82589994cce13p+0, 0x1.8471a4623c7adp+0, 0x1.868d99b4492edp+0, 0x1.88ac7d98a6699p+0,
    0x1.8ace5422aa0dbp+0, 0x1.8cf3216b5448cp+0, 0x1.8f1ae99157736p+0, 0x1.9145b0b91ffc6p+0,
    0x1.93737b0cdc5e5p+0, 0x1.95a44cbc8520fp+0, 0x1.97d829fde4e50p+0, 0x1.9a0f170ca07bap+0,
    0x1.9c49182a3f090p+0, 0x1.9e86319e32323p+0, 0x1.a0c667b5de565p+0, 0x1.a309bec4a2d33p+0,
    0x1.a5503b23e255dp+0, 0x1.a799e1330b358p+0, 0x1.a9e6b5579fdbfp+0, 0x1.ac36bbfd3f37ap+0,
    0x1.ae89f995ad3adp+0, 0x1.b0e07298db666p+0, 0x1.b33a2b84f15fbp+0, 0x1.b59728de5593ap+0,
    0x1.b7f76f2fb5e47p+0, 0x1.ba5b030a1064ap+0, 0x1.bcc1e904bc1d2p+0, 0x1.bf2c25bd71e09p+0,
    0x1.c199bdd85529cp+0, 0x1.c40ab5fffd07ap+0, 0x1.c67f12e57d14bp+0, 0x1.c8f6d9406e7b5p+0,
    0x1.cb720dcef9069p+0, 0x1.cdf0b555dc3fap+0, 0x1.d072d4a07897cp+0, 0x1.d2f87080d89f2p+0,
    0x1.d5818dcfba487p+0, 0x1.d80e316c98398p+0, 0x1.da9e603db3285p+0, 0x1.dd321f301b460p+0,
    0x1.dfc97337b9b5fp+0, 0x1.e264614f5a129p+0, 0x1.e502ee78b3ff6p+0, 0x1.e7a51fbc74c83p+0,
    0x1.ea4afa2a490dap+0, 0x1.ecf482d8e67f1p+0, 0x1.efa1bee615a27p+0, 0x1.f252b376bba97p+0,
    0x1.f50765b6e4540p+0, 0x1.f7bfdad9cbe14p+0, 0x1.fa7c1819e90d8p+0, 0x1.fd3c22b8f71f1p+0,
};

// Every thread of the block calls each; the span is ready after the barrier that follows
// init_b. t: EXP_TABLE doubles of scratch, read by init_b.
__device__ __forceinline__ void exp_span_init_a(double *t) {
    for (int j = threadIdx.x; j < EXP_TABLE; j += blockDim.x) t[j] = EXP2_TABLE[j];
}
__device__ __forceinline__ void exp_span_init_b(double *span, const double *t) {
    for (int i = threadIdx.x; i < EXP_SPAN; i += blockDim.x) span[i] = exp_scale(t[-i & (EXP_TABLE - 1)], -i >> EXP_BITS);
}

__device__ __forceinline__ float exp_span(float xf, const double *span) {
    const double x = (double)xf;
    double k;
    const int ki = exp_index(x, k);
    const double r = fma(-k, EXP_LN2_T, x);
    return (float)(span[min((unsigned)-ki, (unsigned)EXP_SPAN - 1u)] * exp_poly(r));
}

// The same double without a table, for the few pairs a pass evaluates so (the backward's
// near the cut-offs, the pair counter): the span's entry computed on the spot. Inlined:
// as a call it cost the backward 1.5 % (an early street view 434 -> 428 us, 200 k Gaussians
// at 1024 x 768 258 -> 252). FAR: for x down to -700, with the reduction in two steps.
template <bool FAR = false>
__device__ __forceinline__ float exp_once(float xf) {
    const double x = (double)xf;
    double k;
    const int ki = exp_index(x, k);
    const double r = FAR ? fma(-k, EXP_LN2_T_LO, fma(-k, EXP_LN2_T_HI, x)) : fma(-k, EXP_LN2_T, x);
    return (float)(exp_scale(EXP2_TABLE[ki & (EXP_TABLE - 1)], ki >> EXP_BITS) * exp_poly(r));
}

// exp(x) in double, rounded once to float, for any x: the same method with the power of
// two applied to the exponent and the reduction in two steps (within about 5e-16 of
// exp(x)). Evaluated for every float: the correctly rounded result, 0 and infinity
// included. t: the EXP_TABLE entries 2^(j/128) of exp_span_init_a.
__device__ __forceinline__ float exp_wide(float xf, const double *t) {
    if (xf != xf) return xf;
    const double x = (double)fminf(fmaxf(xf, -110.f), 100.f);  // 0 and infinity beyond, as floats
    double k;
    const int ki = exp_index(x, k);
    const double r = fma(-k, EXP_LN2_T_LO, fma(-k, EXP_LN2_T_HI, x));
    return (float)exp_scale(t[ki & (EXP_TABLE - 1)] * exp_poly(r), ki >> EXP_BITS);
}

// Two float32 values in one 64-bit register pair, for sm_100's packed FP32
// instructions (PTX add / mul / fma .rn.f32x2): one instruction issues two IEEE
// single-precision operations, each rounded exactly as its scalar form, so packing
// changes no result -- only the instruction count of an issue-bound kernel.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

struct V2 { float x, y; };
struct V3 { float x, y, z; };
struct Q4 { float x, y, z, w; };  // quaternion stored (w, x, y, z) lands in x, y, z, w

__device__ __forceinline__ V3 v3(float x, float y, float z) { return V3{x, y, z}; }
__device__ __forceinline__ V3 add(V3 a, V3 b) { return V3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 sub(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 scl(V3 a, float s) { return V3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ V3 scl(float s, V3 a) { return V3{s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ float dot3(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 ld3(const float *p, int64_t i) { return V3{p[3 * i], p[3 * i + 1], p[3 * i + 2]}; }
__device__ __forceinline__ void st3(float *p, int64_t i, V3 v) {
    p[3 * i] = v.x;
    p[3 * i + 1] = v.y;
    p[3 * i + 2] = v.z;
}
__device__ __forceinline__ float clamp01(float v) { return fminf(fmaxf(v, 0.f), 1.f); }
__device__ __forceinline__ V3 unit(V3 a) { return scl(a, 1.f / sqrtf(dot3(a, a))); }

struct M3 {
    V3 c[3];
};
__device__ __forceinline__ M3 m3(float a0, float a1, float a2, float b0, float b1, float b2, float d0, float d1,
                                 float d2) {
    M3 m;
    m.c[0] = V3{a0, a1, a2};
    m.c[1] = V3{b0, b1, b2};
    m.c[2] = V3{d0, d1, d2};
    return m;
}
__device__ __forceinline__ float el(const V3 &v, int r) { return r == 0 ? v.x : (r == 1 ? v.y : v.z); }
// Column-major product R[j][i] = sum_k A[k][i] * B[j][k], k in order 0,1,2
__device__ __forceinline__ M3 mul(const M3 &A, const M3 &B) {
    M3 R;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        float r0 = A.c[0].x * el(B.c[j], 0) + A.c[1].x * el(B.c[j], 1) + A.c[2].x * el(B.c[j], 2);
        float r1 = A.c[0].y * el(B.c[j], 0) + A.c[1].y * el(B.c[j], 1) + A.c[2].y * el(B.c[j], 2);
        float r2 = A.c[0].z * el(B.c[j], 0) + A.c[1].z * el(B.c[j], 1) + A.c[2].z * el(B.c[j], 2);
        R.c[j] = V3{r0, r1, r2};
    }
    return R;
}
__device__ __forceinline__ M3 tr(const M3 &A) {
    return m3(A.c[0].x, A.c[1].x, A.c[2].x, A.c[0].y, A.c[1].y, A.c[2].y, A.c[0].z, A.c[1].z, A.c[2].z);
}
__device__ __forceinline__ M3 plus(const M3 &A, const M3 &B) {
    M3 R;
    R.c[0] = add(A.c[0], B.c[0]);
    R.c[1] = add(A.c[1], B.c[1]);
    R.c[2] = add(A.c[2], B.c[2]);
    return R;
}
__device__ __forceinline__ M3 smul(float s, const M3 &A) {
    M3 R;
    R.c[0] = scl(A.c[0], s);
    R.c[1] = scl(A.c[1], s);
    R.c[2] = scl(A.c[2], s);
    return R;
}

// Rotation from the (w,x,y,z) quaternion, normalised (core/cpu/msplat_cpu.cpp:77-84)
__device__ __forceinline__ M3 rotmat(Q4 q) {
    float s = 1.f / sqrtf(q.w * q.w + q.x * q.x + q.y * q.y + q.z * q.z);
    float w = q.x * s, x = q.y * s, y = q.z * s, z = q.w * s;
    return m3(1.f - 2.f * (y * y + z * z), 2.f * (x * y + w * z), 2.f * (x * z - w * y), 2.f * (x * y - w * z),
              1.f - 2.f * (x * x + z * z), 2.f * (y * z + w * x), 2.f * (x * z + w * y), 2.f * (y * z - w * x),
              1.f - 2.f * (x * x + y * y));
}

__device__ __forceinline__ M3 diag_scale(V3 s, float g) {
    M3 S = m3(1.f, 0.f, 0.f, 0.f, 1.f, 0.f, 0.f, 0.f, 1.f);
    S.c[0].x = g * s.x;
    S.c[1].y = g * s.y;
    S.c[2].z = g * s.z;
    return S;
}

// 3D covariance R S S^T R^T, upper triangle (core/cpu/msplat_cpu.cpp:94-100)
__device__ __forceinline__ void cov3d_of(V3 s, float g, Q4 q, float *cov) {
    M3 M = mul(rotmat(q), diag_scale(s, g));
    M3 t = mul(M, tr(M));
    cov[0] = t.c[0].x;
    cov[1] = t.c[0].y;
    cov[2] = t.c[0].z;
    cov[3] = t.c[1].y;
    cov[4] = t.c[1].z;
    cov[5] = t.c[2].z;
}

// Two floats as a half2 (low half first), each rounded toward +infinity (values
// beyond the half range become +inf, or -65504 from below).
__device__ __forceinline__ uint32_t pack_half2_up(float lo, float hi) {
    const __half l = __float2half_ru(lo), h = __float2half_ru(hi);
    return (uint32_t)__half_as_ushort(l) | ((uint32_t)__half_as_ushort(h) << 16);
}
__device__ __forceinline__ float2 unpack_half2(uint32_t v) {
    return make_float2(__half2float(__ushort_as_half((unsigned short)(v & 0xffffu))),
                       __half2float(__ushort_as_half((unsigned short)(v >> 16))));
}

// One splat record per Gaussian, read by the rasterizer: centre, conic, sigmoid
// opacity, raw SH colour, depth, and the extents of the region where it can be
// composited (alpha >= 1/255): the half-widths of its box and its half-extents along
// the diagonals x + y and x - y, each a half-precision float rounded up (a region
// never shrinks; -inf marks a splat that never reaches 1/255, +inf an extent with no
// bound). 48 bytes, loaded as three float4.
struct __align__(16) Splat {
    float x, y, cx, cy;   // pixel centre, conic (a, b)
    float cz, op, r, g;   // conic c, sigmoid(opacity), raw colour r g
    float b, depth;       // raw colour b, view depth
    uint32_t box, diag;   // half2 (ex, ey) and half2 (hp, hm)
};
constexpr int SPLAT_FLOATS = sizeof(Splat) / sizeof(float);

// Pixels of a 16x16 tile owned by one warp: an 8x4 block (warp w covers columns
// 8 * (w % 2) .. +7 and rows 4 * (w / 2) .. +3), compact so that per-warp culling
// against a Gaussian's box skips as much as possible.
__device__ __forceinline__ void tile_pixel(int t, int &lx, int &ly) {
    const int w = t >> 5, l = t & 31;
    lx = ((w & 1) << 3) + (l & 7);
    ly = ((w >> 1) << 2) + (l >> 3);
}
// The thread index tile_pixel maps to pixel (lx, ly) of the tile (its inverse).
__device__ __forceinline__ int tile_index(int lx, int ly) {
    return ((((ly >> 2) << 1) + (lx >> 3)) << 5) + ((ly & 3) << 3) + (lx & 7);
}

// Counter-based RNG: PCG hash + Box-Muller (core/cpu/msplat_cpu.cpp:304-323)
__host__ __device__ __forceinline__ uint32_t pcg_hash(uint32_t v) {
    uint32_t s = v * 747796405u + 2891336453u;
    uint32_t w = ((s >> ((s >> 28u) + 4u)) ^ s) * 277803737u;
    return (w >> 22u) ^ w;
}
__host__ __device__ __forceinline__ float rand_unif(uint32_t seed, uint32_t ctr) {
    uint32_t h = pcg_hash(seed ^ pcg_hash(ctr));
    return ((float)(h >> 8) + 0.5f) * (1.0f / 16777216.0f);
}

// Adam with precomputed step_size = lr / bc1 (core/cpu/msplat_cpu.cpp:293-300)
__device__ __forceinline__ void adam_step(float &p, float &m1, float &m2, float g, float ss, float b1, float b2,
                                          float bc2, float eps) {
    float m = b1 * m1 + (1.0f - b1) * g;
    float v = b2 * m2 + (1.0f - b2) * g * g;
    p -= ss * m / (sqrtf(v) / bc2 + eps);
    m1 = m;
    m2 = v;
}

}  // namespace msplat
