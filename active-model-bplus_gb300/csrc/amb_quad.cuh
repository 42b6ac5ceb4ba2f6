// Four adjacent columns of one row as two packed FP32 pairs, and the canonical operations on them
// (amb_canon.cuh): a packed instruction rounds each half as the scalar one, so the bits are the same
// in half the issue slots.
#pragma once

#include "amb_canon.cuh"

namespace amb
{
    // Canon's constants as duplicated pairs, which packed operations read from the constant bank,
    // and the Philox round keys of the seed.
    struct QuadStencil
    {
        float2 lA, lB, lC, lD, gxa, gxb, gya, gyb;
        float2 ny8[4], nx8[4], py8[4], px8[4];
        float2 ndy, jx1, jx3, dyInv, tx1, tx3, dt, ndt, p1, p3;
    };
    struct QuadModel
    {
        float2 a, b, c, nkappa, lambda, zeta, mag;
        uint32_t rk0[10], rk1[10];
    };
    struct QuadCoef
    {
        QuadStencil s;
        QuadModel m;
        __host__ explicit QuadCoef(const StepParams& p)
        {
            const Canon<float> k(p);
            const auto d = [](float v) { return make_float2(v, v); };
            s.lA = d(k.lA); s.lB = d(k.lB); s.lC = d(k.lC); s.lD = d(k.lD);
            s.gxa = d(k.gxa); s.gxb = d(k.gxb); s.gya = d(k.gya); s.gyb = d(k.gyb);
            for (int j = 0; j < 4; ++j)
            {
                s.ny8[j] = d(k.ny8[j]); s.nx8[j] = d(k.nx8[j]);
                s.py8[j] = d(k.py8[j]); s.px8[j] = d(k.px8[j]);
            }
            s.ndy = d(k.ndy); s.jx1 = d(k.jx1); s.jx3 = d(k.jx3);
            s.dyInv = d(k.dyInv); s.tx1 = d(k.tx1); s.tx3 = d(k.tx3);
            s.dt = d(k.dt); s.ndt = d(k.ndt); s.p1 = d(k.p1); s.p3 = d(k.p3);
            m.a = d(k.a); m.b = d(k.b); m.c = d(k.c);
            m.nkappa = d(k.nkappa); m.lambda = d(k.lambda); m.zeta = d(k.zeta); m.mag = d(k.mag);
            for (int r = 0; r < 10; ++r)
            {
                m.rk0[r] = uint32_t(p.seed) + uint32_t(r) * 0x9E3779B9u;
                m.rk1[r] = uint32_t(p.seed >> 32) + uint32_t(r) * 0xBB67AE85u;
            }
        }
    };
    // The two parts from different places (one stencil for many models).
    struct QuadCoefParts
    {
        const QuadStencil& s;
        const QuadModel& m;
    };

    struct Quad
    {
        float2 a, b;
    };

    __device__ __forceinline__ float2 sub2(float2 x, float2 y) { return __fadd2_rn(x, make_float2(-y.x, -y.y)); }
    __device__ __forceinline__ Quad operator+(Quad x, Quad y) { return {__fadd2_rn(x.a, y.a), __fadd2_rn(x.b, y.b)}; }
    __device__ __forceinline__ Quad operator-(Quad x, Quad y) { return {sub2(x.a, y.a), sub2(x.b, y.b)}; }
    __device__ __forceinline__ Quad operator*(Quad x, Quad y) { return {__fmul2_rn(x.a, y.a), __fmul2_rn(x.b, y.b)}; }
    __device__ __forceinline__ Quad operator*(float2 c, Quad x) { return {__fmul2_rn(c, x.a), __fmul2_rn(c, x.b)}; }
    __device__ __forceinline__ Quad fma4(float2 c, Quad x, Quad y) { return {__ffma2_rn(c, x.a, y.a), __ffma2_rn(c, x.b, y.b)}; }
    __device__ __forceinline__ Quad fma4(float2 c, Quad x, float2 y) { return {__ffma2_rn(c, x.a, y), __ffma2_rn(c, x.b, y)}; }
    __device__ __forceinline__ Quad fma4(Quad x, Quad y, Quad z) { return {__ffma2_rn(x.a, y.a, z.a), __ffma2_rn(x.b, y.b, z.b)}; }
    __device__ __forceinline__ Quad fma4(Quad x, Quad y, float2 z) { return {__ffma2_rn(x.a, y.a, z), __ffma2_rn(x.b, y.b, z)}; }
    __device__ __forceinline__ Quad quad(float4 v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }
    __device__ __forceinline__ float4 vec(Quad v) { return make_float4(v.a.x, v.a.y, v.b.x, v.b.y); }
    __device__ __forceinline__ Quad zero_quad() { return {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
    __device__ __forceinline__ Quad load_quad(const float* p) { return quad(*reinterpret_cast<const float4*>(p)); }
    __device__ __forceinline__ void store_quad(float* p, Quad v) { *reinterpret_cast<float4*>(p) = vec(v); }

    // left + right and right - left neighbours of four columns, l to their left and r to their right
    __device__ __forceinline__ Quad nsum(float l, Quad v, float r)
    {
        return {make_float2(__fadd_rn(l, v.a.y), __fadd_rn(v.a.x, v.b.x)),
                make_float2(__fadd_rn(v.a.y, v.b.y), __fadd_rn(v.b.x, r))};
    }
    __device__ __forceinline__ Quad ndiff(float l, Quad v, float r)
    {
        return {make_float2(__fsub_rn(v.a.y, l), __fsub_rn(v.b.x, v.a.x)),
                make_float2(__fsub_rn(v.b.y, v.a.y), __fsub_rn(r, v.b.x))};
    }

    // sum_j c_j (g[+j] - g[-j]) along x at the columns of c, from the quads l and r beside it: the even
    // offsets are aligned pairs, the odd ones are formed as scalars
    __device__ __forceinline__ Quad d8x(const float2 (&k)[4], Quad l, Quad c, Quad r)
    {
        const Quad d1{make_float2(__fsub_rn(c.a.y, l.b.y), __fsub_rn(c.b.x, c.a.x)),
                      make_float2(__fsub_rn(c.b.y, c.a.y), __fsub_rn(r.a.x, c.b.x))};
        const Quad d2{sub2(c.b, l.b), sub2(r.a, c.a)};
        const Quad d3{make_float2(__fsub_rn(c.b.y, l.a.y), __fsub_rn(r.a.x, l.b.x)),
                      make_float2(__fsub_rn(r.a.y, l.b.y), __fsub_rn(r.b.x, c.a.x))};
        const Quad d4{sub2(r.a, l.a), sub2(r.b, l.b)};
        Quad s = k[0] * d1;
        s = fma4(k[1], d2, s);
        s = fma4(k[2], d3, s);
        return fma4(k[3], d4, s);
    }
}
