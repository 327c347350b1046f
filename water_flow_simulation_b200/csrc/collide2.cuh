// collide2.cuh -- the force-free collision on two cells at a time, in packed float32.
// Included inside the anonymous namespace of lbm_kernels.cu, after fused_common.cuh.
#pragma once

// Two cells at a time: packed float32 operations (FFMA2 and kin), each half rounded as the scalar
// operation is.
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, both(-1.0f), a); }
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(1.0f / a.x, 1.0f / a.y); }
__device__ __forceinline__ float2 sqrt2(float2 a) { return make_float2(sqrtf(a.x), sqrtf(a.y)); }

// collide() without body force on two cells at once, bit for bit.  DEV: on deviations, `d` holding
// raw storage values (f_i - w_i) * scale on entry and on exit; else populations (scale 1).  The
// deviation form is the same update: with dr = rho - 1 and S = sum c c (f - w) (so that
// sum c c f = I/3 + S), the non-equilibrium stress is Pi = S - rho u u - dr I/3, and the
// post-collision deviation is w_i [ (A0 - 1) + c.B + c.C.c ].  UX2: see collide().
// Why packed: the plain kernels are bound by memory and by how many loads their warps keep in
// flight; the scalar collision took about 43 % of the issue slots of the 16-bit one.  Packed, the
// arithmetic takes half the slots and, done a pair at a time, few enough registers for 20 warps
// per SM instead of 12.
template <bool DEV, bool UX2>
__device__ __forceinline__ void collide2(float2 (&d)[Q], float scale, float inv_scale, float tau0, float csmag2,
                                         float2& r, float2& ux, float2& uy, float2& uz)
{
    const float2 s1 = add2(d[1], d[2]), d1 = sub2(d[1], d[2]);
    const float2 s3 = add2(d[3], d[4]), d3 = sub2(d[3], d[4]);
    const float2 s5 = add2(d[5], d[6]), d5 = sub2(d[5], d[6]);
    const float2 s7 = add2(d[7], d[8]), d7 = sub2(d[7], d[8]);
    const float2 s9 = add2(d[9], d[10]), d9 = sub2(d[9], d[10]);
    const float2 s11 = add2(d[11], d[12]), d11 = sub2(d[11], d[12]);
    const float2 s13 = add2(d[13], d[14]), d13 = sub2(d[13], d[14]);
    const float2 s15 = add2(d[15], d[16]), d15 = sub2(d[15], d[16]);
    const float2 s17 = add2(d[17], d[18]), d17 = sub2(d[17], d[18]);
    const float2 sum = add2(add2(add2(d[0], add2(add2(s1, s3), s5)), add2(add2(s7, s9), s11)),
                            add2(add2(s13, s15), s17));
    // the scale is a power of two: products with it are exact, wherever they are taken
    const float2 dr = DEV ? mul2(sum, both(inv_scale)) : sum;            // rho - 1, or rho
    r = DEV ? add2(both(1.0f), dr) : sum;
    const float2 ir = rcp2(r), irs = DEV ? mul2(ir, both(inv_scale)) : ir;
    ux = mul2(add2(add2(add2(add2(d1, d7), d9), d11), d13), irs);
    uy = mul2(add2(add2(sub2(add2(d3, d7), d9), d15), d17), irs);
    uz = mul2(sub2(add2(sub2(add2(d5, d11), d13), d15), d17), irs);
    const float2 rx = mul2(r, ux), ry = mul2(r, uy), rz = mul2(r, uz);
    const float2 rxx = mul2(rx, ux), ryy = mul2(ry, uy), rzz = mul2(rz, uz);
    const float2 rxy = mul2(rx, uy), rxz = mul2(rx, uz), ryz = mul2(ry, uz);
    // n.. = -Pi..: the negated stress and 1/tau - 1 carry no sign changes into the products below
    const float2 nis = both(DEV ? -inv_scale : -1.0f), third = both(1.0f / 3.0f);
    const float2 nxx = fma2(third, dr, fma2(add2(add2(add2(add2(s1, s7), s9), s11), s13), nis, rxx));
    const float2 nyy = fma2(third, dr, fma2(add2(add2(add2(add2(s3, s7), s9), s15), s17), nis, ryy));
    const float2 nzz = fma2(third, dr, fma2(add2(add2(add2(add2(s5, s11), s13), s15), s17), nis, rzz));
    const float2 nxy = fma2(sub2(s7, s9), nis, rxy), nxz = fma2(sub2(s11, s13), nis, rxz),
                 nyz = fma2(sub2(s15, s17), nis, ryz);

    const float2 qd = fma2(nzz, nzz, fma2(nxx, nxx, mul2(nyy, nyy)));
    const float2 qo = fma2(nyz, nyz, fma2(nxy, nxy, mul2(nxz, nxz)));
    const float2 qn = sqrt2(fma2(both(2.0f), qo, qd));
    const float tau0sq = mul_rn(tau0, tau0), smag = mul_rn(18.0f * 1.41421356f, csmag2);
    const float2 tau = mul2(both(0.5f), add2(both(tau0), sqrt2(fma2(mul2(both(smag), qn), ir, both(tau0sq)))));
    const float2 nk = add2(rcp2(tau), both(-1.0f));                       // 1/tau - 1

    const float2 usq = fma2(uz, uz, UX2 ? fma2(uy, uy, mul2(ux, ux)) : fma2(ux, ux, mul2(uy, uy)));
    const float2 A0 = fma2(both(-1.5f), fma2(nk, add2(add2(nxx, nyy), nzz), mul2(r, usq)), dr);
    const float2 r3 = mul2(both(3.0f), r), n3 = mul2(both(-3.0f), r);
    const float2 Bx = mul2(r3, ux), By = mul2(r3, uy), Bz = mul2(r3, uz);
    const float2 Cxx = fma2(nk, nxx, rxx), Cyy = fma2(nk, nyy, ryy), Czz = fma2(nk, nzz, rzz);
    const float2 Cxy = fma2(nk, nxy, rxy), Cxz = fma2(nk, nxz, rxz), Cyz = fma2(nk, nyz, ryz);

    // w_i (A0 + c.B + c.C.c), C's factors 4.5 (diagonal) and 9 (off-diagonal) applied here; c.B is
    // rounded before it is added on populations, fused in ux (and along the axes) on deviations
    const float2 w0 = both(DEV ? wgt(0) * scale : wgt(0)), w1 = both(DEV ? wgt(1) * scale : wgt(1)),
                 w2 = both(DEV ? wgt(7) * scale : wgt(7));
    const float2 h = both(4.5f), p9 = both(9.0f), n9 = both(-9.0f);
    d[0] = mul2(w0, A0);
    const float2 bx = fma2(h, Cxx, A0), by = fma2(h, Cyy, A0), bz = fma2(h, Czz, A0);
    d[1] = mul2(w1, DEV ? fma2(r3, ux, bx) : add2(bx, Bx));  d[2] = mul2(w1, DEV ? fma2(n3, ux, bx) : sub2(bx, Bx));
    d[3] = mul2(w1, DEV ? fma2(r3, uy, by) : add2(by, By));  d[4] = mul2(w1, DEV ? fma2(n3, uy, by) : sub2(by, By));
    d[5] = mul2(w1, DEV ? fma2(r3, uz, bz) : add2(bz, Bz));  d[6] = mul2(w1, DEV ? fma2(n3, uz, bz) : sub2(bz, Bz));
    const float2 bxy = fma2(h, Cyy, bx), bxz = fma2(h, Czz, bx), byz = fma2(h, Czz, by);
    float2 b, B;
    b = fma2(p9, Cxy, bxy); B = DEV ? fma2(r3, ux, By) : add2(Bx, By);
    d[7] = mul2(w2, add2(b, B));  d[8] = mul2(w2, sub2(b, B));
    b = fma2(n9, Cxy, bxy); B = DEV ? fma2(r3, ux, mul2(n3, uy)) : sub2(Bx, By);
    d[9] = mul2(w2, add2(b, B));  d[10] = mul2(w2, sub2(b, B));
    b = fma2(p9, Cxz, bxz); B = DEV ? fma2(r3, ux, Bz) : add2(Bx, Bz);
    d[11] = mul2(w2, add2(b, B)); d[12] = mul2(w2, sub2(b, B));
    b = fma2(n9, Cxz, bxz); B = DEV ? fma2(r3, ux, mul2(n3, uz)) : sub2(Bx, Bz);
    d[13] = mul2(w2, add2(b, B)); d[14] = mul2(w2, sub2(b, B));
    b = fma2(p9, Cyz, byz); B = add2(By, Bz);
    d[15] = mul2(w2, add2(b, B)); d[16] = mul2(w2, sub2(b, B));
    b = fma2(n9, Cyz, byz); B = sub2(By, Bz);
    d[17] = mul2(w2, add2(b, B)); d[18] = mul2(w2, sub2(b, B));
}
