// d3q19.cuh -- D3Q19 lattice constants and the per-cell physics shared by every kernel.
//
// The velocity set, weights, opposite and lid-mirror maps are the reference's
// (floodsim/lbm3d.py:16-21); they are constexpr functions so that, inside fully
// unrolled direction loops, every c_i, w_i and index folds to a literal.
#pragma once
#include <cmath>
#include <cstdint>

namespace wfs {

constexpr int Q = 19;

__host__ __device__ constexpr int cx(int i) {
    return (i == 1 || i == 7 || i == 9 || i == 11 || i == 13) ? 1
         : (i == 2 || i == 8 || i == 10 || i == 12 || i == 14) ? -1 : 0;
}
__host__ __device__ constexpr int cy(int i) {
    return (i == 3 || i == 7 || i == 10 || i == 15 || i == 17) ? 1
         : (i == 4 || i == 8 || i == 9 || i == 16 || i == 18) ? -1 : 0;
}
__host__ __device__ constexpr int cz(int i) {
    return (i == 5 || i == 11 || i == 14 || i == 15 || i == 18) ? 1
         : (i == 6 || i == 12 || i == 13 || i == 16 || i == 17) ? -1 : 0;
}
__host__ __device__ constexpr int opp(int i) { return i == 0 ? 0 : ((i & 1) ? i + 1 : i - 1); }
// reflection in the rigid lid: swaps the +z and -z member of each z-moving pair
__host__ __device__ constexpr int mirz(int i) {
    return i == 5 ? 6 : i == 6 ? 5 : i == 11 ? 13 : i == 13 ? 11 : i == 12 ? 14 : i == 14 ? 12
         : i == 15 ? 17 : i == 17 ? 15 : i == 16 ? 18 : i == 18 ? 16 : i;
}
__host__ __device__ constexpr float wgt(int i) {
    return i == 0 ? 1.0f / 3.0f : (i < 7 ? 1.0f / 18.0f : 1.0f / 36.0f);
}
__host__ __device__ constexpr double wgt64(int i) {
    return i == 0 ? 1.0 / 3.0 : (i < 7 ? 1.0 / 18.0 : 1.0 / 36.0);
}

// Element of the population array (19 planes of S cells) that direction I pulls for the cell with
// element index `own` in a plane (fk its flag word): at a wall the opposite population of the cell
// itself, across an x end the cell's own, under the lid the mirrored one, else the neighbour's.
// The planes' bases and the offsets are uniform, so a lane selects one and adds.  64-bit sums: the
// opposite direction's plane is S cells away, so own and offset together pass 2^31 on lattices of
// more than 2^30 cells (16-bit storage of 1.5e9 cells fits one GPU).  Int = int32_t, for lattices of up
// to 2^30 cells: 32-bit sums but under the lid, whose mirrored plane may be two away.
template <int I, typename Int = long long>
__host__ __device__ __forceinline__ long long pull_element(Int own, Int plane, int pitch, long long S,
                                                           uint32_t fk, bool lid, bool x_first, bool x_last)
{
    const bool edge = cx(I) == 1 ? x_first : cx(I) == -1 ? x_last : false;
    if constexpr (sizeof(Int) == 4 && cz(I) != -1) {
        Int off = -(cz(I) * plane + cy(I) * pitch + cx(I));
        if (cx(I)) off = edge ? 0 : off;
        if (I > 0) off = (fk & (1u << I)) ? (opp(I) - I) * (Int)S : off;
        return I * S + (own + off);
    }
    long long off = I * S - (cz(I) * plane + (long long)cy(I) * pitch + cx(I));
    if (cz(I) == -1) off = lid ? mirz(I) * S - ((long long)cy(I) * pitch + cx(I)) : off;
    if (cx(I)) off = edge ? I * S : off;
    if (I > 0) off = (fk & (1u << I)) ? opp(I) * S : off;
    return own + off;
}

// Cell flag word (one uint32 per cell).
constexpr uint32_t FLAG_WALLS = 0x0007FFFEu;   // bit i (1..18): pull source of direction i is a wall
constexpr uint32_t FLAG_SOLID = 1u << 19;      // solid cell (never collided)
constexpr uint32_t FLAG_FORCE = 1u << 20;      // body force is non-zero here
constexpr uint32_t FLAG_WALLFN = 1u << 21;     // wall function applies (cf > 0 and a usable wall normal)
constexpr uint32_t FLAG_BEDWALL = 1u << 22;    // bed/bank wall cell: reference speed is the column mean
constexpr uint32_t FLAG_GHOST = 1u << 23;      // x padding beyond nx (treated as solid)

// Float operations with their rounding fixed: a product or sum rounded on its own, a
// multiply-add rounded once.  The collision and the inlet/outlet rule are written in these, so
// that every kernel that inlines them computes the same bits whatever the compiler would fuse.
__host__ __device__ __forceinline__ float mul_rn(float a, float b)
{
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
__host__ __device__ __forceinline__ float add_rn(float a, float b)
{
#ifdef __CUDA_ARCH__
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
__host__ __device__ __forceinline__ float sub_rn(float a, float b)
{
#ifdef __CUDA_ARCH__
    return __fsub_rn(a, b);
#else
    return a - b;
#endif
}
__host__ __device__ __forceinline__ float fma_rn(float a, float b, float c)
{
#ifdef __CUDA_ARCH__
    return __fmaf_rn(a, b, c);
#else
    return fmaf(a, b, c);
#endif
}

// Regularized-BGK + Smagorinsky + Guo collision (floodsim/lbm3d.py:103-137), in
// moment space.  With the half-force velocity u = (j + F/2)/rho and the
// non-equilibrium stress Pi = sum c c f - rho (u u + I/3), the reference's
//   feq_i + (1 - om) (fneq_i + fneq1_i) + src_i
// is exactly  w_i [ A0 + c_i.B + c_i.C.c_i ]  with
//   A0 = rho - 1.5 rho u^2 - 1.5 (1-om) tr Pi - 3 sf u.F
//   B  = 3 rho u + (3 sf - 1.5 (1-om)) F
//   C  = 4.5 [ rho u u + (1-om) Pi + sf (u F + F u) ]      (sf = 1 - om/2)
// which needs no per-direction equilibrium.  On return f holds the post-collision
// populations and r/ux/uy/uz the cell's density and velocity.
// FORCED false: no body force (the terms in F drop out).
// UX2: round ux^2 on its own in |u|^2 (kernels that also accumulate ux^2 share the product), else uy^2.
template <bool FORCED, bool UX2 = false>
__host__ __device__ __forceinline__ void collide(float (&f)[Q], float fx, float fy, float fz, float tau0, float csmag2,
                                        float& r, float& ux, float& uy, float& uz)
{
    const float s1 = f[1] + f[2], d1 = f[1] - f[2];
    const float s3 = f[3] + f[4], d3 = f[3] - f[4];
    const float s5 = f[5] + f[6], d5 = f[5] - f[6];
    const float s7 = f[7] + f[8], d7 = f[7] - f[8];
    const float s9 = f[9] + f[10], d9 = f[9] - f[10];
    const float s11 = f[11] + f[12], d11 = f[11] - f[12];
    const float s13 = f[13] + f[14], d13 = f[13] - f[14];
    const float s15 = f[15] + f[16], d15 = f[15] - f[16];
    const float s17 = f[17] + f[18], d17 = f[17] - f[18];
    r = f[0] + (s1 + s3 + s5) + (s7 + s9 + s11) + (s13 + s15 + s17);
    const float jx = d1 + d7 + d9 + d11 + d13;
    const float jy = d3 + d7 - d9 + d15 + d17;
    const float jz = d5 + d11 - d13 + d15 - d17;
    const float sxx = s1 + s7 + s9 + s11 + s13;
    const float syy = s3 + s7 + s9 + s15 + s17;
    const float szz = s5 + s11 + s13 + s15 + s17;
    const float sxy = s7 - s9, sxz = s11 - s13, syz = s15 - s17;

    const float ir = 1.0f / r;
    ux = mul_rn(FORCED ? fma_rn(0.5f, fx, jx) : jx, ir);
    uy = mul_rn(FORCED ? fma_rn(0.5f, fy, jy) : jy, ir);
    uz = mul_rn(FORCED ? fma_rn(0.5f, fz, jz) : jz, ir);
    // the products r u u serve both the stress and the equilibrium
    const float rx = mul_rn(r, ux), ry = mul_rn(r, uy), rz = mul_rn(r, uz);
    const float rxx = mul_rn(rx, ux), ryy = mul_rn(ry, uy), rzz = mul_rn(rz, uz);
    const float rxy = mul_rn(rx, uy), rxz = mul_rn(rx, uz), ryz = mul_rn(ry, uz);
    const float third = -(1.0f / 3.0f);
    const float pxx = fma_rn(third, r, sub_rn(sxx, rxx)), pyy = fma_rn(third, r, sub_rn(syy, ryy)),
                pzz = fma_rn(third, r, sub_rn(szz, rzz));
    const float pxy = sub_rn(sxy, rxy), pxz = sub_rn(sxz, rxz), pyz = sub_rn(syz, ryz);

    const float qd = fma_rn(pzz, pzz, fma_rn(pxx, pxx, mul_rn(pyy, pyy)));
    const float qo = fma_rn(pyz, pyz, fma_rn(pxy, pxy, mul_rn(pxz, pxz)));
    const float qn = sqrtf(fma_rn(2.0f, qo, qd));
    const float tau0sq = mul_rn(tau0, tau0), smag = mul_rn(18.0f * 1.41421356f, csmag2);
    const float tau = mul_rn(0.5f, add_rn(tau0, sqrtf(fma_rn(mul_rn(smag, qn), ir, tau0sq))));
    const float om = 1.0f / tau;
    const float k1 = sub_rn(1.0f, om);

    const float usq = fma_rn(uz, uz, UX2 ? fma_rn(uy, uy, mul_rn(ux, ux)) : fma_rn(ux, ux, mul_rn(uy, uy)));
    const float trace = add_rn(add_rn(pxx, pyy), pzz);
    float A0 = fma_rn(-1.5f, fma_rn(k1, trace, mul_rn(r, usq)), r);
    const float r3 = mul_rn(3.0f, r);
    float Bx = mul_rn(r3, ux), By = mul_rn(r3, uy), Bz = mul_rn(r3, uz);
    float Cxx = fma_rn(k1, pxx, rxx), Cyy = fma_rn(k1, pyy, ryy), Czz = fma_rn(k1, pzz, rzz);
    float Cxy = fma_rn(k1, pxy, rxy), Cxz = fma_rn(k1, pxz, rxz), Cyz = fma_rn(k1, pyz, ryz);
    if constexpr (FORCED) {
        const float sf = fma_rn(-0.5f, om, 1.0f);
        const float uF = fma_rn(uz, fz, fma_rn(uy, fy, mul_rn(ux, fx)));
        A0 = fma_rn(mul_rn(-3.0f, sf), uF, A0);
        const float bf = fma_rn(-1.5f, k1, mul_rn(3.0f, sf));
        Bx = fma_rn(bf, fx, Bx);
        By = fma_rn(bf, fy, By);
        Bz = fma_rn(bf, fz, Bz);
        const float sf2 = mul_rn(2.0f, sf);
        Cxx = fma_rn(mul_rn(sf2, ux), fx, Cxx);
        Cyy = fma_rn(mul_rn(sf2, uy), fy, Cyy);
        Czz = fma_rn(mul_rn(sf2, uz), fz, Czz);
        Cxy = fma_rn(sf, fma_rn(fx, uy, mul_rn(ux, fy)), Cxy);
        Cxz = fma_rn(sf, fma_rn(fx, uz, mul_rn(ux, fz)), Cxz);
        Cyz = fma_rn(sf, fma_rn(fy, uz, mul_rn(uy, fz)), Cyz);
    }
    // f_i = w_i (A0 + c.B + c.C.c), C's factors 4.5 (diagonal) and 9 (off-diagonal) applied here
    constexpr float w0 = wgt(0), w1 = wgt(1), w2 = wgt(7);
    f[0] = mul_rn(w0, A0);
    const float bx = fma_rn(4.5f, Cxx, A0), by = fma_rn(4.5f, Cyy, A0), bz = fma_rn(4.5f, Czz, A0);
    f[1] = mul_rn(w1, add_rn(bx, Bx));  f[2] = mul_rn(w1, sub_rn(bx, Bx));
    f[3] = mul_rn(w1, add_rn(by, By));  f[4] = mul_rn(w1, sub_rn(by, By));
    f[5] = mul_rn(w1, add_rn(bz, Bz));  f[6] = mul_rn(w1, sub_rn(bz, Bz));
    const float bxy = fma_rn(4.5f, Cyy, bx), bxz = fma_rn(4.5f, Czz, bx), byz = fma_rn(4.5f, Czz, by);
    float b, B;
    b = fma_rn(9.0f, Cxy, bxy);   B = add_rn(Bx, By);  f[7] = mul_rn(w2, add_rn(b, B));  f[8] = mul_rn(w2, sub_rn(b, B));
    b = fma_rn(-9.0f, Cxy, bxy);  B = sub_rn(Bx, By);  f[9] = mul_rn(w2, add_rn(b, B));  f[10] = mul_rn(w2, sub_rn(b, B));
    b = fma_rn(9.0f, Cxz, bxz);   B = add_rn(Bx, Bz);  f[11] = mul_rn(w2, add_rn(b, B)); f[12] = mul_rn(w2, sub_rn(b, B));
    b = fma_rn(-9.0f, Cxz, bxz);  B = sub_rn(Bx, Bz);  f[13] = mul_rn(w2, add_rn(b, B)); f[14] = mul_rn(w2, sub_rn(b, B));
    b = fma_rn(9.0f, Cyz, byz);   B = add_rn(By, Bz);  f[15] = mul_rn(w2, add_rn(b, B)); f[16] = mul_rn(w2, sub_rn(b, B));
    b = fma_rn(-9.0f, Cyz, byz);  B = sub_rn(By, Bz);  f[17] = mul_rn(w2, add_rn(b, B)); f[18] = mul_rn(w2, sub_rn(b, B));
}

// Direction masks over bits 1..18 (bit i = direction i), for popcount sums over a wall mask.
template <typename P>
__host__ __device__ constexpr uint32_t dir_mask(P pred)
{
    uint32_t m = 0;
    for (int i = 1; i < Q; ++i)
        if (pred(i)) m |= 1u << i;
    return m;
}
__host__ __device__ __forceinline__ int popc32(uint32_t v)
{
#ifdef __CUDA_ARCH__
    return __popc(v);
#else
    return __builtin_popcount(v);
#endif
}

// The wall function's small-integer float64 operations, exact or correctly rounded like the
// general ones they stand for, without the conversion unit's or the square root's latency:
// int_double -- a small signed integer: its bits under the exponent of 2^52, less the bias;
// sqrt_small -- the square root of 0..12, tabulated;
// div_small  -- p / n for n = 1..75 by Markstein's correction (IBM J. Res. Dev. 34, 1990): with y the
//               correctly rounded 1/n and q0 = p y, q0 + (p - q0 n) y rounds to the quotient.
#ifdef __CUDACC__
constexpr int kSmallDivisors = 76;
struct SmallTables {
    double root[13], inverse[kSmallDivisors];
};
constexpr SmallTables small_tables()
{
    SmallTables t{{0.0, 1.0, 1.4142135623730951, 1.7320508075688772, 2.0, 2.23606797749979, 2.449489742783178, 2.6457513110645907, 2.8284271247461903, 3.0, 3.1622776601683795, 3.3166247903554, 3.4641016151377544},
                  {}};
    for (int k = 1; k < kSmallDivisors; ++k) t.inverse[k] = 1.0 / k;
    return t;
}
__device__ __constant__ constexpr SmallTables kSmall = small_tables();
#endif
__host__ __device__ __forceinline__ double int_double(int k)
{
#ifdef __CUDA_ARCH__
    return __hiloint2double(0x43300000, k ^ (int)0x80000000) - 4503601774854144.0;       // 2^52 + 2^31
#else
    return k;
#endif
}
__host__ __device__ __forceinline__ double sqrt_small(int k)
{
#ifdef __CUDA_ARCH__
    return kSmall.root[k];
#else
    return sqrt((double)k);
#endif
}
__host__ __device__ __forceinline__ double div_small(double p, int n)
{
#ifdef __CUDA_ARCH__
    const double y = kSmall.inverse[n], d = int_double(n), q = p * y;
    return fma(fma(-q, d, p), y, q);
#else
    return p / n;
#endif
}

// Wall function (floodsim/lbm3d.py:61-101): moving-wall bounce-back whose tangential
// wall speed u_s makes the momentum a cell gives its wall faces per step equal
// the log-law/Manning shear rho*cf*U^2*area.  `wm` is the cell's wall mask
// (bits 1..18), f[i] at a wall direction already holds the bounced f*_opp,
// (px,py,pz,rw) are the cell's previous-step velocity and density, and
// `uref` the reference speed (<= 0 means: use the local tangential speed).
//
// Evaluated in float64, as the reference's CPU twin does (floodsim/lbm3d.py:230-252):
// the tangent t = u_t/|u_t| is ill-conditioned where |u_t| is small, and in float32
// its rounding alone moves wall cells by ~1e-6 of max|u| per step.
//
// The reference's sums over the wall directions are regrouped so that only one pass over
// the populations remains: with c_i the wall directions' velocities,
//   n = -sum c_i                         (popcounts of the mask: c components are 0, +-1)
//   D = sum (c_i.t) f_i = t . J,          J = sum c_i f_i
//   K = sum w_i (c_i.t)^2 = t^T M t,      M = sum w_i c_i c_i^T  (popcounts again)
// and the update f_i += g w_i (c_i.t) is f_i += w_i c_i.(g t); the unit vectors are never
// formed (see below), which leaves two square roots and two divisions.  The float64 results
// differ from the per-direction sums only by float64 reassociation.
__host__ __device__ __forceinline__ void wall_function(float (&f)[Q], uint32_t wm, float cf, float px, float py, float pz,
                                                       float rw, float uref)
{
    constexpr uint32_t PX = dir_mask([](int i) { return cx(i) == 1; }), NX = dir_mask([](int i) { return cx(i) == -1; });
    constexpr uint32_t PY = dir_mask([](int i) { return cy(i) == 1; }), NY = dir_mask([](int i) { return cy(i) == -1; });
    constexpr uint32_t PZ = dir_mask([](int i) { return cz(i) == 1; }), NZ = dir_mask([](int i) { return cz(i) == -1; });
    constexpr uint32_t AXIS = 0x7Eu;                                          // directions 1..6 (weight 1/18)
    constexpr uint32_t XY_SAME = dir_mask([](int i) { return cx(i) * cy(i) == 1; });
    constexpr uint32_t XY_OPP = dir_mask([](int i) { return cx(i) * cy(i) == -1; });
    constexpr uint32_t XZ_SAME = dir_mask([](int i) { return cx(i) * cz(i) == 1; });
    constexpr uint32_t XZ_OPP = dir_mask([](int i) { return cx(i) * cz(i) == -1; });
    constexpr uint32_t YZ_SAME = dir_mask([](int i) { return cy(i) * cz(i) == 1; });
    constexpr uint32_t YZ_OPP = dir_mask([](int i) { return cy(i) * cz(i) == -1; });
    const uint32_t wx = wm & (PX | NX), wy = wm & (PY | NY), wz = wm & (PZ | NZ);
    const int nwx = popc32(wm & NX) - popc32(wm & PX);
    const int nwy = popc32(wm & NY) - popc32(wm & PY);
    const int nwz = popc32(wm & NZ) - popc32(wm & PZ);
    const int n2 = nwx * nwx + nwy * nwy + nwz * nwz;
    const int afx = (int)(((wm >> 1) & 1u) + ((wm >> 2) & 1u));
    const int afy = (int)(((wm >> 3) & 1u) + ((wm >> 4) & 1u));
    const int afz = (int)(((wm >> 5) & 1u) + ((wm >> 6) & 1u));
    const int a2 = afx * afx + afy * afy + afz * afz;
    if (n2 <= 0 || a2 <= 0) return;
    // Tangential velocity t = p - (p.n) n / |n|^2 (n the integer wall normal: no square root
    // needed for it), ut = |t|.  With the unit tangent t/ut the reference's slip speed is
    //   us0 = (-2 D - rw cf U^2 area) / (6 rw K),  D = (t.J)/ut,  K = (t^T M t)/ut^2,
    // clamped to [-ut, ut], and the update f_i += w_i c_i.(6 rw us t/ut); so with
    //   s = us0/ut = (-2 (t.J) - rw cf U^2 area ut) / (6 rw t^T M t)
    // the update is f_i += w_i c_i.(6 rw clamp(s, -1, 1) t): one square root for ut, one for
    // the face area, one division -- the same quantities as the reference's, regrouped.
    const double area = sqrt_small(a2);
    const double nx = int_double(nwx), ny = int_double(nwy), nz = int_double(nwz);
    const double pn = (double)px * nx + (double)py * ny + (double)pz * nz;
    const double q = div_small(pn, n2);
    const double tx = px - q * nx, ty = py - q * ny, tz = pz - q * nz;
    const double ut = sqrt(tx * tx + ty * ty + tz * tz);
    if (!(ut > 1e-7)) return;
    double jx = 0.0, jy = 0.0, jz = 0.0;
#pragma unroll
    for (int i = 1; i < Q; ++i)
        if (wm & (1u << i)) {
            const double fi = (double)f[i];
            if (cx(i) == 1) jx += fi; else if (cx(i) == -1) jx -= fi;
            if (cy(i) == 1) jy += fi; else if (cy(i) == -1) jy -= fi;
            if (cz(i) == 1) jz += fi; else if (cz(i) == -1) jz -= fi;
        }
    const double tJ = tx * jx + ty * jy + tz * jz;
    const double w1 = (double)wgt(1), w2 = (double)wgt(7);
    const double mxx = w1 * int_double(popc32(wx & AXIS)) + w2 * int_double(popc32(wx & ~AXIS));
    const double myy = w1 * int_double(popc32(wy & AXIS)) + w2 * int_double(popc32(wy & ~AXIS));
    const double mzz = w1 * int_double(popc32(wz & AXIS)) + w2 * int_double(popc32(wz & ~AXIS));
    const double mxy = w2 * int_double(popc32(wm & XY_SAME) - popc32(wm & XY_OPP));
    const double mxz = w2 * int_double(popc32(wm & XZ_SAME) - popc32(wm & XZ_OPP));
    const double myz = w2 * int_double(popc32(wm & YZ_SAME) - popc32(wm & YZ_OPP));
    const double tMt = tx * tx * mxx + ty * ty * myy + tz * tz * mzz + 2.0 * (tx * ty * mxy + tx * tz * mxz + ty * tz * myz);
    if (!(tMt > 0.0)) return;
    const double U = uref > 0.f ? (double)uref : ut;
    const double s0 = (-2.0 * tJ - (double)(rw * cf) * U * U * area * ut) / (6.0 * (double)rw * tMt);
    const double sc = fmin(fmax(s0, -1.0), 1.0);
    const double g = 6.0 * (double)rw * sc;
    const double gx = g * tx, gy = g * ty, gz = g * tz;
#pragma unroll
    for (int i = 1; i < Q; ++i)
        if (wm & (1u << i)) {
            double ct = 0.0;
            if (cx(i)) ct += cx(i) * gx;
            if (cy(i)) ct += cy(i) * gy;
            if (cz(i)) ct += cz(i) * gz;
            f[i] = (float)((double)f[i] + (double)wgt(i) * ct);
        }
}

// Inlet velocity / outlet pressure by non-equilibrium extrapolation
// (floodsim/lbm3d.py:153-174): g = post-collision populations of the interior
// neighbour (x=1 or x=nx-2), out = the boundary cell's new populations,
//   out_i = feq_i(rho_b, u_b) + g_i - feq_i(rho_g, u_g),
// inlet: rho_b = rho_g, u_b = (uin,0,0); outlet: rho_b = rho_out, u_b = u_g.
// The difference of the two second-order equilibria is itself a quadratic form,
//   feq_i(rho_b, u_b) - feq_i(rho_g, u_g) = w_i [A + c_i.B + c_i.C.c_i],
//   A = -1.5 (rho_b u_b^2 - rho_g u_g^2) + (rho_b - rho_g),
//   B = 3 (rho_b u_b - rho_g u_g),  C = 4.5 (rho_b u_b u_b - rho_g u_g u_g),
// so it is evaluated like the collision's output stage (one pass, no per-direction
// equilibria); the result differs from the reference's order of operations only by
// float32 rounding.  `inlet` is a runtime switch, so that one copy of the code serves both ends.
__host__ __device__ __forceinline__ void nebb(bool inlet, const float (&g)[Q], float (&out)[Q], float uin, float rho_out)
{
    const float s1 = g[1] + g[2], d1 = g[1] - g[2];
    const float s3 = g[3] + g[4], d3 = g[3] - g[4];
    const float s5 = g[5] + g[6], d5 = g[5] - g[6];
    const float s7 = g[7] + g[8], d7 = g[7] - g[8];
    const float s9 = g[9] + g[10], d9 = g[9] - g[10];
    const float s11 = g[11] + g[12], d11 = g[11] - g[12];
    const float s13 = g[13] + g[14], d13 = g[13] - g[14];
    const float s15 = g[15] + g[16], d15 = g[15] - g[16];
    const float s17 = g[17] + g[18], d17 = g[17] - g[18];
    const float r = g[0] + (s1 + s3 + s5) + (s7 + s9 + s11) + (s13 + s15 + s17);
    const float mx = d1 + d7 + d9 + d11 + d13;
    const float my = d3 + d7 - d9 + d15 + d17;
    const float mz = d5 + d11 - d13 + d15 - d17;
    const float ir = 1.0f / r;
    const float ux = mul_rn(mx, ir), uy = mul_rn(my, ir), uz = mul_rn(mz, ir);
    const float rb = inlet ? r : rho_out, bx = inlet ? uin : ux, by = inlet ? 0.f : uy, bz = inlet ? 0.f : uz;
    const float usq = fma_rn(uz, uz, fma_rn(ux, ux, mul_rn(uy, uy)));
    const float bsq = fma_rn(bz, bz, fma_rn(bx, bx, mul_rn(by, by)));
    const float A = fma_rn(-1.5f, fma_rn(rb, bsq, -mul_rn(r, usq)), sub_rn(rb, r));
    // rho u and rho u u of the boundary state less those of g
    const float rx = mul_rn(r, ux), ry = mul_rn(r, uy), rz = mul_rn(r, uz);
    const float px = mul_rn(rb, bx), py = mul_rn(rb, by), pz = mul_rn(rb, bz);
    const float jx = sub_rn(px, rx), jy = sub_rn(py, ry), jz = sub_rn(pz, rz);
    const float Bx = mul_rn(3.0f, jx), By = mul_rn(3.0f, jy), Bz = mul_rn(3.0f, jz);
    const float Cxx = fma_rn(px, bx, -mul_rn(rx, ux)), Cyy = fma_rn(py, by, -mul_rn(ry, uy)),
                Czz = fma_rn(pz, bz, -mul_rn(rz, uz));
    const float Cxy = fma_rn(px, by, -mul_rn(rx, uy)), Cxz = fma_rn(px, bz, -mul_rn(rx, uz)),
                Cyz = fma_rn(py, bz, -mul_rn(ry, uz));
    constexpr float w0 = wgt(0), w1 = wgt(1), w2 = wgt(7);
    out[0] = fma_rn(w0, A, g[0]);
    const float bxx = fma_rn(4.5f, Cxx, A), byy = fma_rn(4.5f, Cyy, A), bzz = fma_rn(4.5f, Czz, A);
    out[1] = fma_rn(w1, fma_rn(3.0f, jx, bxx), g[1]);  out[2] = fma_rn(w1, fma_rn(-3.0f, jx, bxx), g[2]);
    out[3] = fma_rn(w1, fma_rn(3.0f, jy, byy), g[3]);  out[4] = fma_rn(w1, fma_rn(-3.0f, jy, byy), g[4]);
    out[5] = fma_rn(w1, fma_rn(3.0f, jz, bzz), g[5]);  out[6] = fma_rn(w1, fma_rn(-3.0f, jz, bzz), g[6]);
    const float bxy = fma_rn(4.5f, Cyy, bxx), bxz = fma_rn(4.5f, Czz, bxx), byz = fma_rn(4.5f, Czz, byy);
    float b, c;
    b = fma_rn(9.0f, Cxy, bxy);   c = fma_rn(3.0f, jx, By);
    out[7] = fma_rn(w2, add_rn(b, c), g[7]);   out[8] = fma_rn(w2, sub_rn(b, c), g[8]);
    b = fma_rn(-9.0f, Cxy, bxy);  c = fma_rn(3.0f, jx, -By);
    out[9] = fma_rn(w2, add_rn(b, c), g[9]);   out[10] = fma_rn(w2, sub_rn(b, c), g[10]);
    b = fma_rn(9.0f, Cxz, bxz);   c = fma_rn(3.0f, jx, Bz);
    out[11] = fma_rn(w2, add_rn(b, c), g[11]); out[12] = fma_rn(w2, sub_rn(b, c), g[12]);
    b = fma_rn(-9.0f, Cxz, bxz);  c = fma_rn(3.0f, jx, -Bz);
    out[13] = fma_rn(w2, add_rn(b, c), g[13]); out[14] = fma_rn(w2, sub_rn(b, c), g[14]);
    b = fma_rn(9.0f, Cyz, byz);   c = add_rn(By, Bz);
    out[15] = fma_rn(w2, add_rn(b, c), g[15]); out[16] = fma_rn(w2, sub_rn(b, c), g[16]);
    b = fma_rn(-9.0f, Cyz, byz);  c = sub_rn(By, Bz);
    out[17] = fma_rn(w2, add_rn(b, c), g[17]); out[18] = fma_rn(w2, sub_rn(b, c), g[18]);
}

}  // namespace wfs
