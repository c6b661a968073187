// Butterflies of the runtime-radix kernel (rx_kernel.cuh) on 16-byte vectors.
//
// A vector holds one complex value of each of W sequences: two in f32, as
// (re0, re1, im0, im1) so that every operation is one packed f32x2
// instruction, one in f64.  All transforms here are forward ones: an inverse
// pass reads its input in reversed index order instead.
#pragma once

#include <cuda_runtime.h>

#include "pb_fft.cuh"

namespace pb {

// two f32 values advanced by one instruction
struct Q2 { float2 v; };
__device__ __forceinline__ Q2 qadd(Q2 a, Q2 b) { return Q2{__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ Q2 qmul(Q2 a, Q2 b) { return Q2{__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ Q2 qfma(Q2 a, Q2 b, Q2 c) { return Q2{__ffma2_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ Q2 qsub(Q2 a, Q2 b) { return Q2{__ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v)}; }
__device__ __forceinline__ double qadd(double a, double b) { return a + b; }
__device__ __forceinline__ double qsub(double a, double b) { return a - b; }
__device__ __forceinline__ double qmul(double a, double b) { return a * b; }
__device__ __forceinline__ double qfma(double a, double b, double c) { return fma(a, b, c); }
template <typename Q> __device__ __forceinline__ Q qc(double c);
template <> __device__ __forceinline__ Q2 qc<Q2>(double c) { return Q2{make_float2((float)c, (float)c)}; }
template <> __device__ __forceinline__ double qc<double>(double c) { return c; }

template <typename R> struct Vec;
template <> struct Vec<float> { using Q = Q2; static constexpr int W = 2; };
template <> struct Vec<double> { using Q = double; static constexpr int W = 1; };
template <typename Q> struct __align__(16) VC { Q x, y; };

template <typename Q> __device__ __forceinline__ VC<Q> vadd(VC<Q> a, VC<Q> b) { return {qadd(a.x, b.x), qadd(a.y, b.y)}; }
template <typename Q> __device__ __forceinline__ VC<Q> vsub(VC<Q> a, VC<Q> b) { return {qsub(a.x, b.x), qsub(a.y, b.y)}; }
// a -+ i b
template <typename Q> __device__ __forceinline__ VC<Q> vaddr(VC<Q> a, VC<Q> b) { return {qadd(a.x, b.y), qsub(a.y, b.x)}; }
template <typename Q> __device__ __forceinline__ VC<Q> vsubr(VC<Q> a, VC<Q> b) { return {qsub(a.x, b.y), qadd(a.y, b.x)}; }
// v * w
template <typename Q> __device__ __forceinline__ VC<Q> vtw(VC<Q> v, VC<Q> w) {
  const Q nwy = qmul(w.y, qc<Q>(-1.0));
  return {qfma(v.y, nwy, qmul(v.x, w.x)), qfma(v.x, w.y, qmul(v.y, w.x))};
}
// What rounding the constant k to the type took from it (lo: what rounding it
// to f64 took), 0 where that is at most 0.3 of the unit roundoff.
template <typename Q> __device__ __forceinline__ double kres(double k, double lo);
template <> __device__ __forceinline__ double kres<Q2>(double k, double) {
  const double d = k - (double)(float)k, q = (k < 0.0 ? -k : k) * (0.3 / 16777216.0);
  return d > q || -d > q ? d : 0.0;
}
template <> __device__ __forceinline__ double kres<double>(double, double lo) { return lo; }
// v * (c - i s), constants with their residues cl and sl.  The residues'
// products come first and the larger constant's last.  A constant's rounding
// error is of the size of the arithmetic's and the same in every line, and a
// radix-16 stage rotates by constants where radix-8 stages of the same length
// hardly do.  4096^2 points f32, forward and back, against 64 bits: 2.8e-7
// without the residues, 2.4e-7 with them, 2.6e-7 in the generic kernel's four
// radix-8 stages (392, 400 and 2330 us).
template <typename Q> __device__ __forceinline__ VC<Q> vrotc(VC<Q> v, double c, double cl, double s, double sl) {
  VC<Q> a = {qc<Q>(0.0), qc<Q>(0.0)};
  bool any = false;
  auto cosine = [&](double k) {
    if (k == 0.0) return;
    a = any ? VC<Q>{qfma(v.x, qc<Q>(k), a.x), qfma(v.y, qc<Q>(k), a.y)} : VC<Q>{qmul(v.x, qc<Q>(k)), qmul(v.y, qc<Q>(k))};
    any = true;
  };
  auto sine = [&](double k) {
    if (k == 0.0) return;
    a = any ? VC<Q>{qfma(v.y, qc<Q>(k), a.x), qfma(v.x, qc<Q>(-k), a.y)}
            : VC<Q>{qmul(v.y, qc<Q>(k)), qmul(v.x, qc<Q>(-k))};
    any = true;
  };
  cosine(cl);
  sine(sl);
  if (c * c < s * s) {
    cosine(c);
    sine(s);
  } else {
    sine(s);
    cosine(c);
  }
  return a;
}

// cos(2 pi i/N) and sin(2 pi i/N), correctly rounded; cl and sl are what the
// rounding took from them, 0 where that is at most 0.3 of the unit roundoff.
template <int N>
struct RxRoots;
template <>
struct RxRoots<3> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[3] = {1.0, -0.5, -0.5};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[3] = {0.0, 0.8660254037844386, -0.8660254037844386};
    return t[i];
  }
  static __host__ __device__ constexpr double cl(int i) {
    constexpr double t[3] = {0.0, 0.0, 0.0};
    return t[i];
  }
  static __host__ __device__ constexpr double sl(int i) {
    constexpr double t[3] = {0.0, 5.0175421109034514e-17, -5.0175421109034514e-17};
    return t[i];
  }
};
template <>
struct RxRoots<5> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[5] = {1.0, 0.30901699437494745, -0.8090169943749475, -0.8090169943749475, 0.30901699437494745};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[5] = {0.0, 0.9510565162951535, 0.5877852522924731, -0.5877852522924731, -0.9510565162951535};
    return t[i];
  }
  static __host__ __device__ constexpr double cl(int i) {
    constexpr double t[5] = {0.0, -2.716057601841253e-17, 2.716057601841253e-17, 2.716057601841253e-17,
        -2.716057601841253e-17};
    return t[i];
  }
  static __host__ __device__ constexpr double sl(int i) {
    constexpr double t[5] = {0.0, 4.0934500900087295e-17, 0.0, 0.0, -4.0934500900087295e-17};
    return t[i];
  }
};
template <>
struct RxRoots<6> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[6] = {1.0, 0.5, -0.5, -1.0, -0.5, 0.5};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[6] = {0.0, 0.8660254037844386, 0.8660254037844386, 0.0, -0.8660254037844386, -0.8660254037844386};
    return t[i];
  }
  static __host__ __device__ constexpr double cl(int i) {
    constexpr double t[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    return t[i];
  }
  static __host__ __device__ constexpr double sl(int i) {
    constexpr double t[6] = {0.0, 5.0175421109034514e-17, 5.0175421109034514e-17, 0.0, -5.0175421109034514e-17,
        -5.0175421109034514e-17};
    return t[i];
  }
};
template <>
struct RxRoots<7> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[7] = {1.0, 0.6234898018587335, -0.2225209339563144, -0.9009688679024191,
        -0.9009688679024191, -0.2225209339563144, 0.6234898018587335};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[7] = {0.0, 0.7818314824680298, 0.9749279121818236, 0.4338837391175581, -0.4338837391175581,
        -0.9749279121818236, -0.7818314824680298};
    return t[i];
  }
  static __host__ __device__ constexpr double cl(int i) {
    constexpr double t[7] = {0.0, 4.716099920540896e-17, -1.1412494827220627e-17, 0.0, 0.0, -1.1412494827220627e-17,
        4.716099920540896e-17};
    return t[i];
  }
  static __host__ __device__ constexpr double sl(int i) {
    constexpr double t[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    return t[i];
  }
};
template <>
struct RxRoots<9> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[9] = {1.0, 0.766044443118978, 0.17364817766693036, -0.5, -0.9396926207859084,
        -0.9396926207859084, -0.5, 0.17364817766693036, 0.766044443118978};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[9] = {0.0, 0.6427876096865394, 0.984807753012208, 0.8660254037844386, 0.3420201433256687,
        -0.3420201433256687, -0.8660254037844386, -0.984807753012208, -0.6427876096865394};
    return t[i];
  }
  static __host__ __device__ constexpr double cl(int i) {
    constexpr double t[9] = {0.0, 0.0, -1.0090493350843633e-17, 0.0, 4.3850932840020416e-17, 4.3850932840020416e-17,
        0.0, -1.0090493350843633e-17, 0.0};
    return t[i];
  }
  static __host__ __device__ constexpr double sl(int i) {
    constexpr double t[9] = {0.0, -3.659607900790949e-17, 3.905108875799298e-17, 5.0175421109034514e-17,
        2.0136016534644645e-17, -2.0136016534644645e-17, -5.0175421109034514e-17, -3.905108875799298e-17,
        3.659607900790949e-17};
    return t[i];
  }
};
template <>
struct RxRoots<10> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[10] = {1.0, 0.8090169943749475, 0.30901699437494745, -0.30901699437494745,
        -0.8090169943749475, -1.0, -0.8090169943749475, -0.30901699437494745, 0.30901699437494745,
        0.8090169943749475};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[10] = {0.0, 0.5877852522924731, 0.9510565162951535, 0.9510565162951535, 0.5877852522924731,
        0.0, -0.5877852522924731, -0.9510565162951535, -0.9510565162951535, -0.5877852522924731};
    return t[i];
  }
  static __host__ __device__ constexpr double cl(int i) {
    constexpr double t[10] = {0.0, -2.716057601841253e-17, -2.716057601841253e-17, 2.716057601841253e-17,
        2.716057601841253e-17, 0.0, 2.716057601841253e-17, 2.716057601841253e-17, -2.716057601841253e-17,
        -2.716057601841253e-17};
    return t[i];
  }
  static __host__ __device__ constexpr double sl(int i) {
    constexpr double t[10] = {0.0, 0.0, 4.0934500900087295e-17, 4.0934500900087295e-17, 0.0, 0.0, 0.0,
        -4.0934500900087295e-17, -4.0934500900087295e-17, 0.0};
    return t[i];
  }
};
template <>
struct RxRoots<11> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[11] = {1.0, 0.8412535328311812, 0.41541501300188644, -0.14231483827328514,
        -0.6548607339452851, -0.9594929736144974, -0.9594929736144974, -0.6548607339452851, -0.14231483827328514,
        0.41541501300188644, 0.8412535328311812};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[11] = {0.0, 0.5406408174555976, 0.9096319953545183, 0.9898214418809327, 0.7557495743542583,
        0.28173255684142967, -0.28173255684142967, -0.7557495743542583, -0.9898214418809327, -0.9096319953545183,
        -0.5406408174555976};
    return t[i];
  }
};
template <>
struct RxRoots<12> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[12] = {1.0, 0.8660254037844386, 0.5, 0.0, -0.5, -0.8660254037844386, -1.0,
        -0.8660254037844386, -0.5, 0.0, 0.5, 0.8660254037844386};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[12] = {0.0, 0.5, 0.8660254037844386, 1.0, 0.8660254037844386, 0.5, 0.0, -0.5,
        -0.8660254037844386, -1.0, -0.8660254037844386, -0.5};
    return t[i];
  }
  static __host__ __device__ constexpr double cl(int i) {
    constexpr double t[12] = {0.0, 5.0175421109034514e-17, 0.0, 0.0, 0.0, -5.0175421109034514e-17, 0.0,
        -5.0175421109034514e-17, 0.0, 0.0, 0.0, 5.0175421109034514e-17};
    return t[i];
  }
  static __host__ __device__ constexpr double sl(int i) {
    constexpr double t[12] = {0.0, 0.0, 5.0175421109034514e-17, 0.0, 5.0175421109034514e-17, 0.0, 0.0, 0.0,
        -5.0175421109034514e-17, 0.0, -5.0175421109034514e-17, 0.0};
    return t[i];
  }
};
template <>
struct RxRoots<13> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[13] = {1.0, 0.8854560256532099, 0.5680647467311558, 0.12053668025532305,
        -0.3546048870425356, -0.7485107481711011, -0.970941817426052, -0.970941817426052, -0.7485107481711011,
        -0.3546048870425356, 0.12053668025532305, 0.5680647467311558, 0.8854560256532099};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[13] = {0.0, 0.46472317204376856, 0.8229838658936564, 0.992708874098054, 0.9350162426854148,
        0.6631226582407952, 0.23931566428755777, -0.23931566428755777, -0.6631226582407952, -0.9350162426854148,
        -0.992708874098054, -0.8229838658936564, -0.46472317204376856};
    return t[i];
  }
};
template <>
struct RxRoots<14> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[14] = {1.0, 0.9009688679024191, 0.6234898018587335, 0.2225209339563144, -0.2225209339563144,
        -0.6234898018587335, -0.9009688679024191, -1.0, -0.9009688679024191, -0.6234898018587335,
        -0.2225209339563144, 0.2225209339563144, 0.6234898018587335, 0.9009688679024191};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[14] = {0.0, 0.4338837391175581, 0.7818314824680298, 0.9749279121818236, 0.9749279121818236,
        0.7818314824680298, 0.4338837391175581, 0.0, -0.4338837391175581, -0.7818314824680298, -0.9749279121818236,
        -0.9749279121818236, -0.7818314824680298, -0.4338837391175581};
    return t[i];
  }
  static __host__ __device__ constexpr double cl(int i) {
    constexpr double t[14] = {0.0, 0.0, 4.716099920540896e-17, 1.1412494827220627e-17, -1.1412494827220627e-17,
        -4.716099920540896e-17, 0.0, 0.0, 0.0, -4.716099920540896e-17, -1.1412494827220627e-17, 1.1412494827220627e-17,
        4.716099920540896e-17, 0.0};
    return t[i];
  }
  static __host__ __device__ constexpr double sl(int i) {
    constexpr double t[14] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    return t[i];
  }
};
template <>
struct RxRoots<15> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[15] = {1.0, 0.9135454576426009, 0.6691306063588582, 0.30901699437494745,
        -0.10452846326765347, -0.5, -0.8090169943749475, -0.9781476007338057, -0.9781476007338057,
        -0.8090169943749475, -0.5, -0.10452846326765347, 0.30901699437494745, 0.6691306063588582,
        0.9135454576426009};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[15] = {0.0, 0.4067366430758002, 0.7431448254773942, 0.9510565162951535, 0.9945218953682733,
        0.8660254037844386, 0.5877852522924731, 0.20791169081775934, -0.20791169081775934, -0.5877852522924731,
        -0.8660254037844386, -0.9945218953682733, -0.9510565162951535, -0.7431448254773942, -0.4067366430758002};
    return t[i];
  }
};
template <>
struct RxRoots<16> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[16] = {1.0, 0.9238795325112867, 0.7071067811865476, 0.3826834323650898, 0.0,
        -0.3826834323650898, -0.7071067811865476, -0.9238795325112867, -1.0, -0.9238795325112867,
        -0.7071067811865476, -0.3826834323650898, 0.0, 0.3826834323650898, 0.7071067811865476, 0.9238795325112867};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[16] = {0.0, 0.3826834323650898, 0.7071067811865476, 0.9238795325112867, 1.0,
        0.9238795325112867, 0.7071067811865476, 0.3826834323650898, 0.0, -0.3826834323650898, -0.7071067811865476,
        -0.9238795325112867, -1.0, -0.9238795325112867, -0.7071067811865476, -0.3826834323650898};
    return t[i];
  }
  static __host__ __device__ constexpr double cl(int i) {
    constexpr double t[16] = {0.0, 0.0, -4.833646656726457e-17, 0.0, 0.0, 0.0, 4.833646656726457e-17, 0.0, 0.0, 0.0,
        4.833646656726457e-17, 0.0, 0.0, 0.0, -4.833646656726457e-17, 0.0};
    return t[i];
  }
  static __host__ __device__ constexpr double sl(int i) {
    constexpr double t[16] = {0.0, 0.0, -4.833646656726457e-17, 0.0, 0.0, 0.0, -4.833646656726457e-17, 0.0, 0.0, 0.0,
        4.833646656726457e-17, 0.0, 0.0, 0.0, 4.833646656726457e-17, 0.0};
    return t[i];
  }
};
template <>
struct RxRoots<17> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[17] = {1.0, 0.9324722294043558, 0.7390089172206591, 0.44573835577653825, 0.092268359463302,
        -0.2736629900720829, -0.6026346363792564, -0.8502171357296141, -0.9829730996839018, -0.9829730996839018,
        -0.8502171357296141, -0.6026346363792564, -0.2736629900720829, 0.092268359463302, 0.44573835577653825,
        0.7390089172206591, 0.9324722294043558};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[17] = {0.0, 0.3612416661871529, 0.6736956436465572, 0.8951632913550623, 0.9957341762950345,
        0.961825643172819, 0.7980172272802395, 0.5264321628773558, 0.18374951781657034, -0.18374951781657034,
        -0.5264321628773558, -0.7980172272802395, -0.961825643172819, -0.9957341762950345, -0.8951632913550623,
        -0.6736956436465572, -0.3612416661871529};
    return t[i];
  }
};
template <>
struct RxRoots<19> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[19] = {1.0, 0.9458172417006346, 0.7891405093963936, 0.5469481581224269, 0.24548548714079915,
        -0.08257934547233232, -0.4016954246529695, -0.6772815716257411, -0.8794737512064891, -0.9863613034027223,
        -0.9863613034027223, -0.8794737512064891, -0.6772815716257411, -0.4016954246529695, -0.08257934547233232,
        0.24548548714079915, 0.5469481581224269, 0.7891405093963936, 0.9458172417006346};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[19] = {0.0, 0.3246994692046835, 0.6142127126896678, 0.8371664782625285, 0.9694002659393304,
        0.9965844930066698, 0.9157733266550574, 0.7357239106731316, 0.47594739303707356, 0.1645945902807339,
        -0.1645945902807339, -0.47594739303707356, -0.7357239106731316, -0.9157733266550574, -0.9965844930066698,
        -0.9694002659393304, -0.8371664782625285, -0.6142127126896678, -0.3246994692046835};
    return t[i];
  }
};
template <>
struct RxRoots<23> {
  static __host__ __device__ constexpr double c(int i) {
    constexpr double t[23] = {1.0, 0.9629172873477992, 0.8544194045464886, 0.6825531432186541, 0.46006503773115215,
        0.20345601305263378, -0.06824241336467098, -0.33487961217098616, -0.5766803221148672, -0.7757112907044198,
        -0.917211301505453, -0.9906859460363308, -0.9906859460363308, -0.917211301505453, -0.7757112907044198,
        -0.5766803221148672, -0.33487961217098616, -0.06824241336467098, 0.20345601305263378, 0.46006503773115215,
        0.6825531432186541, 0.8544194045464886, 0.9629172873477992};
    return t[i];
  }
  static __host__ __device__ constexpr double s(int i) {
    constexpr double t[23] = {0.0, 0.2697967711570243, 0.5195839500354336, 0.7308359642781241, 0.8878852184023752,
        0.9790840876823229, 0.9976687691905392, 0.9422609221188205, 0.816969893010442, 0.6310879443260528,
        0.39840108984624145, 0.1361666490962466, -0.1361666490962466, -0.39840108984624145, -0.6310879443260528,
        -0.816969893010442, -0.9422609221188205, -0.9976687691905392, -0.9790840876823229, -0.8878852184023752,
        -0.7308359642781241, -0.5195839500354336, -0.2697967711570243};
    return t[i];
  }
};

template <typename Q, int RAD> struct VB;
template <typename Q> struct VB<Q, 2> {
  static __device__ __forceinline__ void run(VC<Q>* v) { VC<Q> a = v[0]; v[0] = vadd(a, v[1]); v[1] = vsub(a, v[1]); }
};
template <typename Q> struct VB<Q, 4> {
  static __device__ __forceinline__ void run(VC<Q>* v) {
    VC<Q> t0 = vadd(v[0], v[2]), t1 = vsub(v[0], v[2]), t2 = vadd(v[1], v[3]), t3 = vsub(v[1], v[3]);
    v[0] = vadd(t0, t2); v[2] = vsub(t0, t2); v[1] = vaddr(t1, t3); v[3] = vsubr(t1, t3);
  }
};
template <typename Q> struct VB<Q, 8> {
  static __device__ __forceinline__ void run(VC<Q>* v) {
    const Q h = qc<Q>(0.70710678118654752440), nh = qc<Q>(-0.70710678118654752440);
    VC<Q> e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    VB<Q, 4>::run(e);
    VB<Q, 4>::run(o);
    v[0] = vadd(e[0], o[0]); v[4] = vsub(e[0], o[0]);
    const VC<Q> t1 = vaddr(o[1], o[1]);  // o(1 - i)
    v[1] = {qfma(t1.x, h, e[1].x), qfma(t1.y, h, e[1].y)};
    v[5] = {qfma(t1.x, nh, e[1].x), qfma(t1.y, nh, e[1].y)};
    v[2] = vaddr(e[2], o[2]); v[6] = vsubr(e[2], o[2]);
    const VC<Q> t3 = vsubr(o[3], o[3]);  // o(1 + i); W^3 o = -h (1 + i) o
    v[3] = {qfma(t3.x, nh, e[3].x), qfma(t3.y, nh, e[3].y)};
    v[7] = {qfma(t3.x, h, e[3].x), qfma(t3.y, h, e[3].y)};
  }
};
// Radices 3, 5 and 7.  RES: the constants with their residues (f64 sin(2 pi / 3)
// is off by half the unit roundoff: 1296 points f64, forward and back, 4.3e-16
// without, 3.8e-16 on the generic kernel).
template <typename Q, int RAD, bool RES> struct VBOdd {
  static __device__ __forceinline__ void run(VC<Q>* v) {
    constexpr int H = (RAD - 1) / 2;
    VC<Q> a[H], b[H];
#pragma unroll
    for (int p = 1; p <= H; ++p) { a[p - 1] = vadd(v[p], v[RAD - p]); b[p - 1] = vsub(v[p], v[RAD - p]); }
    VC<Q> s0 = v[0];
    const VC<Q> v0 = v[0];
#pragma unroll
    for (int p = 0; p < H; ++p) s0 = vadd(s0, a[p]);
    v[0] = s0;
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      VC<Q> A = v0, B;
#pragma unroll
      for (int p = 1; p <= H; ++p) {
        const int i = (p * q) % RAD;
        const Q c = qc<Q>(RxRoots<RAD>::c(i)), s = qc<Q>(RxRoots<RAD>::s(i));
        const double cl = RES ? kres<Q>(RxRoots<RAD>::c(i), RxRoots<RAD>::cl(i)) : 0.0;
        const double sl = RES ? kres<Q>(RxRoots<RAD>::s(i), RxRoots<RAD>::sl(i)) : 0.0;
        if (cl != 0.0) A = {qfma(a[p - 1].x, qc<Q>(cl), A.x), qfma(a[p - 1].y, qc<Q>(cl), A.y)};
        A = {qfma(a[p - 1].x, c, A.x), qfma(a[p - 1].y, c, A.y)};
        const Q sf = sl != 0.0 ? qc<Q>(sl) : s;
        if (p == 1) B = {qmul(b[0].x, sf), qmul(b[0].y, sf)};
        else B = {qfma(b[p - 1].x, sf, B.x), qfma(b[p - 1].y, sf, B.y)};
        if (sl != 0.0) B = {qfma(b[p - 1].x, s, B.x), qfma(b[p - 1].y, s, B.y)};
      }
      v[q] = vaddr(A, B);
      v[RAD - q] = vsubr(A, B);
    }
  }
};
template <typename Q> struct VB<Q, 3> : VBOdd<Q, 3, true> {};
template <typename Q> struct VB<Q, 5> : VBOdd<Q, 5, true> {};
template <typename Q> struct VB<Q, 7> : VBOdd<Q, 7, true> {};
// Butterfly of v, each output handed to emit(r, value) as soon as it is known:
// the outputs of the larger odd radices are not held next to their inputs.
template <typename Q, int RAD, typename F>
__device__ __forceinline__ void vb_emit(VC<Q>* v, F&& emit) {
  if constexpr (RAD == 11 || RAD == 13 || RAD > 16) {
    constexpr int H = (RAD - 1) / 2;
    VC<Q> s0 = v[0];
#pragma unroll
    for (int p = 1; p <= H; ++p) {
      const VC<Q> t = v[p];
      v[p] = vadd(t, v[RAD - p]);
      v[RAD - p] = vsub(t, v[RAD - p]);
      s0 = vadd(s0, v[p]);
    }
    emit(0, s0);
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      VC<Q> A = v[0], B;
#pragma unroll
      for (int p = 1; p <= H; ++p) {
        const int i = (p * q) % RAD;
        const Q c = qc<Q>(RxRoots<RAD>::c(i)), s = qc<Q>(RxRoots<RAD>::s(i));
        A = {qfma(v[p].x, c, A.x), qfma(v[p].y, c, A.y)};
        if (p == 1)
          B = {qmul(v[RAD - 1].x, s), qmul(v[RAD - 1].y, s)};
        else
          B = {qfma(v[RAD - p].x, s, B.x), qfma(v[RAD - p].y, s, B.y)};
      }
      emit(q, vaddr(A, B));
      emit(RAD - q, vsubr(A, B));
    }
  } else {
    VB<Q, RAD>::run(v);
#pragma unroll
    for (int r = 0; r < RAD; ++r) emit(r, v[r]);
  }
}

// The inner DFTs of a composite radix.
template <typename Q, int RAD, bool RES>
__device__ __forceinline__ void vb_inner(VC<Q>* v) {
  if constexpr (RAD % 2 == 1)
    VBOdd<Q, RAD, RES>::run(v);
  else
    VB<Q, RAD>::run(v);
}
template <typename Q, int R1, int R2, bool RES = true> struct VBComp {
  static __device__ __forceinline__ void run(VC<Q>* v) {
    constexpr int NN = R1 * R2;
    VC<Q> y[R2][R1];
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) {
      VC<Q> t[R1];
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) t[n1] = v[R2 * n1 + n2];
      vb_inner<Q, R1, RES>(t);
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) {
        const int e = (n2 * k1) % NN;
        if (e == 0)
          y[n2][k1] = t[k1];
        else if (4 * e == NN)
          y[n2][k1] = {t[k1].y, qmul(t[k1].x, qc<Q>(-1.0))};
        else if (2 * e == NN)
          y[n2][k1] = {qmul(t[k1].x, qc<Q>(-1.0)), qmul(t[k1].y, qc<Q>(-1.0))};
        else if constexpr (RES)
          y[n2][k1] = vrotc(t[k1], RxRoots<NN>::c(e), kres<Q>(RxRoots<NN>::c(e), RxRoots<NN>::cl(e)), RxRoots<NN>::s(e),
                            kres<Q>(RxRoots<NN>::s(e), RxRoots<NN>::sl(e)));
        else
          y[n2][k1] = vrotc(t[k1], RxRoots<NN>::c(e), 0.0, RxRoots<NN>::s(e), 0.0);
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      VC<Q> t[R2];
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) t[n2] = y[n2][k1];
      vb_inner<Q, R2, RES>(t);
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) v[k1 + R1 * k2] = t[k2];
    }
  }
};
template <typename Q> struct VB<Q, 6> : VBComp<Q, 2, 3> {};
template <typename Q> struct VB<Q, 9> : VBComp<Q, 3, 3> {};
template <typename Q> struct VB<Q, 10> : VBComp<Q, 2, 5> {};
template <typename Q> struct VB<Q, 12> : VBComp<Q, 4, 3> {};
template <typename Q> struct VB<Q, 14> : VBComp<Q, 2, 7> {};
// 15 without the residues is more exact than radices 3 and 5 in turn (255 points,
// forward and back: 0.9 of that error), and 255^3 f64 takes 757 us, 777 with them
template <typename Q> struct VB<Q, 15> : VBComp<Q, 3, 5, false> {};
template <typename Q> struct VB<Q, 16> : VBComp<Q, 4, 4> {};
}  // namespace pb
