// Fused pass with stage radices chosen at run time, for the lengths that have
// no compiled kernel of their own: C2C, R2C, C2R and the real-to-real kinds on
// any length whose prime factors are at most 31, and (BS) Bluestein's chirp-z
// form of the others: two transforms of the convolution length without leaving
// shared memory, the chirp and the kernel multiplied in as their first stages
// read the rows.  Bluestein passes of the generic kernel ran at 0.06-0.17 TB/s
// (DST-I 100 and 256, DCT-I 384); here 0.15-0.34, and 0.5-0.8 on DCT-II 257
// and DCT-IV 94.  C2C, R2C and C2R convolutions up to 1024 points keep the
// compiled kernel (mr_bs.cuh), which is 1.1-1.7 times faster than this one.
//
// Persistent CTAs walk the pass's tiles.  The lines of the next tile are
// copied to a staging area by cp.async while the current tile is transformed,
// so no registers hold data in flight.  Two sequences (f32) or one (f64) form
// a 16-byte vector, and a row buffer holds element i of all sequences of the
// tile in row i: a butterfly reads and writes whole vectors, one twiddle, one
// index computation and one packed instruction serve both sequences, and the
// transposed store (the fused pencil transpose) reads its runs of the
// destination's innermost axis directly.
//
//   first stage   staged lines -> butterfly -> rows (or, with `pre`, a pass
//                 that forms the rows: the real-to-real kinds' reordering and
//                 pre-twiddles, and lengths with a prime above 23)
//   middle stages rows -> rows, alternating between two buffers
//   last stage    C2C: butterfly outputs go to memory from registers; the
//                 other kinds read the finished rows back (the Hermitian
//                 split, post-twiddles) and store
//
// The real-to-real pre- and post-processing works on vectors too: DCT-II of 384
// f32 lines 1.00 -> 1.50 TB/s against the same code per value.
//
// Inverse transforms read their input in reversed index order, X^-1[k] =
// DFT(x[-q])[k], so only forward butterflies exist.
//
// What bounds it: global- and shared-memory latency and barriers at 16 warps per
// SM, not HBM (ncu: 255-point C2C f64 DRAM 24-30%, issue 33-36%, LSU data pipe
// 32-40%; 4096-point C2C f32 24-29%, 36-39%, 36-42%).
// Against the generic kernel on the same passes (B200, forward + inverse):
// 255^3 R2C f64 3.43 -> 0.76 ms, 4096^2 C2C f32 2.30 -> 0.40 ms; single
// transposed C2C passes run at 2.4-3.9 TB/s.  Measured choices: tiles of about
// 2000 points with 128 threads and four CTAs per SM beat tiles of twice the
// lines with 256 threads (384 points: 3.9 against 3.1 TB/s); 80 registers and
// more CTAs lose to 128 and fewer (3.8 against 3.9); loading straight into
// registers instead of staging loses (3.3); twiddles from shared memory beat
// global memory (2.8 against 2.4 TB/s at 1000 points) while they fit.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "pb_device.cuh"
#include "pb_launch.cuh"
#include "rx_fft.cuh"
#include "rx_plan.hpp"

namespace pb {

template <typename R>
using RxV = VC<typename Vec<R>::Q>;

template <int N>
__device__ __forceinline__ void rx_cp_async(void* s, const void* g) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(s);
  if constexpr (N == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(g) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(a), "l"(g), "n"(N) : "memory");
}
__device__ __forceinline__ void rx_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void rx_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// vector (re, im) of W sequences from scalars
__device__ __forceinline__ VC<Q2> rx_pack(float x0, float y0, float x1, float y1) {
  return VC<Q2>{Q2{make_float2(x0, x1)}, Q2{make_float2(y0, y1)}};
}

// Copies one tile's lines into the staging area (line l, element q at
// l*sl + q*sq).  E is the element type.  Lines run along the threads of a
// group; 16-byte copies where the source row and the staging row allow it.
template <typename E>
__device__ __forceinline__ void rx_stage_lines(E* S, const RxArgs& X, const TileAddr& ta) {
  constexpr int VF = 16 / (int)sizeof(E);
  const PassArgs& A = X.p;
  const RxGeom& g = X.g;
  const int nt = blockDim.x, tid = threadIdx.x, n = A.n_in;
  const E* in = reinterpret_cast<const E*>(A.in) + ta.src0;
  if (A.src_k_contig) {
    int lg = 31 - __clz(nt) - (31 - __clz(A.lines));
    if (lg < 3) lg = 3;
    const int tpl = 1 << lg, q0 = tid & (tpl - 1);
    const bool srow = (g.sl & (VF - 1)) == 0;
    for (int l = tid >> lg; l < ta.lines; l += nt >> lg) {
      const E* p = in + (long long)l * ta.srcb;
      E* s = S + l * g.sl;
      int q = q0;
      if (VF > 1 && srow && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        const int nv = n / VF;
        for (; q < nv; q += tpl) rx_cp_async<16>(s + q * VF, p + q * VF);
        q = nv * VF + q0;
      }
      for (; q < n; q += tpl) rx_cp_async<(int)sizeof(E)>(s + q, p + q);
    }
  } else {
    const int nc = (A.lines + VF - 1) / VF;  // chunks of VF adjacent lines per element
    const unsigned mc = fdiv_magic(nc);
    const int total = n * nc;
    for (int i = tid; i < total; i += nt) {
      const int q = (int)fdiv(i, nc, mc), l = (i - q * nc) * VF;
      const E* p = in + (long long)q * ta.srcq + (long long)l * ta.srcb;
      E* s = S + q * g.sq + l;
      if (VF > 1 && ta.srcb == 1 && l + VF <= ta.lines && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        rx_cp_async<16>(s, p);
      } else {
#pragma unroll
        for (int j = 0; j < VF; ++j)
          if (l + j < ta.lines) rx_cp_async<(int)sizeof(E)>(s + j, p + (long long)j * ta.srcb);
      }
    }
  }
  // the missing partner of an odd last line of a pair is zero
  if (A.kind != P_C2C && !(A.kind == P_R2R && A.in_complex) && (ta.lines & 1)) {
    E z;
    memset(&z, 0, sizeof(E));
    for (int q = tid; q < n; q += nt) S[ta.lines * g.sl + q * g.sq] = z;
  }
}

template <typename R, int KIND>
__device__ __forceinline__ void rx_stage(unsigned char* S, const RxArgs& X, const TileAddr& ta) {
  using C = typename Cx<R>::T;
  if (KIND == P_R2C || (KIND == P_R2R && !X.p.in_complex))
    rx_stage_lines<R>(reinterpret_cast<R*>(S), X, ta);
  else
    rx_stage_lines<C>(reinterpret_cast<C*>(S), X, ta);
}

// FFT input of vector g at staging offset o (= element * sq): C2C lines, or
// line pairs x + iy of real data.
template <typename R, int KIND>
__device__ __forceinline__ RxV<R> rx_fetch_at(const unsigned char* S, int base, int sl, int o) {
  using C = typename Cx<R>::T;
  if constexpr (KIND == P_C2C) {
    const C* p = reinterpret_cast<const C*>(S) + base + o;
    if constexpr (sizeof(R) == 4) {
      const C a = p[0], b = p[sl];
      return rx_pack(a.x, a.y, b.x, b.y);
    } else {
      const C a = p[0];
      return RxV<R>{a.x, a.y};
    }
  } else {
    const R* p = reinterpret_cast<const R*>(S) + base + o;
    if constexpr (sizeof(R) == 4)
      return rx_pack(p[0], p[sl], p[2 * sl], p[3 * sl]);
    else
      return RxV<R>{p[0], p[sl]};
  }
}

// C2R: Hermitian extension X + iY of the half spectra of lines 2s and 2s + 1
// at element q of the (index-reversed for a positive exponent) sequence.
template <typename R, bool BS>
__device__ __forceinline__ RxV<R> rx_fetch_c2r(const unsigned char* S, const RxArgs& X, int g, int q) {
  using C = typename Cx<R>::T;
  const PassArgs& A = X.p;
  const int m = A.m;
  if (!BS && A.inv && q != 0) q = m - q;
  const bool mirror = 2 * q > m;
  const int hq = mirror ? m - q : q;
  const bool edge = hq == 0 || 2 * hq == m;
  const R w = (A.pre_mode == W_HALF_INTERIOR && !edge) ? R(A.pre_factor) : R(1);
  const R sg = edge ? R(0) : (mirror ? -w : w);  // weight of the imaginary parts
  const int sl = X.g.sl;
  auto one = [&](int s, R& x, R& y) {
    const C* p = reinterpret_cast<const C*>(S) + (2 * s) * sl + hq * X.g.sq;
    const C a = p[0], b = p[sl];
    const R ay = edge ? R(0) : a.y * sg, by = edge ? R(0) : b.y * sg;
    x = a.x * w - by;
    y = ay + b.x * w;
  };
  if constexpr (sizeof(R) == 4) {
    R x0, y0, x1, y1;
    one(2 * g, x0, y0);
    one(2 * g + 1, x1, y1);
    return rx_pack(x0, y0, x1, y1);
  } else {
    R x0, y0;
    one(g, x0, y0);
    return RxV<R>{x0, y0};
  }
}

// lines of the staging area per vector
template <typename R, int KIND>
__device__ __forceinline__ constexpr int rx_lines_per_vec() {
  return Vec<R>::W * (KIND == P_C2C ? 1 : 2);
}

// Row of element i: padded by one row after every `pad` (magic mp).
__device__ __forceinline__ int rx_row(int i, int pad, unsigned mp) { return pad ? i + (int)fdiv(i, pad, mp) : i; }

// Stage 0 (no twiddles) from the staged lines.
template <typename R, int KIND, int RAD>
__device__ __forceinline__ void rx_first(const unsigned char* S, RxV<R>* out, const RxArgs& X) {
  using Q = typename Vec<R>::Q;
  const PassArgs& A = X.p;
  const int m = A.m, NB = m / RAD, lgG = X.g.lgG, P = X.g.P, total = NB << lgG;
  const int sl = X.g.sl, sq = X.g.sq;
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    const int g = it & ((1 << lgG) - 1), jb = it >> lgG;
    RxV<R> v[RAD];
    if constexpr (KIND == P_C2R) {
#pragma unroll
      for (int r = 0; r < RAD; ++r) v[r] = rx_fetch_c2r<R, false>(S, X, g, jb + r * NB);
    } else {
      // element jb + r*NB, or m - jb - r*NB (0 for element 0) when inverse
      const int base = g * rx_lines_per_vec<R, KIND>() * sl;
      const int b0 = (A.inv ? m - jb : jb) * sq, st = (A.inv ? -NB : NB) * sq;
      v[0] = rx_fetch_at<R, KIND>(S, base, sl, (A.inv && jb == 0) ? 0 : b0);
#pragma unroll
      for (int r = 1; r < RAD; ++r) v[r] = rx_fetch_at<R, KIND>(S, base, sl, b0 + r * st);
    }
    RxV<R>* o = out + jb * (RAD + (X.g.pad ? 1 : 0)) * P + g;
    vb_emit<Q, RAD>(v, [&](int r, const RxV<R>& x) { o[r * P] = x; });
  }
}

// Rows from the staged lines without a stage (lengths whose stage 0 is a
// direct-sum prime, and Bluestein passes, whose chirp carries the sign).
template <typename R, int KIND, bool BS>
__device__ __forceinline__ void rx_rows(const unsigned char* S, RxV<R>* out, const RxArgs& X) {
  const PassArgs& A = X.p;
  const int m = A.m, lgG = X.g.lgG, P = X.g.P, total = m << lgG;
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    const int g = it & ((1 << lgG) - 1), q = it >> lgG;
    if constexpr (KIND == P_C2R) {
      out[q * P + g] = rx_fetch_c2r<R, BS>(S, X, g, q);
    } else {
      const int e = (!BS && A.inv && q != 0) ? m - q : q;
      out[q * P + g] = rx_fetch_at<R, KIND>(S, g * rx_lines_per_vec<R, KIND>() * X.g.sl, X.g.sl, e * X.g.sq);
    }
  }
}

// Stockham stage: butterfly jb (k = jb mod NS) takes rows jb + r*len/RAD times
// W^{k r} and writes rows (jb - k)*RAD + k + r*NS.  The first stage of each of
// a Bluestein pass's two transforms (kMidMul, NS = 1) multiplies row i by
// vector i of `mul` (the chirp, rows from `lim` on are zero; the convolution
// kernel); its very last stage (kMidOut) reads the inverse transform off in
// reversed order, row i being output len - i, and multiplies the outputs
// below `lim` by the chirp.
enum { kMidPlain = 0, kMidMul = 1, kMidOut = 2 };
template <typename Q>
__device__ __forceinline__ VC<Q> rx_ldg(const VC<Q>* p) {
  const float4 f = __ldg(reinterpret_cast<const float4*>(p));
  VC<Q> r;
  *reinterpret_cast<float4*>(&r) = f;
  return r;
}
// ip, op: the padding of the rows read and written.
template <typename R, int RAD, int MODE>
__device__ __forceinline__ void rx_mid(const RxV<R>* in, RxV<R>* out, const RxArgs& X, int NS, const RxV<R>* tw,
                                       const RxV<R>* mul, int lim, int ip, int op) {
  using Q = typename Vec<R>::Q;
  const int len = X.g.len, NB = len / RAD, lgG = X.g.lgG, P = X.g.P, total = NB << lgG;
  const unsigned mNS = fdiv_magic(NS), mpad = X.g.pad ? fdiv_magic(X.g.pad) : 0;
  // NB (after stage 0) and NS (of later stages) are multiples of the padding
  const int rs = (NB + (ip ? NB / ip : 0)) * P, ws = (NS + (op && NS > 1 ? NS / op : 0)) * P;
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    const int g = it & ((1 << lgG) - 1), jb = it >> lgG;
    const int k = MODE == kMidMul ? 0 : jb - (int)fdiv(jb, NS, mNS) * NS;
    const RxV<R>* p = in + rx_row(jb, ip, mpad) * P + g;
    RxV<R> v[RAD];
    if constexpr (MODE == kMidMul) {
#pragma unroll
      for (int r = 0; r < RAD; ++r) {
        const int i = jb + r * NB;
        v[r] = i < lim ? vtw(p[r * rs], rx_ldg(mul + i)) : RxV<R>{qc<Q>(0.0), qc<Q>(0.0)};
      }
    } else {
#pragma unroll
      for (int r = 0; r < RAD; ++r) v[r] = p[r * rs];
      if (NS > 1) {
        const RxV<R>* t = tw + k;
#pragma unroll
        for (int r = 1; r < RAD; ++r) v[r] = vtw(v[r], t[(r - 1) * NS]);
      }
    }
    if constexpr (MODE == kMidOut) {
      vb_emit<Q, RAD>(v, [&](int r, const RxV<R>& x) {
        const int i = (jb - k) * RAD + k + r * NS, o = i == 0 ? 0 : len - i;
        if (o < lim) out[o * P + g] = vtw(x, rx_ldg(mul + o));
      });
    } else {
      RxV<R>* o = out + rx_row((jb - k) * RAD + k, op, mpad) * P + g;
      vb_emit<Q, RAD>(v, [&](int r, const RxV<R>& x) { o[r * ws] = x; });
    }
  }
}

// The same for a prime radix above kRxRegRadix: outputs h and RAD - h as
// direct sums over the pairs (p, RAD - p) read from the rows, so no butterfly
// sits in registers.  `roots` are the RAD-th roots.
template <typename R>
__device__ __forceinline__ void rx_mid_prime(const RxV<R>* in, RxV<R>* out, const RxArgs& X, int RAD, int NS,
                                             const RxV<R>* tw, const RxV<R>* roots, int ip, int op) {
  const int NB = X.g.len / RAD, lgG = X.g.lgG, P = X.g.P;
  const int H = (RAD - 1) / 2, total = (NB * (H + 1)) << lgG;
  const unsigned mNS = fdiv_magic(NS), mNB = fdiv_magic(NB), mpad = X.g.pad ? fdiv_magic(X.g.pad) : 0;
  const int rs = (NB + (ip ? NB / ip : 0)) * P, ws = (NS + (op && NS > 1 ? NS / op : 0)) * P;
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    const int g = it & ((1 << lgG) - 1), b = it >> lgG;
    const int h = (int)fdiv(b, NB, mNB), jb = b - h * NB;
    const int k = jb - (int)fdiv(jb, NS, mNS) * NS;
    const RxV<R>* p = in + rx_row(jb, ip, mpad) * P + g;
    const RxV<R> v0 = p[0];
    RxV<R> a = v0, c = {qc<typename Vec<R>::Q>(0.0), qc<typename Vec<R>::Q>(0.0)};
    int idx = 0;
    for (int i = 1; i <= H; ++i) {
      RxV<R> u = p[i * rs], w = p[(RAD - i) * rs];
      if (NS > 1) {
        u = vtw(u, tw[(i - 1) * NS + k]);
        w = vtw(w, tw[(RAD - i - 1) * NS + k]);
      }
      idx += h;
      if (idx >= RAD) idx -= RAD;
      const RxV<R> t = roots[idx];  // (cos, -sin)
      const RxV<R> s = vadd(u, w), d = vsub(u, w);
      a = {qfma(s.x, t.x, a.x), qfma(s.y, t.x, a.y)};
      c = {qfma(d.x, t.y, c.x), qfma(d.y, t.y, c.y)};
    }
    RxV<R>* o = out + rx_row((jb - k) * RAD + k, op, mpad) * P + g;
    // sum over d * (-i sin): a + i c with c carrying -sin
    if (h == 0) {
      o[0] = a;
    } else {
      o[h * ws] = vsubr(a, c);
      o[(RAD - h) * ws] = vaddr(a, c);
    }
  }
}

// Destination of one tile: address of output k of line 0 and the line stride.
struct RxDst {
  int mode;  // 0 transposed, 1 direct, 2 direct split across the ranks
  long long dst0;
  int dstb;
  const PieceAddr* prow;  // rows of the pieces, rebased to k = 0
  int np, nout;
  unsigned mnout;
  int lines;
  __device__ __forceinline__ const PieceAddr* piece(int k) const {
    return prow + (np > 1 ? (int)fdiv((unsigned)((k + 1) * np - 1), nout, mnout) : 0);
  }
  __device__ __forceinline__ long long at(int k, int l) const {
    if (mode == 1) return dst0 + (long long)l * dstb + k;
    const PieceAddr* r = piece(k);
    return mode == 0 ? r->rowbase + (long long)k * r->stride + l : r->rowbase + k + (long long)l * r->stride;
  }
};

// two adjacent complex values
__device__ __forceinline__ void rx_put2(float2* o, float2 a, float2 b, bool second) {
  if (second && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
    *reinterpret_cast<float4*>(o) = make_float4(a.x, a.y, b.x, b.y);
  } else {
    o[0] = a;
    if (second) o[1] = b;
  }
}

// Vector w of C2C results (output k of lines l .. l + W - 1) to memory.
template <typename R>
__device__ __forceinline__ void rx_put_c2c(typename Cx<R>::T* out, const RxDst& D, int k, int l, RxV<R> w) {
  if constexpr (sizeof(R) == 4) {
    const float2 a = make_float2(w.x.v.x, w.y.v.x), b = make_float2(w.x.v.y, w.y.v.y);
    const long long o = D.at(k, l);
    if (D.mode == 0) {
      rx_put2(out + o, a, b, l + 1 < D.lines);
    } else {
      out[o] = a;
      if (l + 1 < D.lines) out[D.at(k, l + 1)] = b;
    }
  } else {
    out[D.at(k, l)] = make_double2(w.x, w.y);
  }
}

// Work item of a store loop over n rows.  Lanes along the vectors of a row for
// a transposed store, whose row is adjacent in the destination, and for tiles
// of up to four vectors: a warp then covers at least eight adjacent elements
// of each line and reads whole rows.  Lanes along the rows otherwise.
constexpr int kRxWideRow = 2;  // log2 of the vectors
__device__ __forceinline__ void rx_item(int it, int lgG, int n, unsigned mn, bool tr, int& g, int& k) {
  if (tr || lgG <= kRxWideRow) {
    g = it & ((1 << lgG) - 1);
    k = it >> lgG;
  } else {
    g = (int)fdiv(it, n, mn);
    k = it - g * n;
  }
}

// Last stage of a C2C pass, stored from registers.
template <typename R, int RAD, bool TR>
__device__ __forceinline__ void rx_last(const RxV<R>* in, const RxArgs& X, const RxV<R>* tw, const RxDst& D) {
  using Q = typename Vec<R>::Q;
  using C = typename Cx<R>::T;
  const int NB = X.p.m / RAD, lgG = X.g.lgG, P = X.g.P, total = NB << lgG;
  const int pad = X.g.pad, rs = (NB + (pad ? NB / pad : 0)) * P;
  const unsigned mNB = fdiv_magic(NB), mpad = pad ? fdiv_magic(pad) : 0;
  const Q sc = qc<Q>(X.p.scale);
  C* out = reinterpret_cast<C*>(X.p.out);
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    int g, jb;
    rx_item(it, lgG, NB, mNB, TR, g, jb);
    const int l = g * Vec<R>::W;
    if (l >= D.lines) continue;
    const RxV<R>* p = in + rx_row(jb, pad, mpad) * P + g;
    RxV<R> v[RAD];
#pragma unroll
    for (int r = 0; r < RAD; ++r) v[r] = p[r * rs];
    const RxV<R>* t = tw + jb;
#pragma unroll
    for (int r = 1; r < RAD; ++r) v[r] = vtw(v[r], t[(r - 1) * NB]);
    if (!TR && D.mode == 1) {
      C* o = out + D.dst0 + (long long)l * D.dstb + jb;
      const bool two = sizeof(R) == 4 && l + 1 < D.lines;
      vb_emit<Q, RAD>(v, [&](int r, const RxV<R>& x) {
        const RxV<R> w = {qmul(x.x, sc), qmul(x.y, sc)};
        if constexpr (sizeof(R) == 4) {
          o[r * NB] = make_float2(w.x.v.x, w.y.v.x);
          if (two) o[D.dstb + r * NB] = make_float2(w.x.v.y, w.y.v.y);
        } else {
          o[r * NB] = make_double2(w.x, w.y);
        }
      });
    } else {
      vb_emit<Q, RAD>(v, [&](int r, const RxV<R>& x) {
        rx_put_c2c<R>(out, D, jb + r * NB, l, RxV<R>{qmul(x.x, sc), qmul(x.y, sc)});
      });
    }
  }
}

// Finished rows to memory: C2C.
template <typename R>
__device__ __forceinline__ void rx_store_c2c(const RxV<R>* rows, const RxArgs& X, const RxDst& D) {
  using Q = typename Vec<R>::Q;
  const int n = X.p.m, lgG = X.g.lgG, total = n << lgG;
  const unsigned mn = fdiv_magic(n);
  const Q sc = qc<Q>(X.p.scale);
  typename Cx<R>::T* out = reinterpret_cast<typename Cx<R>::T*>(X.p.out);
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    int g, k;
    rx_item(it, lgG, n, mn, D.mode == 0, g, k);
    const int l = g * Vec<R>::W;
    if (l >= D.lines) continue;
    const RxV<R> v = rows[k * X.g.P + g];
    rx_put_c2c<R>(out, D, k, l, RxV<R>{qmul(v.x, sc), qmul(v.y, sc)});
  }
}

// R2C: the half spectra of a sequence's two real lines.
template <typename R>
__device__ __forceinline__ void rx_store_r2c(const RxV<R>* rows, const RxArgs& X, const RxDst& D) {
  using Q = typename Vec<R>::Q;
  using C = typename Cx<R>::T;
  const PassArgs& A = X.p;
  const int n = A.m, h = n / 2 + 1, lgG = X.g.lgG, total = h << lgG, P = X.g.P;
  const unsigned mh = fdiv_magic(h);
  C* out = reinterpret_cast<C*>(A.out);
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    int g, k;
    rx_item(it, lgG, h, mh, D.mode == 0, g, k);
    const int l = g * 2 * Vec<R>::W;
    if (l >= D.lines) continue;
    const RxV<R> a = rows[k * P + g], b = rows[(k == 0 ? 0 : n - k) * P + g];
    double f = A.scale * 0.5;
    if (A.post_mode == W_HALF_INTERIOR && k != 0 && 2 * k != n) f *= A.post_factor;
    const Q q = qc<Q>(f);
    const Q xr = qmul(qadd(a.x, b.x), q), xi = qmul(qsub(a.y, b.y), q);
    const Q yr = qmul(qadd(a.y, b.y), q), yi = qmul(qsub(b.x, a.x), q);
    if constexpr (sizeof(R) == 4) {
      const C v[4] = {make_float2(xr.v.x, xi.v.x), make_float2(yr.v.x, yi.v.x), make_float2(xr.v.y, xi.v.y),
                      make_float2(yr.v.y, yi.v.y)};
      if (D.mode == 0) {
        C* o = out + D.at(k, l);
        rx_put2(o, v[0], v[1], l + 1 < D.lines);
        if (l + 2 < D.lines) rx_put2(o + 2, v[2], v[3], l + 3 < D.lines);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (l + j < D.lines) out[D.at(k, l + j)] = v[j];
      }
    } else {
      out[D.at(k, l)] = make_double2(xr, xi);
      if (l + 1 < D.lines) out[D.at(k, l + 1)] = make_double2(yr, yi);
    }
  }
}

// Output k of 2W adjacent real lines l ..
template <typename R>
__device__ __forceinline__ void rx_put_real(R* out, const RxDst& D, int k, int l, const R* v) {
  constexpr int NV = 2 * Vec<R>::W;
  if (D.mode == 0) {
    R* o = out + D.at(k, l);
    if (l + NV <= D.lines && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
      if constexpr (sizeof(R) == 4)
        *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
      else
        *reinterpret_cast<double2*>(o) = make_double2(v[0], v[1]);
    } else {
#pragma unroll
      for (int j = 0; j < NV; ++j)
        if (l + j < D.lines) o[j] = v[j];
    }
  } else {
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (l + j < D.lines) out[D.at(k, l + j)] = v[j];
  }
}

// C2R: the real and imaginary parts are the two real lines.
template <typename R>
__device__ __forceinline__ void rx_store_c2r(const RxV<R>* rows, const RxArgs& X, const RxDst& D) {
  const PassArgs& A = X.p;
  const int n = A.m, lgG = X.g.lgG, total = n << lgG;
  const unsigned mn = fdiv_magic(n);
  const R sc = R(A.scale);
  R* out = reinterpret_cast<R*>(A.out);
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    int g, k;
    rx_item(it, lgG, n, mn, D.mode == 0, g, k);
    const int l = g * 2 * Vec<R>::W;
    if (l >= D.lines) continue;
    const RxV<R> z = rows[k * X.g.P + g];
    R v[2 * Vec<R>::W];
    if constexpr (sizeof(R) == 4) {
      v[0] = z.x.v.x * sc;
      v[1] = z.y.v.x * sc;
      v[2] = z.x.v.y * sc;
      v[3] = z.y.v.y * sc;
    } else {
      v[0] = z.x * sc;
      v[1] = z.y * sc;
    }
    rx_put_real<R>(out, D, k, l, v);
  }
}

// ---- real-to-real kinds, a vector of sequences at a time.  A sequence is a
// pair p: two real lines 2p, 2p + 1 or the parts of complex line p; kinds IV and
// the odd-N forms of kinds I take one sequence per line or part.

__device__ __forceinline__ Q2 rx_q(float a, float b) { return Q2{make_float2(a, b)}; }
__device__ __forceinline__ float rx_lane(Q2 q, int w) { return w ? q.v.y : q.v.x; }
__device__ __forceinline__ double rx_lane(double q, int) { return q; }
template <typename Q>
__device__ __forceinline__ Q rx_neg(Q a) {
  return qmul(a, qc<Q>(-1.0));
}

// Part c of the pairs of vector g at element q of the staged lines.
template <typename R>
__device__ __forceinline__ typename Vec<R>::Q rx_part(const unsigned char* S, const RxArgs& X, int g, int c, int q) {
  using Q = typename Vec<R>::Q;
  const PassArgs& A = X.p;
  const int sl = X.g.sl, o = q * X.g.sq;
  const R* p = reinterpret_cast<const R*>(S);
  Q v;
  if constexpr (sizeof(R) == 4) {
    if (A.in_complex)
      v = rx_q(p[2 * (2 * g * sl + o) + c], p[2 * ((2 * g + 1) * sl + o) + c]);
    else
      v = rx_q(p[(4 * g + c) * sl + o], p[(4 * g + 2 + c) * sl + o]);
  } else {
    v = A.in_complex ? p[2 * (g * sl + o) + c] : p[(2 * g + c) * sl + o];
  }
  if (A.pre_mode != W_NONE && weight_hit(A.pre_mode, q, A.n)) v = qmul(v, qc<Q>(A.pre_factor));
  return v;
}
// Element q of the lines (or parts) that are the sequences of vector g, kinds
// with a sequence per line.
template <typename R>
__device__ __forceinline__ typename Vec<R>::Q rx_line(const unsigned char* S, const RxArgs& X, int g, int q) {
  using Q = typename Vec<R>::Q;
  const PassArgs& A = X.p;
  const int sl = X.g.sl, o = q * X.g.sq;
  const R* p = reinterpret_cast<const R*>(S);
  Q v;
  if constexpr (sizeof(R) == 4) {
    if (A.in_complex)
      v = rx_q(p[2 * (g * sl + o)], p[2 * (g * sl + o) + 1]);
    else
      v = rx_q(p[2 * g * sl + o], p[(2 * g + 1) * sl + o]);
  } else {
    v = A.in_complex ? p[2 * ((g >> 1) * sl + o) + (g & 1)] : p[g * sl + o];
  }
  if (A.pre_mode != W_NONE && weight_hit(A.pre_mode, q, A.n)) v = qmul(v, qc<Q>(A.pre_factor));
  return v;
}
template <typename R>
__device__ __forceinline__ RxV<R> rx_dup(typename Cx<R>::T w) {
  if constexpr (sizeof(R) == 4)
    return rx_pack(w.x, w.y, w.x, w.y);
  else
    return RxV<R>{w.x, w.y};
}

// FFT input rows of a real-to-real pass from the staged lines (the
// definitions of the generic kernel): Makhoul's reordering and pre-twiddle for
// kinds II / III, the half-length (odd n: zero-padded) form of kinds IV, the
// symmetric extensions of kinds I or their odd-N split.
template <typename R, int SUB, bool BS>
__device__ __forceinline__ void rx_pre_r2r(const unsigned char* S, RxV<R>* rows, const RxArgs& X) {
  using Q = typename Vec<R>::Q;
  using C = typename Cx<R>::T;
  const PassArgs& A = X.p;
  const int n = A.n, m = A.m, P = X.g.P, lgG = X.g.lgG, total = m << lgG;
  const C* aux0 = reinterpret_cast<const C*>(A.aux0);
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    const int g = it & ((1 << lgG) - 1), q = it >> lgG;
    RxV<R> z;
    if constexpr (SUB == S_DCT2 || SUB == S_DST2) {
      const int idx = (2 * q < n) ? 2 * q : 2 * (n - 1 - q) + 1;
      z = {rx_part<R>(S, X, g, 0, idx), rx_part<R>(S, X, g, 1, idx)};
      if (SUB == S_DST2 && (idx & 1)) z = {rx_neg(z.x), rx_neg(z.y)};
    } else if constexpr (SUB == S_DCT3 || SUB == S_DST3) {
      const int i0 = SUB == S_DST3 ? n - 1 - q : q;
      const Q ux = rx_part<R>(S, X, g, 0, i0), uy = rx_part<R>(S, X, g, 1, i0);
      Q vx = qc<Q>(0.0), vy = vx;
      if (q > 0) {
        const int i1 = SUB == S_DST3 ? q - 1 : n - q;
        vx = rx_part<R>(S, X, g, 0, i1);
        vy = rx_part<R>(S, X, g, 1, i1);
      }
      const RxV<R> w = rx_dup<R>(aux0[q]);
      const RxV<R> Vx = vtw(RxV<R>{ux, rx_neg(vx)}, w), Vy = vtw(RxV<R>{uy, rx_neg(vy)}, w);
      z = vsubr(Vx, Vy);  // Vx + i Vy
    } else if constexpr (SUB == S_DCT4 || SUB == S_DST4) {
      if ((n & 1) == 0) {
        const int i0 = 2 * q, i1 = n - 1 - 2 * q;
        const int j0 = SUB == S_DST4 ? n - 1 - i0 : i0, j1 = SUB == S_DST4 ? n - 1 - i1 : i1;
        z = vtw(RxV<R>{rx_line<R>(S, X, g, j0), rx_line<R>(S, X, g, j1)}, rx_dup<R>(aux0[q]));
      } else if (q < n) {
        const Q x = rx_line<R>(S, X, g, SUB == S_DST4 ? n - 1 - q : q);
        const RxV<R> w = rx_dup<R>(aux0[q]);
        z = {qmul(x, w.x), qmul(x, w.y)};
      } else {
        z = {qc<Q>(0.0), qc<Q>(0.0)};
      }
    } else if constexpr (SUB == S_DST1_ODD || SUB == S_DCT1_ODD) {
      // c = x_q -+ x_{m-q}, b = (-1)^q (x_q +- x_{m-q}): mr_r2r.cuh
      constexpr bool DST = SUB == S_DST1_ODD;
      Q x0 = qc<Q>(0.0), x1 = x0;
      if (!DST || q > 0) {
        x0 = rx_line<R>(S, X, g, DST ? q - 1 : q);
        x1 = rx_line<R>(S, X, g, DST ? m - q - 1 : m - q);
      }
      const Q sum = qadd(x0, x1), dif = qsub(x0, x1), bq = DST ? sum : dif;
      z = {DST ? dif : sum, (q & 1) ? rx_neg(bq) : bq};
    } else if constexpr (SUB == S_DCT1) {
      const int idx = q <= n - 1 ? q : m - q;
      z = {rx_part<R>(S, X, g, 0, idx), rx_part<R>(S, X, g, 1, idx)};
    } else if constexpr (SUB == S_DST1) {
      if (q == 0 || q == n + 1) {
        z = {qc<Q>(0.0), qc<Q>(0.0)};
      } else {
        const int idx = q <= n ? q - 1 : m - q - 1;
        z = {rx_part<R>(S, X, g, 0, idx), rx_part<R>(S, X, g, 1, idx)};
        if (q > n) z = {rx_neg(z.x), rx_neg(z.y)};
      }
    } else {  // DHT
      z = {rx_part<R>(S, X, g, 0, q), rx_part<R>(S, X, g, 1, q)};
    }
    rows[((!BS && A.inv && q != 0) ? m - q : q) * P + g] = z;
  }
}

// Outputs of a real-to-real pass from the finished rows.
template <typename R, int SUB>
__device__ __forceinline__ void rx_post_r2r(const RxV<R>* rows, const RxArgs& X, const RxDst& D) {
  using Q = typename Vec<R>::Q;
  using C = typename Cx<R>::T;
  const PassArgs& A = X.p;
  constexpr bool iv4 = r2r_seq_per_line(SUB);
  constexpr int W = Vec<R>::W;
  const int n = A.n, P = X.g.P, lgG = X.g.lgG, total = n << lgG;
  const unsigned mn = fdiv_magic(n);
  const Q h = qc<Q>(0.5);
  const C* aux0 = reinterpret_cast<const C*>(A.aux0);
  const C* aux1 = reinterpret_cast<const C*>(A.aux1);
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    int g, k;
    rx_item(it, lgG, n, mn, D.mode == 0, g, k);
    // first destination line of the vector: its values are parts 0 and 1 of W
    // pairs, or (kinds with a sequence per line) of W lines or parts
    const int l = iv4 ? (A.out_complex ? (g * W) >> 1 : g * W) : (A.out_complex ? g * W : 2 * g * W);
    if (l >= D.lines) continue;
    double fs = A.scale;
    if (A.post_mode != W_NONE && weight_hit(A.post_mode, k, n)) fs *= A.post_factor;
    const Q f = qc<Q>(fs);
    Q v0, v1 = qc<Q>(0.0);
    if constexpr (SUB == S_DCT2 || SUB == S_DST2 || SUB == S_DHT) {
      const int kk = SUB == S_DST2 ? n - 1 - k : k;
      const RxV<R> a = rows[kk * P + g], b = rows[(kk == 0 ? 0 : n - kk) * P + g];
      // twice the spectra of the pair's two parts
      const Q vx = qadd(a.x, b.x), vy = qsub(a.y, b.y), ux = qadd(a.y, b.y), uy = qsub(b.x, a.x);
      if constexpr (SUB == S_DHT) {
        v0 = qmul(qsub(vx, vy), h);
        v1 = qmul(qsub(ux, uy), h);
      } else {
        const RxV<R> w = rx_dup<R>(aux0[kk]);
        v0 = qfma(rx_neg(w.y), vy, qmul(w.x, vx));
        v1 = qfma(rx_neg(w.y), uy, qmul(w.x, ux));
      }
    } else if constexpr (SUB == S_DCT3 || SUB == S_DST3) {
      const RxV<R> z = rows[((k & 1) ? n - 1 - (k >> 1) : (k >> 1)) * P + g];
      const bool neg = SUB == S_DST3 && (k & 1);
      v0 = neg ? rx_neg(z.x) : z.x;
      v1 = neg ? rx_neg(z.y) : z.y;
    } else if constexpr (SUB == S_DST1_ODD || SUB == S_DCT1_ODD) {
      const int kk = SUB == S_DST1_ODD ? k + 1 : k;
      int i = (kk & 1) ? (kk + A.m) >> 1 : kk >> 1;
      if (SUB == S_DCT1_ODD && i == A.m) i = 0;
      const RxV<R> z = rows[i * P + g];
      if (SUB == S_DST1_ODD)
        v0 = (kk & 1) ? z.x : rx_neg(z.y);
      else
        v0 = (kk & 1) ? z.y : z.x;
    } else if constexpr (iv4) {
      if ((n & 1) == 0) {
        const int kk = (k & 1) ? (n - 1 - k) >> 1 : k >> 1;
        const RxV<R> z = vtw(rows[kk * P + g], rx_dup<R>(aux1[kk]));
        v0 = (k & 1) ? qmul(z.y, qc<Q>(-2.0)) : qmul(z.x, qc<Q>(2.0));
      } else {
        v0 = qmul(vtw(rows[k * P + g], rx_dup<R>(aux1[k])).x, qc<Q>(2.0));
      }
      if (SUB == S_DST4 && (k & 1)) v0 = rx_neg(v0);
    } else if constexpr (SUB == S_DCT1) {
      const RxV<R> z = rows[k * P + g];
      v0 = z.x;
      v1 = z.y;
    } else {  // DST-I
      const RxV<R> z = rows[(k + 1) * P + g];
      v0 = rx_neg(z.y);
      v1 = z.x;
    }
    v0 = qmul(v0, f);
    v1 = qmul(v1, f);
    R* out = reinterpret_cast<R*>(A.out);
    if constexpr (iv4) {
      // values of sequences gW ..: lines, or parts of a complex line
      if (A.out_complex) {
        R* o = out + 2 * D.at(k, l);
        if constexpr (W == 2)
          *reinterpret_cast<C*>(o) = mk<C, R>(rx_lane(v0, 0), rx_lane(v0, 1));
        else
          o[g & 1] = rx_lane(v0, 0);
      } else {
#pragma unroll
        for (int w = 0; w < W; ++w)
          if (l + w < D.lines) out[D.at(k, l + w)] = rx_lane(v0, w);
      }
    } else if (A.out_complex) {
      C* oc = reinterpret_cast<C*>(A.out);
      if constexpr (W == 2) {
        const C a = mk<C, R>(rx_lane(v0, 0), rx_lane(v1, 0)), b = mk<C, R>(rx_lane(v0, 1), rx_lane(v1, 1));
        const long long o = D.at(k, l);
        if (D.mode == 0) {
          rx_put2(reinterpret_cast<float2*>(oc + o), a, b, l + 1 < D.lines);
        } else {
          oc[o] = a;
          if (l + 1 < D.lines) oc[D.at(k, l + 1)] = b;
        }
      } else {
        oc[D.at(k, l)] = mk<C, R>(rx_lane(v0, 0), rx_lane(v1, 0));
      }
    } else {
      R v[2 * W];
#pragma unroll
      for (int w = 0; w < W; ++w) {
        v[2 * w] = rx_lane(v0, w);
        v[2 * w + 1] = rx_lane(v1, w);
      }
      rx_put_real<R>(out, D, k, l, v);
    }
  }
}

// radices of the convolution lengths, and of the other lengths
#define RX_RADICES_BS(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(12) X(14) X(15) X(16)
#define RX_RADICES(X) RX_RADICES_BS(X) X(11) X(13) X(17) X(19) X(23)
#define RX_SUBS(X)  \
  X(S_DST1_ODD) X(S_DCT1_ODD) \
  X(S_DCT1) X(S_DCT2) X(S_DCT3) X(S_DCT4) X(S_DST1) X(S_DST2) X(S_DST3) X(S_DST4) X(S_DHT)

// TR: the pass stores transposed (C2C only; the other kinds choose at run
// time).  BS: the m-point transform as a Bluestein convolution of length g.len.
template <typename R, int KIND, bool TR, bool BS>
__global__ void __launch_bounds__(kRxMaxThreads, 1) rx_kernel(const __grid_constant__ RxArgs X) {
  extern __shared__ __align__(16) unsigned char smem[];
  using V = RxV<R>;
  const PassArgs& A = X.p;
  const RxGeom& g = X.g;
  if (pb_rejected(A.gate)) return;
  long long tile = blockIdx.x;
  const long long step = gridDim.x, end = A.ntiles;
  if (tile >= end) return;
  const int tid = threadIdx.x, nt = blockDim.x;
  V* b0 = reinterpret_cast<V*>(smem);
  V* b1 = b0 + g.bufv;
  V* W = reinterpret_cast<V*>(smem + g.off_tw);
  unsigned char* S = smem + g.off_stage;
  TileAddr* desc = reinterpret_cast<TileAddr*>(smem + g.off_desc);     // tiles i, i+1, i+2
  PieceAddr* prow = reinterpret_cast<PieceAddr*>(desc + 3);            // pieces of tiles i, i+1
  const V* Wg = reinterpret_cast<const V*>(A.twiddle);
  const V* tw = g.tw_smem ? W : Wg;
  const TileAddr* tiles = reinterpret_cast<const TileAddr*>(A.tile_tab);
  const PieceAddr* pieces = reinterpret_cast<const PieceAddr*>(A.piece_tab);
  const int mode = KIND == P_C2C && TR ? 0 : A.dst_k_contig;
  const int np = mode == 1 ? 0 : A.npieces;
  RxDst D;
  D.mode = mode;
  D.np = np;
  D.nout = A.n_out;
  D.mnout = fdiv_magic(A.n_out);
  // this thread's piece starts at output index pst
  const long long pst = np > 0 ? (long long)A.n_out * tid / np : 0;

  if (tid == 0) {
    desc[0] = load_tile(tiles, tile);
    if (tile + step < end) desc[1] = load_tile(tiles, tile + step);
  }
  if (tid < np) prow[tid] = pieces[tile * np + tid];
  for (int i = tid; i < g.tw_smem; i += nt) W[i] = Wg[i];
  __syncthreads();
  pb_dependency_wait();  // the tables above belong to the plan; the data is read from here on
  rx_stage<R, KIND>(S, X, desc[0]);
  rx_cp_commit();

  int par = 0;
  for (int i = 0;; i = i == 2 ? 0 : i + 1, tile += step, par ^= kRxMaxPieces) {
    rx_cp_wait();
    PieceAddr* pr = prow + par;
    PieceAddr* pr_next = prow + (par ^ kRxMaxPieces);
    if (tid < np) {
      PieceAddr pa = pr[tid];
      pa.rowbase -= mode == 0 ? pst * pa.stride : pst;
      pr[tid] = pa;
    }
    __syncthreads();  // staged lines, descriptors and pieces in place; the previous tile's rows are free
    const TileAddr& ta = desc[i];
    const TileAddr& tn = desc[i == 2 ? 0 : i + 1];
    D.dst0 = ta.dst0;
    D.dstb = ta.dstb;
    D.lines = ta.lines;
    D.prow = pr;

    int s0 = 1, NS = 1;
    if constexpr (KIND == P_R2R) {
      s0 = 0;
      switch (A.sub) {
#define X_(u) \
  case u: rx_pre_r2r<R, u, BS>(S, b0, X); break;
        RX_SUBS(X_)
#undef X_
      }
    } else {
      if (BS || g.pre) {
        s0 = 0;
        rx_rows<R, KIND, BS>(S, b0, X);
      } else if constexpr (!BS) {
        NS = A.radix[0];
        switch (A.radix[0]) {
#define X_(r) \
  case r: rx_first<R, KIND, r>(S, b0, X); break;
          RX_RADICES(X_)
#undef X_
        }
      }
    }
    __syncthreads();
    const bool has_next = tile + step < end;
    if (!has_next) pb_allow_successor();
    if (has_next) {
      if (!g.alias) rx_stage<R, KIND>(S, X, tn);
      if (tid == 0 && tile + 2 * step < end) {
        TileAddr* d = desc + (i == 0 ? 2 : i - 1);
        const TileAddr* t = tiles + tile + 2 * step;
        rx_cp_async<16>(d, t);
        rx_cp_async<16>(reinterpret_cast<char*>(d) + 16, reinterpret_cast<const char*>(t) + 16);
      }
      if (tid < np) rx_cp_async<16>(pr_next + tid, pieces + (tile + step) * np + tid);
      rx_cp_commit();
    }
    V *in = b0, *out = b1;
    // a C2C pass ends with the stage that stores; the others finish the rows
    const bool fused =
        !BS && KIND == P_C2C && A.nstages > s0 && A.radix[A.nstages - 1] <= kRxRegRadix && A.nstages > 1;
    const int last = fused ? A.nstages - 1 : A.nstages;
    auto swap = [&] {
      __syncthreads();
      V* u = in;
      in = out;
      out = u;
    };
    if constexpr (BS) {
      const V* chirp = reinterpret_cast<const V*>(A.bs_chirp);
      const V* ker = reinterpret_cast<const V*>(A.bs_kernel);
      for (int f = 0; f < 2; ++f) {
        const V* mul = f ? ker : chirp;
        const int lim = f ? g.len : A.m;
        switch (A.radix[0]) {
#define X_(r) \
  case r: rx_mid<R, r, kMidMul>(in, out, X, 1, nullptr, mul, lim, 0, g.pad); break;
          RX_RADICES_BS(X_)
#undef X_
        }
        swap();
        NS = A.radix[0];
        for (int s = 1; s < A.nstages; ++s) {
          const int rad = A.radix[s];
          const V* t = tw + g.twoff[s];
          if (f == 1 && s == A.nstages - 1) {
            switch (rad) {
#define X_(r) \
  case r: rx_mid<R, r, kMidOut>(in, out, X, NS, t, chirp, A.m, g.pad, 0); break;
              RX_RADICES_BS(X_)
#undef X_
            }
          } else {
            switch (rad) {
#define X_(r) \
  case r: rx_mid<R, r, kMidPlain>(in, out, X, NS, t, nullptr, 0, g.pad, s + 1 < A.nstages ? g.pad : 0); break;
              RX_RADICES_BS(X_)
#undef X_
            }
          }
          swap();
          NS *= rad;
        }
      }
    } else {
      for (int s = s0; s < last; ++s) {
        const int rad = A.radix[s];
        const V* t = tw + g.twoff[s];
        // the stages' rows are padded; the rows formed before stage 0 and the
        // finished ones are not
        const int ip = s > 0 ? g.pad : 0, op = s + 1 < A.nstages ? g.pad : 0;
        switch (rad) {
#define X_(r) \
  case r: rx_mid<R, r, kMidPlain>(in, out, X, NS, t, nullptr, 0, ip, op); break;
          RX_RADICES(X_)
#undef X_
          default: rx_mid_prime<R>(in, out, X, rad, NS, t, t + (s > 0 ? (rad - 1) * NS : 0), ip, op); break;
        }
        swap();
        NS *= rad;
      }
    }
    if constexpr (KIND == P_C2C && BS) {
      rx_store_c2c<R>(in, X, D);
    } else if constexpr (KIND == P_C2C) {
      if (fused) {
        const V* t = tw + g.twoff[last];
        switch (A.radix[last]) {
#define X_(r) \
  case r: rx_last<R, r, TR>(in, X, t, D); break;
          RX_RADICES(X_)
#undef X_
        }
      } else {
        rx_store_c2c<R>(in, X, D);
      }
    } else if constexpr (KIND == P_R2C) {
      rx_store_r2c<R>(in, X, D);
    } else if constexpr (KIND == P_C2R) {
      rx_store_c2r<R>(in, X, D);
    } else {
      switch (A.sub) {
#define X_(u) \
  case u: rx_post_r2r<R, u>(in, X, D); break;
        RX_SUBS(X_)
#undef X_
      }
    }
    if (!has_next) break;
    if (g.alias) {
      __syncthreads();  // the staging area is the second row buffer
      rx_stage<R, KIND>(S, X, tn);
      rx_cp_commit();
    }
  }
}

// ---- in place: long C2C and R2C lines (g.ip), a butterfly per thread and stage.  A stage's rows are all read before any is written, so
// one row buffer serves and two CTAs fit on an SM; the lines go from memory
// into registers, and the other CTA computes meanwhile.

template <typename R, int KIND, int RAD>
__device__ __forceinline__ void rx_ip_first(const TileAddr& ta, RxV<R>* rows, const RxArgs& X) {
  using Q = typename Vec<R>::Q;
  using E = std::conditional_t<KIND == P_C2C, typename Cx<R>::T, R>;
  const PassArgs& A = X.p;
  const int m = A.m, NB = m / RAD, lgG = X.g.lgG, g = threadIdx.x & ((1 << lgG) - 1), jb = threadIdx.x >> lgG;
  if (jb >= NB) return;
  constexpr int NL = Vec<R>::W * (KIND == P_C2C ? 1 : 2);  // lines of a vector
  const long long sq = A.src_k_contig ? 1 : ta.srcq, lb = ta.srcb;
  const E* in = reinterpret_cast<const E*>(A.in) + ta.src0 + g * NL * lb;
  const int lines = ta.lines - g * NL;
  RxV<R> v[RAD];
#pragma unroll
  for (int r = 0; r < RAD; ++r) {
    // element jb + r*NB, or its mirror m - element when inverse
    const int q = jb + r * NB;
    const E* p = in + (long long)((A.inv && q != 0) ? m - q : q) * sq;
    E x[NL];
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      if (l < lines)
        x[l] = p[l * lb];
      else
        memset(&x[l], 0, sizeof(E));
    }
    if constexpr (KIND == P_C2C) {
      if constexpr (sizeof(R) == 4)
        v[r] = rx_pack(x[0].x, x[0].y, x[1].x, x[1].y);
      else
        v[r] = RxV<R>{x[0].x, x[0].y};
    } else {
      if constexpr (sizeof(R) == 4)
        v[r] = rx_pack(x[0], x[1], x[2], x[3]);
      else
        v[r] = RxV<R>{x[0], x[1]};
    }
  }
  RxV<R>* o = rows + (jb * (RAD + (X.g.pad ? 1 : 0)) << lgG) + g;
  vb_emit<Q, RAD>(v, [&](int r, const RxV<R>& x) { o[r << lgG] = x; });
}

template <typename R, int RAD>
__device__ __forceinline__ void rx_ip_mid(RxV<R>* rows, const RxArgs& X, int NS, const RxV<R>* tw, int op) {
  using Q = typename Vec<R>::Q;
  const int NB = X.g.len / RAD, pad = X.g.pad, lgG = X.g.lgG;
  const bool act = (int)threadIdx.x < NB << lgG;
  const int it = act ? threadIdx.x : 0;  // idle threads read along, and write nothing
  const int g = it & ((1 << lgG) - 1), jb = it >> lgG;
  const unsigned mpad = pad ? fdiv_magic(pad) : 0;
  const int rs = (NB + (pad ? NB / pad : 0)) << lgG, ws = (NS + (op ? NS / op : 0)) << lgG;
  const int k = jb - (int)fdiv(jb, NS, fdiv_magic(NS)) * NS;
  RxV<R> v[RAD];
  const RxV<R>* p = rows + (rx_row(jb, pad, mpad) << lgG) + g;
#pragma unroll
  for (int r = 0; r < RAD; ++r) v[r] = p[r * rs];
  const RxV<R>* t = tw + k;
#pragma unroll
  for (int r = 1; r < RAD; ++r) v[r] = vtw(v[r], t[(r - 1) * NS]);
  // the block barrier, its own in each radix's code: a shared one would keep the
  // values of every radix alive across it
  asm volatile("bar.sync 0; // radix %0" ::"n"(RAD) : "memory");
  if (act) {
    RxV<R>* o = rows + (rx_row((jb - k) * RAD + k, op, mpad) << lgG) + g;
    vb_emit<Q, RAD>(v, [&](int r, const RxV<R>& x) { o[r * ws] = x; });
  }
}

template <typename R, int KIND, bool TR>
__global__ void __launch_bounds__(kRxMaxThreads, 1) rx_inplace_kernel(const __grid_constant__ RxArgs X) {
  extern __shared__ __align__(16) unsigned char smem[];
  using V = RxV<R>;
  const PassArgs& A = X.p;
  const RxGeom& g = X.g;
  if (pb_rejected(A.gate)) return;
  long long tile = blockIdx.x;
  const long long step = gridDim.x, end = A.ntiles;
  if (tile >= end) return;
  const int tid = threadIdx.x, nt = blockDim.x;
  V* rows = reinterpret_cast<V*>(smem);
  V* W = reinterpret_cast<V*>(smem + g.off_tw);
  TileAddr* desc = reinterpret_cast<TileAddr*>(smem + g.off_desc);  // tiles i, i+1
  PieceAddr* prow = reinterpret_cast<PieceAddr*>(desc + 3);         // pieces of tiles i, i+1
  const V* Wg = reinterpret_cast<const V*>(A.twiddle);
  const V* tw = g.tw_smem ? W : Wg;
  const TileAddr* tiles = reinterpret_cast<const TileAddr*>(A.tile_tab);
  const PieceAddr* pieces = reinterpret_cast<const PieceAddr*>(A.piece_tab);
  const int mode = KIND == P_C2C && TR ? 0 : A.dst_k_contig;
  const int np = mode == 1 ? 0 : A.npieces;
  RxDst D;
  D.mode = mode;
  D.np = np;
  D.nout = A.n_out;
  D.mnout = fdiv_magic(A.n_out);
  const long long pst = np > 0 ? (long long)A.n_out * tid / np : 0;
  if (tid == 0) desc[0] = load_tile(tiles, tile);
  if (tid < np) prow[tid] = pieces[tile * np + tid];
  for (int i = tid; i < g.tw_smem; i += nt) W[i] = Wg[i];
  pb_dependency_wait();  // the tables above belong to the plan; the data is read from here on

  for (int par = 0;; par ^= 1, tile += step) {
    rx_cp_wait();
    PieceAddr* pr = prow + par * kRxMaxPieces;
    if (tid < np) {
      PieceAddr pa = pr[tid];
      pa.rowbase -= mode == 0 ? pst * pa.stride : pst;
      pr[tid] = pa;
    }
    __syncthreads();  // descriptor, pieces and twiddles in place; the previous tile's rows are free
    const TileAddr& ta = desc[par];
    D.dst0 = ta.dst0;
    D.dstb = ta.dstb;
    D.lines = ta.lines;
    D.prow = pr;
    const bool has_next = tile + step < end;
    if (has_next) {
      if (tid == 0) {
        char* d = reinterpret_cast<char*>(desc + (par ^ 1));
        const char* t = reinterpret_cast<const char*>(tiles + tile + step);
        rx_cp_async<16>(d, t);
        rx_cp_async<16>(d + 16, t + 16);
      }
      if (tid < np) rx_cp_async<16>(prow + (par ^ 1) * kRxMaxPieces + tid, pieces + (tile + step) * np + tid);
      rx_cp_commit();
    } else {
      pb_allow_successor();
    }
    switch (A.radix[0]) {
#define X_(r) \
  case r: rx_ip_first<R, KIND, r>(ta, rows, X); break;
      RX_RADICES(X_)
#undef X_
    }
    __syncthreads();
    int NS = A.radix[0];
    const int last = KIND == P_C2C ? A.nstages - 1 : A.nstages;
    for (int s = 1; s < last; ++s) {
      const V* t = tw + g.twoff[s];
      const int op = s + 1 < A.nstages ? g.pad : 0;
      switch (A.radix[s]) {
#define X_(r) \
  case r: rx_ip_mid<R, r>(rows, X, NS, t, op); break;
        RX_RADICES(X_)
#undef X_
      }
      __syncthreads();
      NS *= A.radix[s];
    }
    if constexpr (KIND == P_C2C) {
      const V* t = tw + g.twoff[last];
      switch (A.radix[last]) {
#define X_(r) \
  case r: rx_last<R, r, TR>(rows, X, t, D); break;
        RX_RADICES(X_)
#undef X_
      }
    } else {
      rx_store_r2c<R>(rows, X, D);
    }
    if (!has_next) break;
  }
}

}  // namespace pb
