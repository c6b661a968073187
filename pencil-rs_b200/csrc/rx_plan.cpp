// Stage radices, tile geometry and twiddle tables of the runtime-radix pass
// kernel.
#include "rx_plan.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

namespace pb {

std::vector<int> rx_radices(int m) {
  static const int radices[] = {31, 29, 23, 19, 17, 16, 15, 14, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  if (m < 2) return {};
  // fewest stages, then the smallest largest radix, over the divisors of m
  constexpr int kInf = 1 << 20;
  std::vector<int> st(m + 1, kInf), mx(m + 1, 0), ch(m + 1, 0);
  st[1] = 0;
  for (int d = 2; d <= m; ++d) {
    if (m % d) continue;
    for (int r : radices) {
      if (d % r || st[d / r] >= kInf) continue;
      const int s = st[d / r] + 1, x = std::max(mx[d / r], r);
      if (s < st[d] || (s == st[d] && x < mx[d])) {
        st[d] = s;
        mx[d] = x;
        ch[d] = r;
      }
    }
  }
  std::vector<int> out;
  if (st[m] >= kInf || st[m] > kRxMaxStages) return out;
  for (int d = m; d > 1; d /= ch[d]) out.push_back(ch[d]);
  std::sort(out.begin(), out.end());
  // stage 0: a direct-sum prime (it has no twiddles there), else an odd radix,
  // whose outputs fall on distinct shared-memory banks
  size_t first = 0;
  for (size_t i = 0; i < out.size(); ++i)
    if (out[i] & 1) {
      first = i;
      break;
    }
  if (out.back() > kRxRegRadix) first = out.size() - 1;
  std::swap(out[0], out[first]);
  return out;
}

template <typename R>
std::vector<R> rx_twiddles(const std::vector<int>& radix, const R* roots) {
  long long m = 1;
  for (int r : radix) m *= r;
  std::vector<R> t;
  auto put = [&](long long q) {
    for (int c = 0; c < 2; ++c)
      for (size_t w = 0; w < 8 / sizeof(R); ++w) t.push_back(roots[2 * q + c]);
  };
  long long ns = 1;
  for (size_t s = 0; s < radix.size(); ++s) {
    const int rad = radix[s];
    if (s > 0)
      for (int r = 1; r < rad; ++r)
        for (long long k = 0; k < ns; ++k) put(k * r * (m / (ns * rad)));
    if (rad > kRxRegRadix)
      for (int i = 0; i < rad; ++i) put(i * (m / rad));
    ns *= rad;
  }
  return t;
}
template std::vector<float> rx_twiddles(const std::vector<int>&, const float*);
template std::vector<double> rx_twiddles(const std::vector<int>&, const double*);

// Real lines per FFT sequence, doubled: C2C 2 (one line), line pairs 4, the
// kinds with a sequence per line 2 (real data) or 1 (complex data: a sequence per component).
static int lines_x2(const PassArgs& A) {
  if (A.kind == P_C2C) return 2;
  if (A.kind == P_R2C || A.kind == P_C2R) return 4;
  const bool iv4 = r2r_seq_per_line(A.sub);
  if (A.in_complex) return iv4 ? 1 : 2;
  return iv4 ? 2 : 4;
}

bool rx_geometry(const PassArgs& A, int real_bytes, int max_smem, RxGeom* g) {
  std::memset(g, 0, sizeof(*g));
  g->max_smem = max_smem;
  g->len = A.bs_m2 ? A.bs_m2 : A.m;
  const int W = real_bytes == 4 ? 2 : 1;
  const int nseq = A.lines * 2 / lines_x2(A);
  int G = std::max(1, (nseq + W - 1) / W);
  while ((1 << g->lgG) < G) ++g->lgG;
  G = 1 << g->lgG;
  // an odd row pitch lets lanes that walk along the rows (stores to lines
  // contiguous in the destination from tiles of more than four vectors) hit
  // distinct banks; the other stores read whole rows and need none
  g->P = (A.dst_k_contig != 0 && G > 4) ? G + 1 : G;
  g->pre = (A.kind == P_R2R || A.bs_m2 || A.radix[0] > kRxRegRadix) ? 1 : 0;
  // stage 0 writes rows at multiples of its radix: with an even one and less
  // than eight vectors to a row, one row of padding after every radix[0] rows
  // puts them on distinct banks (4096 = 16*16*16 points: half of the
  // wavefronts were conflicts)
  g->pad = (A.radix[0] % 2 == 0 && G < 8 && A.nstages > 1) ? A.radix[0] : 0;
  g->bufv = (g->len + (g->pad ? g->len / g->pad : 0)) * g->P;
  long long tw = 0, ns = 1;
  for (int s = 0; s < A.nstages; ++s) {
    g->twoff[s] = (int)tw;
    if (s > 0) tw += (A.radix[s] - 1) * ns;
    if (A.radix[s] > kRxRegRadix) tw += A.radix[s];
    ns *= A.radix[s];
  }
  const int eb = real_bytes * (A.in_complex ? 2 : 1);
  int stage_elems;
  if (A.src_k_contig) {
    // line stride: lanes cover the G vectors of a row and consecutive
    // elements; the stride modulo 8 spreads them over the banks
    int want = G >= 8 ? 1 : 8 / G;
    int align = 1;  // keep 16-byte copies possible
    while (align * eb < 16) align *= 2;
    want = std::max(want, align);
    g->sl = A.n_in;
    while (g->sl % 8 != want % 8) ++g->sl;
    g->sq = 1;
    stage_elems = A.lines * g->sl;
  } else {
    const int align = std::max(1, 16 / eb);
    g->sl = 1;
    g->sq = (A.lines + align - 1) / align * align;
    stage_elems = A.n_in * g->sq;
  }
  const int stage_bytes = (int)((((long long)stage_elems * eb) + 15) & ~15LL);
  const int buf_bytes = g->bufv * 16;
  const int tail = 3 * (int)sizeof(TileAddr) + 2 * kRxMaxPieces * (int)sizeof(PieceAddr);
  // twiddles in shared memory unless they would take the room of the tile
  // itself; staging of its own unless only the aliased form fits
  const int tw_bytes = (int)tw * 16;
  auto fits = [&](bool tws, bool alias) {
    const long long second = alias ? std::max(buf_bytes, stage_bytes) : buf_bytes;
    const long long b = (long long)buf_bytes + second + (tws ? tw_bytes : 0) + (alias ? 0 : stage_bytes) + tail;
    if (b > max_smem) return false;
    g->tw_smem = tws ? (int)tw : 0;
    g->alias = alias ? 1 : 0;
    g->off_tw = buf_bytes + (int)second;
    g->off_stage = alias ? buf_bytes : g->off_tw + (tws ? tw_bytes : 0);
    g->off_desc = g->off_tw + (tws ? tw_bytes : 0) + (alias ? 0 : stage_bytes);
    g->smem = (int)b;
    return true;
  };
  bool ok = fits(true, false) || fits(false, false) || fits(true, true) || fits(false, true);
  // Long lines, whose tile leaves one CTA per SM: C2C and R2C passes run in
  // place, one butterfly per thread and stage.  With one vector per row two
  // CTAs fit and one loads while the other computes (4096 points, direct: 1.9 ->
  // 3.3 TB/s); a transposed C2C store takes two vectors, whose 32-byte runs are
  // worth more than the second CTA (2.62 against 2.20 TB/s f32, 2.84 against
  // 2.17 f64; direct 2.87 against 3.28).
  const int wide = A.kind == P_C2C && A.dst_k_contig == 0 ? 2 : 1;
  int items = 0;
  for (int s = 0; s < A.nstages; ++s) items = std::max(items, g->len / A.radix[s] << g->lgG);
  if ((A.kind == P_C2C || A.kind == P_R2C) && !g->pre && A.nstages > 1 && G <= wide && G == g->P && items <= kRxMaxThreads &&
      (!ok || 2 * (g->smem + 1024) > max_smem)) {
    const int half = (max_smem - 1024) / 2;
    const int room = half - buf_bytes - tail;
    g->ip = 1;
    g->alias = 0;
    g->tw_smem = tw_bytes <= room ? (int)tw : 0;
    g->off_tw = buf_bytes;
    g->off_stage = g->off_desc = buf_bytes + g->tw_smem * 16;
    g->smem = g->off_desc + tail;
    g->threads = std::max(128, (items + 31) / 32 * 32);
    return g->smem <= max_smem;
  }
  if (!ok) return false;
  const long long elems = (long long)nseq * g->len;
  g->threads = elems > 6 * 1024 / (3 - W) ? 512 : elems > 2600 / (3 - W) ? 256 : 128;
  return true;
}

bool rx_choose(PassArgs& A, int real_bytes, int max_smem, long long max_chunk, long long total_lines, int sms) {
  const int len = A.bs_m2 ? A.bs_m2 : A.m;
  const std::vector<int> rad = rx_radices(len);
  if (rad.empty()) return false;
  A.nstages = (int)rad.size();
  for (int s = 0; s < A.nstages; ++s) A.radix[s] = rad[s];
  const int W = real_bytes == 4 ? 2 : 1;
  const int x2 = lines_x2(A);
  // kinds with a sequence per line form a pair of lines from two sequences
  const bool iv4 = A.kind == P_R2R && r2r_seq_per_line(A.sub);
  const int min_seq = std::max(W, iv4 ? 2 : 1);
  // sequences per tile: a power of two, about 2048 points in f32 and 1024 in
  // f64 (more CTAs per SM beat longer tiles), at least four sequences in f32
  // so that a transposed store writes whole 32-byte sectors
  int nseq = min_seq;
  const long long target = real_bytes == 4 ? 2304 : 1152;
  while (nseq < 128 && (long long)(2 * nseq) * len <= target) nseq *= 2;
  if (real_bytes == 4 && nseq < 4) nseq = 4;
  if (real_bytes == 8 && nseq < 2) nseq = 2;
  // no wider than the runs of lines, and enough tiles to fill the device
  while (nseq > min_seq && (long long)(nseq / 2) * x2 / 2 >= max_chunk) nseq /= 2;
  while (nseq > std::max(min_seq, 4) && total_lines * 2 / ((long long)nseq * x2) < 2LL * sms) nseq /= 2;
  RxGeom g;
  for (;;) {
    A.lines = std::max(1, nseq * x2 / 2);
    if (rx_geometry(A, real_bytes, max_smem, &g) && (!g.alias || nseq == min_seq)) return true;
    if (nseq <= min_seq) return false;
    nseq /= 2;
  }
}

}  // namespace pb

namespace pb {

template <int KIND, bool BS>
cudaError_t rx_launch_kind(const RxArgs& X, int real_bytes, int grid, cudaStream_t stream);
template <int KIND, bool BS>
int rx_occupancy_kind(const RxArgs& X, int real_bytes);
#define RX_DECL(K, B)                                                                                \
  template <>                                                                                        \
  cudaError_t rx_launch_kind<K, B>(const RxArgs& X, int real_bytes, int grid, cudaStream_t stream);  \
  template <>                                                                                        \
  int rx_occupancy_kind<K, B>(const RxArgs& X, int real_bytes);
RX_DECL(1, false)
RX_DECL(2, false)
RX_DECL(3, false)
RX_DECL(4, false)
RX_DECL(1, true)
RX_DECL(2, true)
RX_DECL(3, true)
RX_DECL(4, true)
#undef RX_DECL

// The current device's shared memory per block, looked up once per device.
static int smem_limit() {
  static std::atomic<int> known[64];
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 227 * 1024;
  optin = known[dev].load(std::memory_order_relaxed);
  if (optin > 0) return optin;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || optin <= 0)
    return 227 * 1024;
  known[dev].store(optin, std::memory_order_relaxed);
  return optin;
}

cudaError_t launch_rx(const PassArgs& A, int real_bytes, cudaStream_t stream) {
  if (A.ntiles <= 0) return cudaSuccess;
  RxArgs X;
  X.p = A;
  if (!rx_geometry(A, real_bytes, smem_limit(), &X.g)) return cudaErrorInvalidValue;
  long long grid = A.grid_ctas > 0 ? A.grid_ctas : A.ntiles;
  if (grid > A.ntiles) grid = A.ntiles;
  switch (A.kind) {
    case P_C2C:
      return A.bs_m2 ? rx_launch_kind<P_C2C, true>(X, real_bytes, (int)grid, stream)
                     : rx_launch_kind<P_C2C, false>(X, real_bytes, (int)grid, stream);
    case P_R2C:
      return A.bs_m2 ? rx_launch_kind<P_R2C, true>(X, real_bytes, (int)grid, stream)
                     : rx_launch_kind<P_R2C, false>(X, real_bytes, (int)grid, stream);
    case P_C2R:
      return A.bs_m2 ? rx_launch_kind<P_C2R, true>(X, real_bytes, (int)grid, stream)
                     : rx_launch_kind<P_C2R, false>(X, real_bytes, (int)grid, stream);
    case P_R2R:
      return A.bs_m2 ? rx_launch_kind<P_R2R, true>(X, real_bytes, (int)grid, stream)
                     : rx_launch_kind<P_R2R, false>(X, real_bytes, (int)grid, stream);
  }
  return cudaErrorInvalidValue;
}

int rx_occupancy(const PassArgs& A, int real_bytes) {
  RxArgs X;
  X.p = A;
  if (!rx_geometry(A, real_bytes, smem_limit(), &X.g)) return 1;
  switch (A.kind) {
    case P_C2C: return A.bs_m2 ? rx_occupancy_kind<P_C2C, true>(X, real_bytes) : rx_occupancy_kind<P_C2C, false>(X, real_bytes);
    case P_R2C: return A.bs_m2 ? rx_occupancy_kind<P_R2C, true>(X, real_bytes) : rx_occupancy_kind<P_R2C, false>(X, real_bytes);
    case P_C2R: return A.bs_m2 ? rx_occupancy_kind<P_C2R, true>(X, real_bytes) : rx_occupancy_kind<P_C2R, false>(X, real_bytes);
    default: return A.bs_m2 ? rx_occupancy_kind<P_R2R, true>(X, real_bytes) : rx_occupancy_kind<P_R2R, false>(X, real_bytes);
  }
}

}  // namespace pb
