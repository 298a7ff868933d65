// FFT plans, twiddle tables and launchers for the x-pencil kernels.
#include <math.h>
#include <stdlib.h>
#include <string.h>
#include <map>
#include <mutex>
#include <utility>

#include <cudaTypedefs.h>

#include "fft.cuh"
#include "ops.cuh"

namespace dftgpu {

namespace {
struct PlanEntry {
  int nst;
  int radix[FFT_MAX_STAGES];
  void *tw;
};
std::map<std::pair<int, int>, PlanEntry> g_plans;   // (n, sizeof(T), + 1 for the small variant) -> plan
std::mutex g_plan_mu;

// FP64 operations per element of a radix-R stage without / with twiddles (the
// powers of two carry theirs inside the butterfly, the others multiply first)
struct RadixCost { int r; double first, rest; };
constexpr RadixCost kRadix[] = { { 16, 9.25, 12 }, { 15, 11.2, 14.9 }, { 12, 8, 11.7 }, { 10, 9.2, 12.8 }, { 9, 9.8, 13.3 },
                                 { 8, 6.5, 9 }, { 6, 6, 9.3 }, { 5, 7.2, 10.4 }, { 4, 4, 6 }, { 3, 4, 6.7 }, { 2, 2, 3 } };
constexpr double kStageCost = 6;   // a pass through shared memory, in the same unit: the fewest stages first

// The cheapest product of radices, the untwiddled first stage included in the
// choice; a small charge on the largest radix prefers 8 x 8 to 16 x 4 (as many
// butterflies in either stage).  Depth-first over at most FFT_MAX_STAGES stages.
void search(int m, int cap, int depth, double cost, int big, int *cur, double *best, int *radix, int *nst) {
  if (m == 1) {
    if (cost + 0.1 * big < *best) {
      *best = cost + 0.1 * big;
      *nst = depth;
      for (int i = 0; i < depth; i++) radix[i] = cur[i];
    }
    return;
  }
  if (depth == FFT_MAX_STAGES || cost >= *best) return;
  for (const RadixCost &k : kRadix)
    if (m % k.r == 0 && k.r <= cap) {
      cur[depth] = k.r;
      search(m / k.r, cap, depth + 1, cost + (depth ? k.rest : k.first) + kStageCost, big > k.r ? big : k.r, cur, best, radix, nst);
    }
}

int factorize_fp64(int n, int cap, int *radix, int *nst) {
  int cur[FFT_MAX_STAGES];
  double best = 1e9;
  *nst = 0;
  search(n, cap, 0, 0.0, 0, cur, &best, radix, nst);
  return best < 1e9 ? DFTGPU_OK : DFTGPU_ERR_SIZE;
}
// FP32 is not bound by operations: few stages, 16 or 8 first (its first stage
// has no twiddles): two steps of 240^3 12.0 ms as 16, 15 and 13.0 as 15, 16;
// one propagation of 120^3 84 us as 8, 15 and 87 as 15, 8, with rms errors of
// 2.17e-7 and 2.29e-7.  A 2 left alone beside a 16: 8 x 4 has
// as many butterflies in both stages (288^3 1173 / 1245 as 16, 9, 2; twenty
// steps of 64^3, z half 32, 2391 / 2475).  A 16 alone stays one stage: 4 x 4
// takes 3 of 24 us off a propagation of 16^3, at 3 % more rms error.
int factorize_fp32(int n, int *radix, int *nst) {
  int m = n, k = 0, a = 0, b = 0, c = 0;
  while (m % 2 == 0) { m /= 2; a++; }
  while (m % 3 == 0) { m /= 3; b++; }
  while (m % 5 == 0) { m /= 5; c++; }
  if (m != 1) return DFTGPU_ERR_SIZE;
  // radix 16 for the power of two, one 8 / 4 / 2 for its rest; 15 = 3 x 5 and
  // 9 = 3 x 3 for the odd part; a rest of 2 or 4 merged with a rest of 3 (6,
  // 12) or 2 with a 5 (10), a 2 that stays alone beside a 16 as 8 x 4
  while (a >= 4) { radix[k++] = 16; a -= 4; }
  const int n16 = k;
  int r2 = 1 << a;
  if (r2 == 8 && n16 == 0) { radix[k++] = 8; r2 = 1; }
  while (b >= 1 && c >= 1) { radix[k++] = 15; b--; c--; }
  while (b >= 2) { radix[k++] = 9; b -= 2; }
  if ((r2 == 2 || r2 == 4) && b == 1) { radix[k++] = 3 * r2; r2 = 1; b = 0; }
  else if (r2 == 2 && c >= 1) { radix[k++] = 10; r2 = 1; c--; }
  if (r2 == 2 && n16 > 0) { radix[n16 - 1] = 8; r2 = 4; }
  if (r2 > 1) radix[k++] = r2;
  if (b == 1) radix[k++] = 3;
  while (c-- > 0) radix[k++] = 5;
  if (k > FFT_MAX_STAGES) return DFTGPU_ERR_SIZE;
  *nst = k;
  return DFTGPU_OK;
}
}  // namespace

int fft_radices(int n, int prec, bool small, int *radix, int *nst) {
  *nst = 0;
  if (n == 1) return DFTGPU_OK;
  return prec == DFTGPU_FP64 ? factorize_fp64(n, small ? 5 : 16, radix, nst) : factorize_fp32(n, radix, nst);
}

template <typename T> int get_plan(int n, FftPlan<T> *plan, bool small) {
  typedef typename cplx_t<T>::type C;
  if (n < 1 || n > FFT_MAX_LINE) {
    set_error(DFTGPU_ERR_SIZE, "FFT length %d outside [1, %d]", n, FFT_MAX_LINE);
    return DFTGPU_ERR_SIZE;
  }
  if (sizeof(T) == 4) small = false;   // one FP32 variant
  std::lock_guard<std::mutex> lock(g_plan_mu);
  auto key = std::make_pair(n, (int) sizeof(T) + small);
  auto it = g_plans.find(key);
  if (it == g_plans.end()) {
    PlanEntry e;
    if (fft_radices(n, sizeof(T) == 8 ? DFTGPU_FP64 : DFTGPU_FP32, small, e.radix, &e.nst) != DFTGPU_OK) {
      set_error(DFTGPU_ERR_SIZE, "FFT length %d is not of the form 2^a 3^b 5^c", n);
      return DFTGPU_ERR_SIZE;
    }
    const size_t nt = plan_table<T>(n);
    C *h = (C *) malloc(sizeof(C) * nt);
    for (int t = 0; t < n; t++) {
      // reduce the angle to [-pi, pi] and evaluate in long double, round once
      long tt = (t <= n / 2) ? t : (long) t - n;
      long double ang = -2.0L * 3.14159265358979323846264338327950288L * (long double) tt / (long double) n;
      const long double cr = cosl(ang), ci = sinl(ang);
      h[t].x = (T) cr;
      h[t].y = (T) ci;
      if constexpr (sizeof(T) == 8) h[n + t] = cos_tan((double) cr, (double) ci);
      if (sizeof(T) == 4) {
        // of the float pairs within one ulp of (cos, sin), take the one
        // closest to the unit circle: independent rounding leaves |w|^2 off 1
        // by up to 1.2e-7, a fixed pattern that biases the norm
        const float fx = (float) cr, fy = (float) ci;
        const float xs[2] = { fx, nextafterf(fx, cr > (long double) fx ? 2.f : -2.f) };
        const float ys[2] = { fy, nextafterf(fy, ci > (long double) fy ? 2.f : -2.f) };
        long double best = -1.0L;
        for (float x : xs)
          for (float y : ys) {
            const long double dev = fabsl((long double) x * x + (long double) y * y - 1.0L);
            if (best < 0 || dev < best) { best = dev; h[t].x = (T) x; h[t].y = (T) y; }
          }
      }
    }
    void *d = nullptr;
    cudaError_t err = cudaMalloc(&d, sizeof(C) * nt);
    if (err == cudaSuccess) err = cudaMemcpy(d, h, sizeof(C) * nt, cudaMemcpyHostToDevice);
    // the table is complete on the device before any stream (also a
    // non-blocking one: a caller's, or a parallel branch) reads it
    if (err == cudaSuccess) err = cudaDeviceSynchronize();
    free(h);
    if (err != cudaSuccess) {
      set_error(DFTGPU_ERR_CUDA, "twiddle table: %s", cudaGetErrorString(err));
      return DFTGPU_ERR_CUDA;
    }
    e.tw = d;
    it = g_plans.emplace(key, e).first;
  }
  plan->n = n;
  plan->nst = it->second.nst;
  for (int i = 0; i < it->second.nst; i++) plan->radix[i] = it->second.radix[i];
  plan->tw = (const C *) it->second.tw;
  return DFTGPU_OK;
}

template int get_plan<float>(int, FftPlan<float> *, bool);
template int get_plan<double>(int, FftPlan<double> *, bool);

const DevLimits &dev_limits() {
  static DevLimits known[64];
  static std::mutex mu;
  static const DevLimits none = { -1, 0, 0 };
  int dev = 0, smem = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return none;
  std::lock_guard<std::mutex> lock(mu);
  DevLimits &d = known[dev];
  if (!d.smem && cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) {
    d.id = dev;
    d.sms = sms;
    d.smem = (size_t) smem;
  }
  return d.smem ? d : none;
}

// About 16 values per thread (one butterfly of radix 16) at 128 threads in
// FP64 and 256 in FP32; fewer lines per CTA while the launch would not give
// every SM four CTAs, down to runs of 64 bytes where a side is strided and in
// FP64 to one full warp of butterflies (an FP64 warp instruction takes its 16 clocks
// of the SM's pipe whatever the number of its active lanes).  Fewer also while
// `ctas` of them do not fit into an SM's shared memory: three for the line and
// convolution passes, as many as their registers allow, two for the kinetic
// pass.  Full potential, us, one / two / three CTAs at least: FP32 288 x 256 x
// 256 3795 / 2901 / 2900, 320^3 9043 / 7333 / 6875, FP64 288^3 52360 / 44870 /
// 42910 (four: FP64 216^3 22080 against 21430); FP32 propagation, two / three
// in the kinetic pass: 288 x 256 x 256 405 / 424, 320^3 1355 / 1379.
int choose_tile(int n, int big, int na, int nb, size_t cplx_bytes, int nbufs, bool strided, size_t table, int ctas, TileShape *t) {
  const DevLimits &dev = dev_limits();
  const size_t hard = dev.smem;
  const int most = cplx_bytes == 16 ? 2560 : 5120;
  int least = strided ? (int) (64 / cplx_bytes) : 1;
  while (cplx_bytes == 16 && least < 32 && least * n < 32 * big) least *= 2;   // a full warp of the largest butterflies
  int B = 32;
  while (B > 1 && (B * n > most || B >= 2 * nb)) B >>= 1;
  if (B < least) B = least;
  while (B > 1 && B >= 2 * nb) B >>= 1;
  while (B > least && (size_t) na * ((nb + B - 1) / B) < (size_t) 4 * dev.sms) B >>= 1;
  auto need = [&](int b) { return (size_t) nbufs * b * Tile::pitch(n) * cplx_bytes + table + (table ? (size_t) b * cplx_bytes : 0); };
  while (B > least && ctas * (need(B) + 1024) > hard + 1024) B >>= 1;   // 1 KB of an SM's is the system's for each
  while (B > 1 && need(B) > hard) B >>= 1;
  if (need(B) > hard) {
    set_error(DFTGPU_ERR_SIZE, "FFT tile for n=%d does not fit in shared memory", n);
    return DFTGPU_ERR_SIZE;
  }
  t->B = B;
  t->logB = 0;
  while ((1 << t->logB) < B) t->logB++;
  int th = (B * n / (cplx_bytes == 16 ? 8 : 4) + 31) / 32 * 32;
  const int cap = cplx_bytes == 16 && B * n <= most ? 128 : 256;
  t->threads = th < 64 ? 64 : th > cap ? cap : th;
  t->smem = need(B);
  return DFTGPU_OK;
}

bool fused_zy_off() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("DFTGPU_FUSED_ZY");
    v = (e && e[0] == '1') ? 0 : 1;
  }
  return v == 1;
}

bool prefetch_ahead_on() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("DFTGPU_PREFETCH_AHEAD");
    v = (e && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

bool factorised_propagation() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("DFTGPU_FACTORISED_PROP");
    v = (e && e[0] == '1') ? 1 : 0;
  }
  return v == 1;
}

bool march_on() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("DFTGPU_MARCH");
    v = (e && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

namespace {
int g_tma = -1;
}
bool tma_on() {
  if (g_tma < 0) {
    const char *e = getenv("DFTGPU_TMA");
    g_tma = (e && e[0] == '0') ? 0 : 1;
  }
  return g_tma == 1;
}
void tma_disable() { g_tma = 0; }

namespace {
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
}

int encode_spec_map(CUtensorMap *map, const void *spec, int nx, int ny, int rows) {
  if (!g_encode) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
      cudaGetLastError();
      set_error(DFTGPU_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
      return DFTGPU_ERR_CUDA;
    }
    g_encode = (PFN_cuTensorMapEncodeTiled_v12000) fn;
  }
  // [rows][nx][ny] of 8-byte elements; box {16 y, 1 x, rows}: 128-byte rows
  const cuuint64_t dims[3] = { (cuuint64_t) ny, (cuuint64_t) nx, (cuuint64_t) rows };
  const cuuint64_t strides[2] = { (cuuint64_t) ny * 8, (cuuint64_t) nx * ny * 8 };
  const cuuint32_t box[3] = { 16, 1, (cuuint32_t) rows }, estr[3] = { 1, 1, 1 };
  const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, const_cast<void *>(spec), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error(DFTGPU_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for a %d x %d x %d spectrum", (int) r, rows, nx, ny);
    return DFTGPU_ERR_CUDA;
  }
  return DFTGPU_OK;
}

bool generic_fft_only() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("DFTGPU_GENERIC_FFT");
    v = (e && e[0] == '1') ? 1 : 0;
  }
  return v == 1;
}

namespace {

double xconv_bytes(const XConvArgs<float> &A, int kxh, int kyh) {
  const double spec = (double) A.nkz * A.nx * A.ny * sizeof(float2);
  double bytes = spec * A.nin;
  for (int o = 0; o < A.nout; o++) bytes += spec * (A.out[o].accumulate ? 2 : 1);
  const float *seen[XC_MAX_TERMS];
  int nseen = 0;
  for (int t = 0; t < XC_MAX_TERMS; t++) {
    const float *k = A.term[t].ker;
    if (!k || A.term[t].kind == KER_UNIT) continue;
    bool dup = false;
    for (int s = 0; s < nseen; s++) dup |= seen[s] == k;
    if (!dup) { seen[nseen++] = k; bytes += (double) A.nkz * kxh * kyh * sizeof(float); }
  }
  return bytes;
}

template <int N> int fast_xconv(const XConvArgs<float> &A) {
  constexpr int B = ff::Shape<N>::B;
  if (A.ny % B || (A.ny / 2) % B || A.nin > 8 || A.nout > 8) return -1;
  ff::XArgsF F;
  memset(&F, 0, sizeof(F));
  F.nx = A.nx; F.ny = A.ny; F.kxh = A.nx / 2 + 1; F.kyh = A.ny / 2 + 1;
  F.nin = A.nin; F.nout = A.nout;
  for (int i = 0; i < A.nin; i++) F.src[i] = A.src[i];
  int multi = -1, nt = 0;
  for (int o = 0; o < A.nout; o++) {
    F.dst[o] = A.out[o].dst;
    F.acc_out[o] = A.out[o].accumulate;
    F.t0[o] = A.out[o].t0;
    F.nterm[o] = A.out[o].nt;
    if (A.out[o].nt > 1) {
      if (multi >= 0) return -1;   // at most one output accumulated in registers
      multi = o;
    }
    if (A.out[o].nt < 1) return -1;
    nt = A.out[o].t0 + A.out[o].nt > nt ? A.out[o].t0 + A.out[o].nt : nt;
  }
  if (nt > 16) return -1;
  F.nslice = 0;
  for (int t = 0; t < nt; t++) {
    F.kind[t] = A.term[t].kind; F.in[t] = A.term[t].in; F.coef[t] = A.term[t].coef;
    F.slot[t] = -1;
    if (A.term[t].kind == KER_UNIT) continue;
    for (int s = 0; s < F.nslice; s++)
      if (F.slice_src[s] == A.term[t].ker) F.slot[t] = s;
    if (F.slot[t] < 0) {
      if (F.nslice == 8) return -1;
      F.slice_src[F.nslice] = A.term[t].ker;
      F.slot[t] = F.nslice++;
    }
  }
  FftPlan<float> p;
  DFT_TRY(get_plan<float>(N, &p));
  F.split = A.split;
  const int smem = ff::xconv_smem<N>(F.split ? 1 : F.nslice);
  // request exactly the dynamic shared memory this launch needs (the kernel
  // also has static shared memory, so the opt-in maximum itself is not valid)
  // MODE 2: one output summing every term; 1: mixed with one multi-term output; 0: single-term outputs
  const int mode = (A.nout == 1 && multi == 0) ? 2 : (multi >= 0 ? 1 : 0);
  static int granted[3] = { 48 * 1024, 48 * 1024, 48 * 1024 };
  if (smem > granted[mode]) {
    if (mode == 2) DFT_CUDA(cudaFuncSetAttribute(ff::xconv_kernel<N, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    else if (mode == 1) DFT_CUDA(cudaFuncSetAttribute(ff::xconv_kernel<N, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    else DFT_CUDA(cudaFuncSetAttribute(ff::xconv_kernel<N, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    granted[mode] = smem;
  }
  ProfScope prof("fft_x_conv", xconv_bytes(A, F.kxh, F.kyh));
  const dim3 grid(A.ny / B, A.nkz, F.split ? A.nout : 1);
  if (mode == 2) launch_pdl(ff::xconv_kernel<N, 2>, grid, 256, smem, rt().stream, p.tw, F, multi);
  else if (mode == 1) launch_pdl(ff::xconv_kernel<N, 1>, grid, 256, smem, rt().stream, p.tw, F, multi);
  else launch_pdl(ff::xconv_kernel<N, 0>, grid, 256, smem, rt().stream, p.tw, F, multi);
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

template <int N> int fast_xkinetic(const KinArgs<float> &A) {
  constexpr int B = ff::Shape<N>::B;
  if (A.ny % B) return -1;
  FftPlan<float> p;
  DFT_TRY(get_plan<float>(N, &p));
  ProfScope prof("fft_x_kinetic", 2.0 * A.nx * A.ny * A.nkz * sizeof(float2));
  auto k = A.cn ? ff::xkinetic_kernel<N, true> : ff::xkinetic_kernel<N, false>;
  launch_pdl(k, dim3(A.ny / B, A.nkz), 256, 0, rt().stream,
      p.tw, A.data, A.ny, A.nz, A.kz0i, make_float2((float) A.cdt.x, (float) A.cdt.y), (float) A.inv_n, (float) A.dkx,
      (float) A.dky, (float) A.dkz, (float) A.kx0, (float) A.ky0, (float) A.kz0, (float) A.h);
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

}  // namespace

template <typename T> int launch_xconv(XConvArgs<T> &A) {
  typedef typename cplx_t<T>::type C;
  // outputs of one term and one input each are independent: one CTA each, but
  // in FP32 only while the inputs fit into L2 together (above that a CTA that
  // takes the inputs one after the other, the next one prefetched, is 1 % of
  // the 256^3 potential faster)
  A.split = A.nout > 1 && A.nin == A.nout &&
            (sizeof(T) == 8 || (double) A.nin * A.nkz * A.nx * A.ny * sizeof(C) <= kBatchBytes);
  for (int o = 0; o < A.nout; o++) A.split &= A.out[o].nt == 1 && A.term[A.out[o].t0].in == o;
  if constexpr (std::is_same<T, float>::value) {
    if (!generic_fft_only()) {
      int rc = -1;
      switch (A.nx) {
        case 64: rc = fast_xconv<64>(A); break;
        case 128: rc = fast_xconv<128>(A); break;
        case 256: rc = fast_xconv<256>(A); break;
        case 512: rc = fast_xconv<512>(A); break;
        case 96: rc = fast_xconv<96>(A); break;
        case 192: rc = fast_xconv<192>(A); break;
        case 384: rc = fast_xconv<384>(A); break;
        default: break;
      }
      if (rc >= 0) return rc;
    }
  }
  DFT_TRY(get_plan<T>(A.nx, &A.plan, small_pass(A.nx, A.nkz, A.ny)));
  A.kxh = A.nx / 2 + 1;
  A.kyh = A.ny / 2 + 1;
  A.acc_buf = 0;
  for (int o = 0; o < A.nout; o++) A.acc_buf |= A.out[o].nt != 1;
  double bytes = 0.0;
  {
    const double spec = (double) A.nkz * A.nx * A.ny * sizeof(C);
    bytes = spec * A.nin;
    for (int o = 0; o < A.nout; o++) bytes += spec * (A.out[o].accumulate ? 2 : 1);
    const T *seen[XC_MAX_TERMS];
    int nseen = 0;
    for (int t = 0; t < XC_MAX_TERMS; t++) {
      const T *k = A.term[t].ker;
      if (!k || A.term[t].kind == KER_UNIT) continue;
      bool dup = false;
      for (int s = 0; s < nseen; s++) dup |= seen[s] == k;
      if (!dup) { seen[nseen++] = k; bytes += (double) A.nkz * A.kxh * A.kyh * sizeof(T); }
    }
  }
  ProfScope prof("fft_x_conv", bytes);
  if (A.nx == 1) {
    launch_pdl(xconv_point_kernel<T>, (A.nkz * A.ny + 127) / 128, 128, 0, rt().stream, A);
    DFT_CHECK_LAUNCH();
    return DFTGPU_OK;
  }
  TileShape t;
  DFT_TRY(choose_tile(A.nx, max_radix(A.plan), A.split ? A.nkz * A.nout : A.nkz, A.ny, sizeof(C), xconv_bufs(A.plan.nst, A.acc_buf), true, 0, 3, &t));
  A.B = t.B;
  A.logB = t.logB;
  DFT_TRY(smem_opt_in<SmemOptIn<XConvArgs<T> (*)()>>(xconv_kernel<T>));
  launch_pdl(xconv_kernel<T>, dim3((A.ny + t.B - 1) / t.B, A.nkz, A.split ? A.nout : 1), t.threads, t.smem, rt().stream, A);
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

template <typename T> int launch_xkinetic(KinArgs<T> &A) {
  typedef typename cplx_t<T>::type C;
  if constexpr (std::is_same<T, float>::value) {
    if (!generic_fft_only()) {
      int rc = -1;
      switch (A.nx) {
        case 64: rc = fast_xkinetic<64>(A); break;
        case 128: rc = fast_xkinetic<128>(A); break;
        case 256: rc = fast_xkinetic<256>(A); break;
        case 512: rc = fast_xkinetic<512>(A); break;
        case 96: rc = fast_xkinetic<96>(A); break;
        case 192: rc = fast_xkinetic<192>(A); break;
        case 384: rc = fast_xkinetic<384>(A); break;
        default: break;
      }
      if (rc >= 0) return rc;
    }
  }
  DFT_TRY(get_plan<T>(A.nx, &A.plan, small_pass(A.nx, A.nkz, A.ny)));
  ProfScope prof("fft_x_kinetic", 2.0 * A.nx * A.ny * A.nkz * sizeof(C));
  return launch_generic_xkinetic<T>(A, rt().stream);
}

template int launch_xconv<float>(XConvArgs<float> &);
template int launch_xconv<double>(XConvArgs<double> &);
template int launch_xkinetic<float>(KinArgs<float> &);
template int launch_xkinetic<double>(KinArgs<double> &);

// ------------------------------------------------------------------ fused z + y passes
namespace {

int *g_zy_fault = nullptr;   // set by a kernel whose wait on an asynchronous copy gave up

template <int NY, int NZ, int CL, bool FWD, class Kern, class... Args>
int launch_zy_cluster(Kern kfn, int nx, Args... args) {
  typedef ff::ZYPlane<NY, NZ, CL> Z;
  static bool attr_done = false;
  if (!attr_done) {
    DFT_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, Z::SMEM));
    attr_done = true;
  }
  if (!async_fault_flag()) return DFTGPU_ERR_CUDA;
  FftPlan<float> pz, p2, py;
  DFT_TRY(get_plan<float>(Z::NZC, &pz));
  DFT_TRY(get_plan<float>(NZ, &p2));
  DFT_TRY(get_plan<float>(NY, &py));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CL, nx);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = Z::SMEM;
  cfg.stream = rt().stream;
  cudaLaunchAttribute at[1];
  memset(at, 0, sizeof(at));
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kfn, (const float2 *) pz.tw, (const float2 *) p2.tw,
                                           (const float2 *) py.tw, args..., nx, g_zy_fault);
  if (e != cudaSuccess) {
    cudaFuncAttributes fa = {};
    cudaFuncGetAttributes(&fa, kfn);
    set_error(DFTGPU_ERR_CUDA, "fused %s pass %dx%d (cluster %d, %d B shared, nx %d): %s; function: %d regs, "
              "max dynamic shared %d B", FWD ? "zy r2c" : "yz c2r", NY, NZ, CL, Z::SMEM, nx, cudaGetErrorString(e),
              fa.numRegs, fa.maxDynamicSharedSizeBytes);
    return DFTGPU_ERR_CUDA;
  }
  return DFTGPU_OK;
}

bool fused_shape(int ny, int nz) {
  return !generic_fft_only() && !fused_zy_off() && ny == nz && (ny == 128 || ny == 256);
}

}  // namespace

int *async_fault_flag() {
  if (!g_zy_fault) {
    if (cudaMalloc(&g_zy_fault, sizeof(int)) != cudaSuccess || cudaMemset(g_zy_fault, 0, sizeof(int)) != cudaSuccess) {
      cudaGetLastError();
      g_zy_fault = nullptr;
      set_error(DFTGPU_ERR_CUDA, "asynchronous-copy fault flag");
      return nullptr;
    }
  }
  return g_zy_fault;
}

int fused_zy_fault() {
  if (!g_zy_fault) return DFTGPU_OK;
  int v = 0;
  DFT_CUDA(cudaMemcpy(&v, g_zy_fault, sizeof(int), cudaMemcpyDeviceToHost));
  if (v) {
    cudaMemset(g_zy_fault, 0, sizeof(int));
    set_error(DFTGPU_ERR_CUDA, "a wait on an asynchronous copy (TMA or fused plane pass) timed out");
    return DFTGPU_ERR_CUDA;
  }
  return DFTGPU_OK;
}

int launch_zy_r2c(const RealPairLoad<float> &ld, float2 *spec, int nx, int ny, int nz) {
  if (!fused_shape(ny, nz)) return -1;
  ProfScope prof("fft_zy_r2c", (double) nx * ny * nz * 4.0 + (double) nx * ny * (nz / 2 + 1) * 8.0);
  if (ny == 128) return launch_zy_cluster<128, 128, 2, true>(ff::zy_r2c_kernel<128, 128, 2>, nx, ld.f, spec);
  return launch_zy_cluster<256, 256, 8, true>(ff::zy_r2c_kernel<256, 256, 8>, nx, ld.f, spec);
}

int launch_yz_c2r(const float2 *spec, const RealPairStore<float> &st, int nx, int ny, int nz) {
  if (!fused_shape(ny, nz)) return -1;
  ProfScope prof("fft_yz_c2r", (double) nx * ny * nz * 4.0 + (double) nx * ny * (nz / 2 + 1) * 8.0);
  if (ny == 128) return launch_zy_cluster<128, 128, 2, false>(ff::yz_c2r_kernel<128, 128, 2>, nx, spec, st.f, st.scale);
  return launch_zy_cluster<256, 256, 8, false>(ff::yz_c2r_kernel<256, 256, 8>, nx, spec, st.f, st.scale);
}

}  // namespace dftgpu
