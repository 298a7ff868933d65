// Elementwise launch, FP64 reductions and 3-D transform sequences shared by
// the grid and OT translation units.
#pragma once

#include "fft.cuh"

namespace dftgpu {

// grid-stride elementwise launch of a device lambda f(i), i < n
template <class F> __global__ void each_kernel(size_t n, F f) {
  pdl_wait();
  for (size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t) gridDim.x * blockDim.x) f(i);
}

// f(0..n-1), independent of one another, spread round-robin over the work
// stream and the auxiliary streams with event fork / join, so that a CUDA
// graph captured from the work stream gets them as parallel branches.  Runs
// on the work stream alone while the profiler is on (per-launch timings), and
// on the branch it is in when called from one.  With more than two items a
// branch the launches are ordinary: CTAs that wait for their own branch keep
// room from the other's.  FP32 propagation, us, programmatic / ordinary:
// 512 x 512 x 128 (7 items) 699 / 662, 512 x 512 x 256 (14) 1351 / 1333, 384^3
// (12) 1503 / 1501; 240^3 (3) 457 / 467, 192^3 (2) 148 / 150.
inline bool &inside_par() {
  static thread_local bool v = false;
  return v;
}
template <class F> int par_for(int n, F f) {
  cudaStream_t *aux;
  cudaEvent_t *ev;
  const int ns = prof_on() || n < 2 || inside_par() ? 1 : par_streams(&aux, &ev);
  if (ns < 2) {
    for (int i = 0; i < n; i++) DFT_TRY(f(i));
    return DFTGPU_OK;
  }
  const cudaStream_t main = rt().stream;
  const int use = ns < n ? ns : n;
  DFT_CUDA(cudaEventRecord(ev[0], main));
  for (int k = 0; k < use - 1; k++) DFT_CUDA(cudaStreamWaitEvent(aux[k], ev[0], 0));
  int rc = DFTGPU_OK;
  inside_par() = true;
  ordinary_launches() = n > 2 * use;
  for (int i = 0; i < n && rc == DFTGPU_OK; i++) {
    rt().stream = i % use == 0 ? main : aux[i % use - 1];
    rc = f(i);
  }
  ordinary_launches() = false;
  inside_par() = false;
  rt().stream = main;
  for (int k = 0; k < use - 1; k++) {
    DFT_CUDA(cudaEventRecord(ev[k + 1], aux[k]));
    DFT_CUDA(cudaStreamWaitEvent(main, ev[k + 1], 0));
  }
  return rc;
}

// bytes: algorithmic bytes the lambda reads and writes (0 if not stated)
template <class F> int launch_each(size_t n, F f, double bytes = 0.0, const char *name = "pointwise") {
  if (n == 0) return DFTGPU_OK;
  int blocks = (int) ((n + 255) / 256);
  int cap = rt().num_sms * 8;
  if (blocks > cap) blocks = cap;
  ProfScope prof(name, bytes);
  launch_pdl(each_kernel<F>, blocks, 256, 0, rt().stream, n, f);
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

// The (x, y) rows of an [nx][ny][nz] grid, threads along z, a row of more
// than 256 values in equal segments of one CTA each: the lambda gets
// f(x, y, z, i) with i the linear index, no index division.  A row's segments
// are neighbours in the grid (blockIdx.x), so that they run together and the
// pass goes through memory once: with the segments outermost, plain FP32
// energy density, us, neighbours / outermost: 384^3 1167 / 1256.  Few rows
// (1-D grids: one) are cut into segments of 32 values, one warp each, so that
// they use many SMs: a 4096-point row's second OT pass took 150 us on one SM.
// Short rows share a CTA (up to 256 threads) while that leaves four CTAs per SM.
struct RowShape { dim3 grid, block; };
inline RowShape row_shape(int nx, int ny, int nz) {
  int nseg = (nz + 255) / 256;
  if ((size_t) nx * ny * nseg < (size_t) 2 * rt().num_sms) nseg = (nz + 31) / 32;
  const int bd = ((nz + nseg - 1) / nseg + 31) / 32 * 32;
  nseg = (nz + bd - 1) / bd;
  int ry = 1;
  while (2 * ry * bd <= 256 && (size_t) nx * nseg * ((ny + 2 * ry - 1) / (2 * ry)) >= (size_t) 4 * rt().num_sms) ry *= 2;
  return RowShape{ dim3(nseg, (ny + ry - 1) / ry, nx), dim3(bd, ry) };
}
template <class F> __device__ __forceinline__ void rows_body(int ny, int nz, F &f) {
  const int y = blockIdx.y * blockDim.y + threadIdx.y, x = blockIdx.z, z = blockIdx.x * blockDim.x + threadIdx.x;
  if (y < ny && z < nz) f(x, y, z, (x * ny + y) * nz + z);
}
template <class F> __global__ void rows_kernel(int ny, int nz, F f) {
  pdl_wait();
  rows_body(ny, nz, f);
}

template <class F> int launch_rows(int nx, int ny, int nz, F f, double bytes = 0.0, const char *name = "pointwise") {
  const RowShape r = row_shape(nx, ny, nz);
  ProfScope prof(name, bytes);
  launch_pdl(rows_kernel<F>, r.grid, r.block, 0, rt().stream, ny, nz, f);
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

// The same with a register budget for MINB resident 256-thread CTAs per SM:
// for latency-bound passes with many independent loads per element.
template <int MINB, class F> __global__ void __launch_bounds__(256, MINB) rows_kernel_b(int ny, int nz, F f) {
  pdl_wait();
  rows_body(ny, nz, f);
}
template <int MINB, class F>
int launch_rows_b(int nx, int ny, int nz, F f, double bytes = 0.0, const char *name = "pointwise") {
  const RowShape r = row_shape(nx, ny, nz);
  ProfScope prof(name, bytes);
  launch_pdl(rows_kernel_b<MINB, F>, r.grid, r.block, 0, rt().stream, ny, nz, f);
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

// periodic neighbours of (x, y, z) along axis a, by comparison (no division)
struct Stencil3 {
  int nx, ny, nz;
  __device__ __forceinline__ void nb(int x, int y, int z, int i, int a, int &ip, int &im) const {
    if (a == 0) {
      const int s = ny * nz;
      ip = x + 1 < nx ? i + s : i + s - nx * s;
      im = x > 0 ? i - s : i - s + nx * s;
    } else if (a == 1) {
      ip = y + 1 < ny ? i + nz : i + nz - ny * nz;
      im = y > 0 ? i - nz : i - nz + ny * nz;
    } else {
      ip = z + 1 < nz ? i + 1 : i + 1 - nz;
      im = z > 0 ? i - 1 : i - 1 + nz;
    }
  }
};

// ---------------------------------------------------------------- reductions
// Deterministic FP64 sum of f(i) over i < n: a fixed grid of RED_BLOCKS
// blocks each sums a fixed strided subset, block partials are combined by a
// single block in a fixed order.  Result left in *slot (device).
constexpr int RED_BLOCKS = 1024;
constexpr int RED_THREADS = 256;

__device__ __forceinline__ double block_sum(double v) {
  __shared__ double sh[RED_THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (l < (int) (blockDim.x >> 5)) ? sh[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  __syncthreads();
  return v;
}

template <int NV, class F> __global__ void reduce_partial_kernel(size_t n, F f, double *partial) {
  pdl_wait();
  double acc[NV];
#pragma unroll
  for (int j = 0; j < NV; j++) acc[j] = 0.0;
  for (size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t) gridDim.x * blockDim.x) {
    double v[NV];
    f(i, v);
#pragma unroll
    for (int j = 0; j < NV; j++) acc[j] += v[j];
  }
#pragma unroll
  for (int j = 0; j < NV; j++) {
    double s = block_sum(acc[j]);
    if (threadIdx.x == 0) partial[j * RED_BLOCKS + blockIdx.x] = s;
  }
}

// after(results) runs on one thread once the results are formed
struct NoAfter { __device__ void operator()(const double *) const {} };
template <int NV, class After>
__global__ void reduce_final_kernel(const double *partial, double *slot, double scale, After after) {
  pdl_wait();
  double res[NV];
#pragma unroll
  for (int j = 0; j < NV; j++) {
    double acc = 0.0;
    for (int i = threadIdx.x; i < RED_BLOCKS; i += blockDim.x) acc += partial[j * RED_BLOCKS + i];
    double s = block_sum(acc);
    res[j] = s * scale;
    if (threadIdx.x == 0) slot[j] = res[j];
  }
  if (threadIdx.x == 0) after(res);
}

// From twelve terms a thread on the partial sums are launched ordinarily: their
// CTAs take equal shares, and placed while the kernel before them still runs
// some SMs get eight of them where seven is the even number.  Kinetic energy,
// FP32, us, programmatic / ordinary: 160^3 193 / 179, 256^3 652 / 591, 384^3 2441
// / 2230, 128^3 107 / 101; 64^3 35.1 / 37.2; but the FP64 energy report of 128^3
// 5349 / 5372.
constexpr size_t kOrdinaryReduce = 12 * (size_t) RED_BLOCKS * RED_THREADS;

// f(i, double v[NV]); results (times scale) to slot[0..NV) on the device.
template <int NV, class F, class After = NoAfter>
int reduce_dev(size_t n, F f, double *slot, double scale, After after = NoAfter()) {
  double *part; size_t np;
  DFT_TRY(reduce_partials(&part, &np));
  ProfScope prof("reduce_fp64", 0.0, 2);
  const bool outer = ordinary_launches();
  ordinary_launches() = outer || n >= kOrdinaryReduce;
  launch_pdl(reduce_partial_kernel<NV, F>, RED_BLOCKS, RED_THREADS, 0, rt().stream, n, f, part);
  ordinary_launches() = outer;
  DFT_CHECK_LAUNCH();
  launch_pdl(reduce_final_kernel<NV, After>, 1, RED_THREADS, 0, rt().stream, part, slot, scale, after);
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

// Same, result copied to the host (synchronises the stream).
template <int NV, class F> int reduce_host(size_t n, F f, double *out, double scale) {
  double *slot = reduce_slots();
  DFT_TRY(reduce_dev<NV>(n, f, slot, scale));
  DFT_CUDA(cudaMemcpyAsync(out, slot, sizeof(double) * NV, cudaMemcpyDeviceToHost, rt().stream));
  DFT_CUDA(cudaStreamSynchronize(rt().stream));
  return DFTGPU_OK;
}

// ---------------------------------------------------------------- functors
// Spectral layout [kz][x][y]; real / complex grids [x][y][z].
template <typename T> struct SpecStoreZ {           // z pass output
  static constexpr bool kBatch = true;
  static constexpr bool kSpecZ = true;
  typename cplx_t<T>::type *spec; int nx, ny;
  typename cplx_t<T>::type *scratch = nullptr;      // as many values as the line, for split lines (fft.cuh)
  __device__ void operator()(int x, int y, int k, typename cplx_t<T>::type v) const {
    spec[((size_t) k * nx + x) * ny + y] = v;
  }
};
// Load functors with kAhead provide prefetch_lines(a, b0, nl, ne), called by
// every thread of a CTA of the line kernels: bring the input of lines
// (a, b0 .. b0+nl-1), elements 0 .. ne-1, into L2 (bulk prefetches).
template <typename T> struct SpecLoadZ {            // z pass input (inverse); its tiles are one short
  static constexpr bool kBatch = true;
  typedef typename cplx_t<T>::type C;                // run per plane, not prefetched ahead
  static constexpr bool kSpecZ = true;
  const C *spec; int nx, ny;
  C *scratch = nullptr;                              // as in SpecStoreZ
  __device__ C operator()(int x, int y, int k) const {
    return spec[((size_t) k * nx + x) * ny + y];
  }
};
template <typename T> struct SpecLineY {            // y pass in place: line (kz, x), element y
  static constexpr bool kBatch = true;
  typedef typename cplx_t<T>::type C;
  static constexpr bool kAhead = true;
  typename cplx_t<T>::type *spec; int nx, ny;
  __device__ void prefetch_lines(int kz, int x0, int nl, int) const {     // nl whole lines, contiguous
    if (threadIdx.x == 0) prefetch_bulk_l2(spec + ((size_t) kz * nx + x0) * ny, (size_t) nl * ny * sizeof(C));
  }
  __device__ typename cplx_t<T>::type operator()(int kz, int x, int y) const {
    return spec[((size_t) kz * nx + x) * ny + y];
  }
  __device__ void operator()(int kz, int x, int y, typename cplx_t<T>::type v) const {
    spec[((size_t) kz * nx + x) * ny + y] = v;
  }
};
template <typename T> struct RealPairLoad {         // packed (f[2e], f[2e+1]) of a real row
  static constexpr bool kLine1D = true;
  static constexpr bool kBatch = true;
  static constexpr bool kAhead = true;
  const T *f; int ny, nz;
  __device__ void prefetch_lines(int x, int y0, int nl, int) const {      // nl whole rows, contiguous
    if (threadIdx.x == 0) prefetch_bulk_l2(f + ((size_t) x * ny + y0) * nz, (size_t) nl * nz * sizeof(T));
  }
  // one vector access per pair: rows start on a multiple of nz (even) values
  __device__ typename cplx_t<T>::type operator()(int x, int y, int e) const {
    const T *row = f + ((size_t) x * ny + y) * nz;
    return *reinterpret_cast<const typename cplx_t<T>::type *>(row + 2 * e);
  }
};
template <typename T> struct RealPairStore {        // real row <- scale * (re, im)
  static constexpr bool kLine1D = true;
  static constexpr bool kBatch = true;
  T *f; int ny, nz; T scale;
  __device__ void operator()(int x, int y, int e, typename cplx_t<T>::type v) const {
    T *row = f + ((size_t) x * ny + y) * nz;
    *reinterpret_cast<typename cplx_t<T>::type *>(row + 2 * e) = mk<T>(v.x * scale, v.y * scale);
  }
};
// (|psi[2e]|^2, |psi[2e+1]|^2) of a wave-function row, also stored into the
// density grid: the density pass (src/ot.c:320) done by the first z pass of rho.
// Algorithmic bytes beyond a real-row load: the psi row is twice as wide, and
// the density row is written (2 real fields).
// Split (fetch / cook): the density stores could alias psi for the compiler,
// so without the split every element's psi loads would wait for the previous
// element's store.
template <typename T> struct DensityPairLoad {
  static constexpr bool kLine1D = true;
  typedef typename cplx_t<T>::type C;
  static constexpr bool kAhead = true, kSplit = true;
  struct Raw { C a, b; T *dst; };
  const C *psi; T *rho; int ny, nz;
  __device__ void prefetch_lines(int x, int y0, int nl, int) const {
    if (threadIdx.x == 0) prefetch_bulk_l2(psi + ((size_t) x * ny + y0) * nz, (size_t) nl * nz * sizeof(C));
  }
  __device__ Raw fetch(int x, int y, int e) const {
    const size_t r = ((size_t) x * ny + y) * nz + 2 * e;
    if constexpr (std::is_same<T, float>::value) {   // the pair as one 16-byte load (r even)
      const float4 q = *reinterpret_cast<const float4 *>(psi + r);
      return Raw{ make_float2(q.x, q.y), make_float2(q.z, q.w), rho + r };
    } else {
      return Raw{ psi[r], psi[r + 1], rho + r };
    }
  }
  __device__ C cook(const Raw &w) const {
    const C d = mk<T>(w.a.x * w.a.x + w.a.y * w.a.y, w.b.x * w.b.x + w.b.y * w.b.y);
    *reinterpret_cast<C *>(w.dst) = d;     // rows hold an even number of values
    return d;
  }
  __device__ C operator()(int x, int y, int e) const { return cook(fetch(x, y, e)); }
};
// P <- scale * (P + (re, im) added to the real parts of P[2e], P[2e+1]): the
// last c2r z pass of the potential adds the merged linear part into P and
// applies the predict-correct scale.  Algorithmic bytes beyond a real-row
// store: P is read and written (3 real fields).
template <typename T> struct PotAddPairStore {
  static constexpr bool kLine1D = true;
  typedef typename cplx_t<T>::type C;
  static constexpr bool kSplit = true;
  C *pot; int ny, nz; T scale;
  __device__ void prefetch(int x, int y, int e) const {
    const size_t r = ((size_t) x * ny + y) * nz + 2 * e;
    if ((r * sizeof(C)) % 32 == 0) prefetch_l2(pot + r);   // one per 32-byte sector
  }
  __device__ void operator()(int x, int y, int e, C v) const {
    const size_t r = ((size_t) x * ny + y) * nz + 2 * e;
    if constexpr (std::is_same<T, float>::value) {   // the pair as one 16-byte access (r even)
      float4 q = *reinterpret_cast<const float4 *>(pot + r);
      q.x += v.x;
      q.z += v.y;
      *reinterpret_cast<float4 *>(pot + r) = make_float4(q.x * scale, q.y * scale, q.z * scale, q.w * scale);
    } else {
      C p0 = pot[r], p1 = pot[r + 1];
      p0.x += v.x;
      p1.x += v.y;
      pot[r] = mk<T>(p0.x * scale, p0.y * scale);
      pot[r + 1] = mk<T>(p1.x * scale, p1.y * scale);
    }
  }
};
template <typename T> struct CplxLoad {
  const typename cplx_t<T>::type *f; int ny, nz;
  __device__ typename cplx_t<T>::type operator()(int x, int y, int e) const {
    return f[((size_t) x * ny + y) * nz + e];
  }
};

// Fused z + y passes of a real field (fft.cu; the cluster kernels are
// instantiated in that one translation unit).  Return -1 when no fused
// instantiation fits the shape (the caller runs the separate passes).
int launch_zy_r2c(const RealPairLoad<float> &ld, float2 *spec, int nx, int ny, int nz);
int launch_yz_c2r(const float2 *spec, const RealPairStore<float> &st, int nx, int ny, int nz);

// y passes over nkz planes of nf spectral buffers (ny = 1: the identity)
template <typename T>
int ypass_batch(typename cplx_t<T>::type *const *spec, int nf, int nx, int ny, int nkz, T sign) {
  if (ny == 1 || nf == 0) return DFTGPU_OK;
  Batch<SpecLineY<T>, LINE_BATCH> io;
  memset(&io, 0, sizeof(io));
  for (int i = 0; i < nf; i++) io.f[i] = SpecLineY<T>{spec[i], nx, ny};
  return launch_lines_batch<T, LINE_C2C, 1, 1, LINE_BATCH>(ny, nkz, nx, nf, sign, io, io);
}
template <typename T> int ypass(typename cplx_t<T>::type *spec, int nx, int ny, int nkz, T sign) {
  return ypass_batch<T>(&spec, 1, nx, ny, nkz, sign);
}

// forward r2c of a real field through its z and y passes, with a custom
// packed-pair loader (fused producer); spec is [nz/2+1][nx][ny]
// extra_bytes: algorithmic bytes of the load / store functor beyond one real field
template <typename T, class Ld>
int rfft_zy(const Ld &ld, typename cplx_t<T>::type *spec, int nx, int ny, int nz, double extra_bytes = 0.0) {
  if constexpr (std::is_same<Ld, RealPairLoad<float>>::value) {
    const int rc = launch_zy_r2c(ld, spec, nx, ny, nz);
    if (rc >= 0) return rc;
  }
  SpecStoreZ<T> st{spec, nx, ny};
  DFT_TRY((launch_lines<T, LINE_R2C, 1, 0>(nz / 2, nx, ny, (T) -1, ld, st, extra_bytes)));
  return ypass<T>(spec, nx, ny, nz / 2 + 1, (T) -1);
}

// inverse: y passes then c2r z pass into a custom consumer st(x, y, e, (v[2e], v[2e+1]))
template <typename T, class St>
int irfft_yz(typename cplx_t<T>::type *spec, const St &st, int nx, int ny, int nz, double extra_bytes = 0.0) {
  if constexpr (std::is_same<St, RealPairStore<float>>::value) {
    const int rc = launch_yz_c2r(spec, st, nx, ny, nz);
    if (rc >= 0) return rc;
  }
  DFT_TRY(ypass<T>(spec, nx, ny, nz / 2 + 1, (T) 1));
  SpecLoadZ<T> ld{spec, nx, ny};
  return launch_lines<T, LINE_C2R, 0, 1>(nz / 2, nx, ny, (T) 1, ld, st, extra_bytes);
}

// ---------------------------------------------------------------- z passes and convolutions
// The z passes of nf real fields, up to LINE_BATCH in one launch; scr: offset of
// each spectrum's scratch in its buffer (spec_scratch(), 0: none).
template <typename T>
int zpass_fwd_n(const T *const *f, typename cplx_t<T>::type *const *spec, int nf, int nx, int ny, int nz, size_t scr) {
  for (int i0 = 0; i0 < nf; i0 += LINE_BATCH) {
    const int m = nf - i0 < LINE_BATCH ? nf - i0 : LINE_BATCH;
    Batch<RealPairLoad<T>, LINE_BATCH> ld;
    Batch<SpecStoreZ<T>, LINE_BATCH> st;
    memset(&ld, 0, sizeof(ld));
    memset(&st, 0, sizeof(st));
    for (int i = 0; i < m; i++) {
      ld.f[i] = RealPairLoad<T>{f[i0 + i], ny, nz};
      st.f[i] = SpecStoreZ<T>{spec[i0 + i], nx, ny, scr ? spec[i0 + i] + scr : nullptr};
    }
    DFT_TRY((launch_lines_batch<T, LINE_R2C, 1, 0, LINE_BATCH>(nz / 2, nx, ny, m, (T) -1, ld, st)));
  }
  return DFTGPU_OK;
}
template <typename T>
int zpass_inv_n(typename cplx_t<T>::type *const *spec, T *const *f, int nf, int nx, int ny, int nz, size_t scr) {
  for (int i0 = 0; i0 < nf; i0 += LINE_BATCH) {
    const int m = nf - i0 < LINE_BATCH ? nf - i0 : LINE_BATCH;
    Batch<SpecLoadZ<T>, LINE_BATCH> ld;
    Batch<RealPairStore<T>, LINE_BATCH> st;
    memset(&ld, 0, sizeof(ld));
    memset(&st, 0, sizeof(st));
    for (int i = 0; i < m; i++) {
      ld.f[i] = SpecLoadZ<T>{spec[i0 + i], nx, ny, scr ? spec[i0 + i] + scr : nullptr};
      st.f[i] = RealPairStore<T>{f[i0 + i], ny, nz, (T) 1};
    }
    DFT_TRY((launch_lines_batch<T, LINE_C2R, 0, 1, LINE_BATCH>(nz / 2, nx, ny, m, (T) 1, ld, st)));
  }
  return DFTGPU_OK;
}

// Convolution of half spectra whose y passes are still to be done: forward y
// passes of the inputs (those in the bit mask ydone have had theirs), x passes
// of A, inverse y passes of the outputs.  Outputs may be inputs, not accumulate.
// FP32 above kBatchBytes of spectra: the two halves of the kz planes on two
// parallel branches, whose launches fill each other's last waves.  Full
// potential, us, in one piece / halves / thirds: 128^3 258 / 252 / 261, 192^3
// 906 / 896 / 927, 256^3 1753 / 1724 / 1749, 512 x 512 x 256 7642 / 7591 / 7659
// (chunks small enough to stay in L2 between the passes: 1732 to 1789 and 8109
// to 8214, their launches are too short).
template <typename T> int convolve(const XConvArgs<T> &A, unsigned ydone) {
  typedef typename cplx_t<T>::type C;
  const size_t plane = (size_t) A.nx * A.ny, oct = (size_t) (A.nx / 2 + 1) * (A.ny / 2 + 1);
  int extra = 0;   // outputs that are not inputs
  for (int o = 0; o < A.nout; o++) {
    bool in = false;
    for (int i = 0; i < A.nin; i++) in |= A.out[o].dst == A.src[i];
    extra += !in;
  }
  int step = A.nkz;
  if (sizeof(T) == 4 && (double) (A.nin + extra) * plane * sizeof(C) * A.nkz > kBatchBytes) step = (A.nkz + 1) / 2;
  return par_for((A.nkz + step - 1) / step, [&](int j) -> int {
    const int k0 = j * step, nk = A.nkz - k0 < step ? A.nkz - k0 : step;
    XConvArgs<T> c = A;
    c.nkz = nk;
    C *y[XC_MAX_OUT];
    int n = 0;
    for (int i = 0; i < A.nin; i++) {
      c.src[i] = A.src[i] + k0 * plane;
      if (!(ydone >> i & 1)) y[n++] = const_cast<C *>(c.src[i]);
    }
    for (int o = 0; o < A.nout; o++) {
      c.out[o].dst = A.out[o].dst + k0 * plane;
      for (int t = A.out[o].t0; t < A.out[o].t0 + A.out[o].nt; t++)
        if (A.term[t].ker) c.term[t].ker = A.term[t].ker + k0 * oct;
    }
    DFT_TRY(ypass_batch<T>(y, n, A.nx, A.ny, nk, (T) -1));
    DFT_TRY(launch_xconv<T>(c));
    for (int o = 0; o < A.nout; o++) y[o] = c.out[o].dst;
    return ypass_batch<T>(y, A.nout, A.nx, A.ny, nk, (T) 1);
  });
}

// forward y, kinetic x and inverse y passes of a complex spectrum [nz][nx][ny],
// in FP32 in chunks of planes that stay in L2 between the passes: one
// propagation, us, whole / 80 / 40 / 20 MB chunks: 256^3 295 / 291 / 270 / 274,
// 240^3 477 / 460 / 457 / 510, 512 x 512 x 256 1371 / 1381 / 1324 / 1300.
constexpr double kKineticChunk = 40e6;
template <typename T> int kinetic_yxy(const KinArgs<T> &K, typename cplx_t<T>::type *spec) {
  const size_t plane = (size_t) K.nx * K.ny;
  int step = K.nz;
  const double bytes = (double) plane * 2 * sizeof(T) * K.nz;
  if (sizeof(T) == 4 && bytes > kKineticChunk) {
    const int n = (int) (bytes / kKineticChunk) + 1;
    step = (K.nz + n - 1) / n;
  }
  return par_for((K.nz + step - 1) / step, [&](int j) -> int {
    KinArgs<T> c = K;
    c.kz0i = j * step;
    c.nkz = K.nz - c.kz0i < step ? K.nz - c.kz0i : step;
    c.data = spec + c.kz0i * plane;
    DFT_TRY(ypass<T>(c.data, K.nx, K.ny, c.nkz, (T) -1));
    DFT_TRY(launch_xkinetic<T>(c));
    return ypass<T>(c.data, K.nx, K.ny, c.nkz, (T) 1);
  });
}

}  // namespace dftgpu
