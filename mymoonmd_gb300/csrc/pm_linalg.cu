// Device linear algebra: CSR SpMV launchers, deterministic BLAS-1 reductions and
// the dense coarse-grid inverse.
#include <algorithm>
#include <cmath>

#include <cooperative_groups.h>

#include "pm_linalg.cuh"

namespace pm {

// ---------------------------------------------------------------- context ---
void ctx_init(pm_ctx* c, int device) {
  c->device = device;
  PM_CUDA(cudaSetDevice(device));
  PM_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
  PM_CUDA(cudaStreamCreateWithFlags(&c->side, cudaStreamNonBlocking));
  PM_CUDA(cudaEventCreateWithFlags(&c->side_event, cudaEventDisableTiming));
  PM_CUDA(cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device));
  PM_CUDA(cudaMallocHost(&c->host_scalars, 64 * sizeof(double)));
  c->dev_scalars.alloc(256);
  c->partials.alloc(4 * kRedBlocks);
  c->n_partials = kRedBlocks;
}

void ctx_destroy(pm_ctx* c) {
  if (c->stream) cudaStreamSynchronize(c->stream);
  c->dev_scalars.release();
  c->partials.release();
  if (c->host_scalars) cudaFreeHost(c->host_scalars);
  c->host_scalars = nullptr;
  if (c->side) cudaStreamSynchronize(c->side);
  if (c->side_event) cudaEventDestroy(c->side_event);
  if (c->side) cudaStreamDestroy(c->side);
  c->side_event = nullptr;
  c->side = nullptr;
  if (c->stream) cudaStreamDestroy(c->stream);
  c->stream = nullptr;
}

static inline int nblocks(long long n, int t) { return int((n + t - 1) / t); }

// -------------------------------------------------------------------- CSR ---
void DevCsr::upload(pm_ctx* c, int nr, int nc, int na, const int* rp, const int* ci,
                    const double* v) {
  n_rows = nr;
  n_cols = nc;
  n_active = na;
  nnz = rp[nr];
  row_ptr.upload(rp, size_t(nr) + 1, c->stream);
  // column indices readable up to nnz rounded up to 4 entries; the tail holds
  // zeros
  cols.alloc(size_t(nnz4()));
  if (nnz) PM_CUDA(cudaMemcpyAsync(cols.p, ci, size_t(nnz) * sizeof(int), cudaMemcpyHostToDevice, c->stream));
  if (nnz4() > nnz)
    PM_CUDA(cudaMemsetAsync(cols.p + nnz, 0, size_t(nnz4() - nnz) * sizeof(int), c->stream));
  if (v) vals.upload(v, size_t(nnz), c->stream);
  else {
    vals.alloc(size_t(nnz));
    if (nnz) PM_CUDA(cudaMemsetAsync(vals.p, 0, vals.bytes(), c->stream));
  }
  drop_sell();  // a new structure: no sliced layout yet
  // measured on GB300. FP64: an instruction costs a sub-core about 75 clocks, so
  // short rows (at most 16 entries on average) take two lanes: half as many
  // additions and Jacobi divisions per row as with four. FP64 cycle of 2D Q1 in us,
  // four lanes / two / one: 128^2 76 / 72 / 78, 256^2 121 / 105 / 103, 512^2
  // 298 / 224 / 221, 1024^2 1315 / 1008 / 965; 2D Q2 128^2 154 / 128 / 144,
  // 512^2 1649 / 1202 / 1261. Long rows: four lanes x eight loads. FP32: eight
  // lanes x sixteen loads in flight (3.9 TB/s vs 3.4 TB/s at four x eight on
  // 15.8 M and 54.5 M nonzeros), short rows four x four
  const double avg = nr ? double(nnz) / nr : 1.0;
  lanes = avg > 16.0 ? 4 : 2;
  unroll = 8;
  lanes32 = avg > 16.0 ? 8 : 4;
  unroll32 = avg > 16.0 ? 16 : 4;
  stream = false;
  std::vector<int> rb = build_row_blocks(nr, rp, kStreamNnz, 1024);
  n_rblocks = rb.empty() ? 0 : int(rb.size()) - 1;
  if (n_rblocks) rblock.upload(rb, c->stream);
  else rblock.release();
  set_single_block();
}

std::vector<int> build_row_blocks(int n_rows, const int* rp, int max_nnz, int max_rows) {
  std::vector<int> rb;
  if (n_rows <= 0) return rb;
  rb.push_back(0);
  int r0 = 0;
  for (int i = 0; i < n_rows; ++i) {
    if (rp[i + 1] - rp[i] > max_nnz) return std::vector<int>();
    if (rp[i + 1] - rp[r0] > max_nnz || i - r0 >= max_rows) {
      rb.push_back(i);
      r0 = i;
    }
  }
  rb.push_back(n_rows);
  return rb;
}

bool build_sell_layout(int n_rows, const int* rp, const int* ci, int L, int window, std::vector<int>& perm,
                       std::vector<int>& off, std::vector<int>& cols, std::vector<int>& src) {
  const int C = 32 / L;
  if (L < 1 || 32 % L != 0 || window % C != 0) throw Error(PM_E_INVALID, "sliced layout: bad lanes or window");
  const int n_sl = (n_rows + C - 1) / C;
  perm.assign(size_t(n_sl) * C, -1);
  // rows sorted by length, longest first, ties in row order, per window
  std::vector<int> idx;
  for (int w0 = 0; w0 < n_rows; w0 += window) {
    const int w1 = std::min(n_rows, w0 + window);
    idx.resize(size_t(w1 - w0));
    for (int i = w0; i < w1; ++i) idx[size_t(i - w0)] = i;
    std::stable_sort(idx.begin(), idx.end(),
                     [&](int a, int b) { return rp[a + 1] - rp[a] > rp[b + 1] - rp[b]; });
    std::copy(idx.begin(), idx.end(), perm.begin() + w0);
  }
  off.assign(size_t(n_sl) + 1, 0);
  int64_t total = 0;
  for (int sl = 0; sl < n_sl; ++sl) {
    int width = 0;
    for (int q = 0; q < C; ++q) {
      const int r = perm[size_t(sl) * C + q];
      if (r >= 0) width = std::max(width, rp[r + 1] - rp[r]);
    }
    total += int64_t(32) * ((width + L - 1) / L);
    if (total > int64_t(0x7fffffff)) return false;
    off[size_t(sl) + 1] = int(total);
  }
  cols.assign(size_t(total), 0);
  src.assign(size_t(total), -1);
  for (int sl = 0; sl < n_sl; ++sl) {
    const int T = (off[size_t(sl) + 1] - off[size_t(sl)]) / 32;
    for (int q = 0; q < C; ++q) {
      const int r = perm[size_t(sl) * C + q];
      const int len = r >= 0 ? rp[r + 1] - rp[r] : 0;
      // padding repeats the row's last column (its x is already cached)
      const int pad_col = len > 0 ? ci[rp[r] + len - 1] : 0;
      for (int t = 0; t < T; ++t)
        for (int sub = 0; sub < L; ++sub) {
          const int j = t * L + sub;
          const size_t slot = size_t(off[size_t(sl)]) + size_t(t) * 32 + size_t(sub) * C + q;
          if (j < len) {
            cols[slot] = ci[rp[r] + j];
            src[slot] = rp[r] + j;
          } else {
            cols[slot] = pad_col;
          }
        }
    }
  }
  return true;
}

void DevCsr::drop_sell() {
  sell_lanes = 0;
  n_slices = 0;
  sell_entries = 0;
  sell64_ok = false;
  sell_perm.release();
  sell_off.release();
  sell_cols.release();
  sell_src.release();
  sell_vals.release();
  sell_vals64.release();
}

void DevCsr::build_sell(pm_ctx* c, int L) {
  const bool had64 = sell_vals64.p != nullptr;
  sell_lanes = 0;
  n_slices = 0;
  sell_entries = 0;
  sell64_ok = false;
  std::vector<int> rp(static_cast<size_t>(n_rows) + 1), ci(static_cast<size_t>(nnz));
  PM_CUDA(cudaMemcpyAsync(rp.data(), row_ptr.p, rp.size() * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  if (nnz) PM_CUDA(cudaMemcpyAsync(ci.data(), cols.p, ci.size() * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  PM_CUDA(cudaStreamSynchronize(c->stream));
  std::vector<int> perm, off, sc, src;
  if (!build_sell_layout(n_rows, rp.data(), ci.data(), L, kSellWindow, perm, off, sc, src)) {
    drop_sell();
    return;
  }
  sell_perm.upload(perm, c->stream);
  sell_off.upload(off, c->stream);
  sell_cols.upload(sc, c->stream);
  sell_src.upload(src, c->stream);
  sell_vals.ensure(sc.size());
  PM_CUDA(cudaStreamSynchronize(c->stream));  // the host vectors go out of scope
  sell_lanes = L;
  n_slices = int(off.size()) - 1;
  sell_entries = int64_t(sc.size());
  sell_max_steps = 0;
  for (int s = 0; s < n_slices; ++s) sell_max_steps = std::max(sell_max_steps, (off[s + 1] - off[s]) / 32);
  if (had64) {  // the FP64 copy follows the new layout
    sell_vals64.ensure(sc.size());
    values_changed(c);
  }
}

void DevCsr::set_single_block() {
  mask = BlockMask{};
  mask.nb = 1;
  mask.start[0] = 0;
  mask.active_end[0] = n_active;
  mask.end[0] = n_rows;
}

void DevCsr::set_blocks(int nb, const int* lengths, const int* actives) {
  if (nb < 1 || nb > 4) throw Error(PM_E_INVALID, "block vectors hold 1..4 blocks");
  mask = BlockMask{};
  mask.nb = nb;
  int off = 0;
  for (int b = 0; b < nb; ++b) {
    mask.start[b] = off;
    mask.active_end[b] = off + actives[b];
    off += lengths[b];
    mask.end[b] = off;
  }
  if (off != n_rows) throw Error(PM_E_INVALID, "block lengths do not add up to the matrix rows");
  n_active = 0;
  for (int b = 0; b < nb; ++b) n_active += actives[b];
}

__global__ void k_d2f(long long n, const double* __restrict__ x, float* __restrict__ y) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] = float(x[i]);
}
__global__ void k_f2d(long long n, const float* __restrict__ x, double* __restrict__ y) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] = double(x[i]);
}

static int grid_for(pm_ctx* c, long long n) {
  long long b = (n + 255) / 256;
  long long cap = (long long)c->num_sms * 8;
  return int(std::max<long long>(1, std::min(b, cap)));
}

template <class TO>
__global__ void k_sell_fill(long long n, const int* __restrict__ src, const double* __restrict__ v,
                            TO* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int k = src[i];
    out[i] = k >= 0 ? TO(v[k]) : TO(0);
  }
}

void DevCsr::values_changed(pm_ctx* c) {
  sell64_ok = false;
  if (sell_lanes && sell_entries && sell_vals64.p) {
    k_sell_fill<double><<<grid_for(c, sell_entries), 256, 0, c->stream>>>(sell_entries, sell_src.p, vals.p,
                                                                         sell_vals64.p);
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
    sell64_ok = true;
    sell_fresh = true;
  }
}

void DevCsr::make_sliced64(pm_ctx* c) {
  const int want = c->sell_shape64 / 100;
  if (want <= 0 || nnz <= c->sell_min_avg * int64_t(n_rows)) return;
  if (sell_lanes == 0) build_sell(c, want);
  if (sell_lanes != want || !sell_entries) return;
  if (!sell_vals64.p) sell_vals64.ensure(size_t(sell_entries));
  if (!sell64_ok) values_changed(c);
}

void DevCsr::make_fp32(pm_ctx* c) {
  // the sliced copy: matrices with more than sell_min_avg entries per row on
  // average; laid out once per lane count
  const int want = c->sell_shape / 100;
  if (want > 0 && want != sell_lanes && nnz > c->sell_min_avg * int64_t(n_rows)) build_sell(c, want);
  if (sell_lanes && sell_entries) {
    k_sell_fill<float><<<grid_for(c, sell_entries), 256, 0, c->stream>>>(sell_entries, sell_src.p, vals.p,
                                                                       sell_vals.p);
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
    sell_fresh = true;
  }
  vals32.ensure(size_t(nnz4()));
  if (nnz4() > nnz)
    PM_CUDA(cudaMemsetAsync(vals32.p + nnz, 0, size_t(nnz4() - nnz) * sizeof(float), c->stream));
  if (nnz) {
    k_d2f<<<grid_for(c, nnz), 256, 0, c->stream>>>(nnz, vals.p, vals32.p);
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
  }
  if (diag.p) {
    diag32.ensure(size_t(n_rows));
    k_d2f<<<grid_for(c, n_rows), 256, 0, c->stream>>>(n_rows, diag.p, diag32.p);
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
  }
}

// diagonal entries (Iteration_jacobi: extract_diagonal_entries); a missing
// diagonal entry is recorded as 0 and reported by the caller
// eight lanes per row, four column indices in flight per lane, the first match
// of the row; the FP32 copy in the same launch. One thread per row walked its
// indices one dependent load after another: 32 us on the 274,625 rows of 3D Q2 on 32^3, 25 us now
__global__ void __launch_bounds__(256)
k_diag(int n, const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ v,
       double* __restrict__ d, float* __restrict__ d32) {
  const int lane = threadIdx.x & 7, i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int beg = i < n ? rp[i] : 0, end = i < n ? rp[i + 1] : 0;
  int at = 0x7fffffff;
  for (int k = beg + lane; k < end && at == 0x7fffffff; k += 32) {
    int col[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) col[u] = k + 8 * u < end ? ci[k + 8 * u] : -1;
#pragma unroll
    for (int u = 3; u >= 0; --u)
      if (col[u] == i) at = k + 8 * u;
  }
#pragma unroll
  for (int off = 4; off; off >>= 1) at = min(at, __shfl_xor_sync(0xffffffffu, at, off));
  if (lane || i >= n) return;
  const double r = at == 0x7fffffff ? 0.0 : v[at];
  d[i] = r;
  if (d32) d32[i] = float(r);
}

void DevCsr::make_diag(pm_ctx* c) {
  diag.ensure(size_t(n_rows));
  if (vals32.p) diag32.ensure(size_t(n_rows));
  if (n_rows) {
    k_diag<<<nblocks(8ll * n_rows, 256), 256, 0, c->stream>>>(n_rows, row_ptr.p, cols.p, vals.p, diag.p,
                                                            vals32.p ? diag32.p : nullptr);
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
  }
}

size_t DevCsr::spmv_bytes(int eb, bool read_y) const {
  // values + column indices + row pointers + x gathered once + y written (+read)
  return size_t(nnz) * (eb + 4) + size_t(n_rows + 1) * 4 + size_t(n_cols) * eb +
         size_t(n_rows) * eb * (read_y ? 2 : 1);
}

template <class TV, class TX, class TA, int G, int EPI>
static void launch_gu(pm_ctx* c, int U, int grid, int n, const int* rp, const int* ci, const TV* v,
                      const TX* x, TX* y, const TX* b, const TX* d, TA alpha, const BlockMask& m) {
  const dim3 gr(grid), bl(256);
  // launched early inside a cycle: its first kernel is launched plainly, so the
  // matrices are complete. 76 us instead of 92 for the launched cycle of 2D Q1 on
  // 128^2 (FP64); a bound on the grid at one block per SM gave 85, bounds at 4, 16
  // and 1000 the same as none
  auto go = [&](auto kern) {
    if (c->in_cycle) launch_pdl(c, kern, gr, bl, 0, n, rp, ci, v, x, y, b, d, x, alpha, m);
    else launch_k(c, kern, gr, bl, 0, n, rp, ci, v, x, y, b, d, x, alpha, m);
  };
  switch (U) {
    case 2: go(csr_kernel<TV, TX, TA, G, 2, EPI>); break;
    case 4: go(csr_kernel<TV, TX, TA, G, 4, EPI>); break;
    case 16: go(csr_kernel<TV, TX, TA, G, 16, EPI>); break;
    default: go(csr_kernel<TV, TX, TA, G, 8, EPI>); break;
  }
}

template <class TV, class TX, class TA, int EPI>
static void launch_epi(pm_ctx* c, int G, int U, int n, const int* rp, const int* ci, const TV* v,
                       const TX* x, TX* y, const TX* b, const TX* d, TA alpha, const BlockMask& m,
                       const int* rblock = nullptr, int n_rblocks = 0) {
  if (n <= 0) return;
  BlockMask mg = m;
  mg.guard = c->guard;
  if (rblock && n_rblocks > 0) {
    csr_stream_kernel<TV, TX, TA, kStreamNnz, EPI><<<n_rblocks, 256, 0, c->stream>>>(
        rblock, rp, ci, v, x, y, b, d, alpha, mg);
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
    return;
  }
  const int grid = nblocks((long long)n * G, 256);
  switch (G) {
    case 1: launch_gu<TV, TX, TA, 1, EPI>(c, U, grid, n, rp, ci, v, x, y, b, d, alpha, mg); break;
    case 2: launch_gu<TV, TX, TA, 2, EPI>(c, U, grid, n, rp, ci, v, x, y, b, d, alpha, mg); break;
    case 4: launch_gu<TV, TX, TA, 4, EPI>(c, U, grid, n, rp, ci, v, x, y, b, d, alpha, mg); break;
    case 8: launch_gu<TV, TX, TA, 8, EPI>(c, U, grid, n, rp, ci, v, x, y, b, d, alpha, mg); break;
    case 16: launch_gu<TV, TX, TA, 16, EPI>(c, U, grid, n, rp, ci, v, x, y, b, d, alpha, mg); break;
    default: launch_gu<TV, TX, TA, 32, EPI>(c, U, grid, n, rp, ci, v, x, y, b, d, alpha, mg); break;
  }
}

cudaEvent_t probe_event(pm_ctx* c) {
  if (!c->probe_pool.empty()) {
    cudaEvent_t e = c->probe_pool.back();
    c->probe_pool.pop_back();
    return e;
  }
  cudaEvent_t e;
  PM_CUDA(cudaEventCreate(&e));
  return e;
}

// algorithmic bytes of one SpMV-family launch: values, column indices, row
// pointers, the gathered vector once, and the per-row vectors the epilogue
// reads and writes
static double epi_bytes(const DevCsr& A, int epi, int eb, int n) {
  double rows_vec = 1.0;  // y written
  if (epi == EPI_AXPY || epi == EPI_PROLONG) rows_vec += 1.0;  // y read
  if (epi == EPI_DEFECT) rows_vec += 1.0;                      // b read
  if (epi == EPI_JACOBI || epi == EPI_RESTRICT_ZERO) rows_vec += 2.0;  // b and diag read; diag read, x0 written
  return double(A.nnz) * (eb + 4) + double(n + 1) * 4 + double(A.n_cols) * eb + double(n) * eb * rows_vec;
}

template <class T>
static const T* sell_values(const DevCsr& A);
template <>
const float* sell_values<float>(const DevCsr& A) { return A.sell_vals.p; }
template <>
const double* sell_values<double>(const DevCsr& A) { return A.sell_vals64.p; }

template <class T, int L, int U, bool P, int EPI>
static void launch_sell_epi(pm_ctx* c, const DevCsr& A, const T* x, T* y, const T* b, const T* d, T alpha,
                            const BlockMask& m) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(nblocks(A.n_slices, 4)));  // four warps (slices) per block
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // plainly after a fill of the sliced values, so that this launch and the early ones
  // after it find them complete (a cycle's first kernel is launched plainly)
  cfg.numAttrs = c->pdl >= 1 && (c->in_cycle || !A.sell_fresh) ? 1 : 0;
  A.sell_fresh = false;
  PM_CUDA(cudaLaunchKernelEx(&cfg, sell_kernel<T, L, U, P, EPI>, A.n_slices, (const int*)A.sell_perm.p,
                             (const int*)A.sell_off.p, (const int*)A.sell_cols.p, sell_values<T>(A), x, y, b, d,
                             alpha, m));
}

template <class T, int L, int U, bool P>
static void launch_sell_shape(pm_ctx* c, const DevCsr& A, int epi, const T* x, T* y, const T* b, const T* d,
                              T alpha, const BlockMask& m) {
  switch (epi) {
    case EPI_AXPY: launch_sell_epi<T, L, U, P, EPI_AXPY>(c, A, x, y, b, d, alpha, m); break;
    case EPI_SET: launch_sell_epi<T, L, U, P, EPI_SET>(c, A, x, y, b, d, alpha, m); break;
    case EPI_DEFECT: launch_sell_epi<T, L, U, P, EPI_DEFECT>(c, A, x, y, b, d, alpha, m); break;
    case EPI_JACOBI: launch_sell_epi<T, L, U, P, EPI_JACOBI>(c, A, x, y, b, d, alpha, m); break;
    case EPI_RESTRICT: launch_sell_epi<T, L, U, P, EPI_RESTRICT>(c, A, x, y, b, d, alpha, m); break;
    case EPI_PROLONG: launch_sell_epi<T, L, U, P, EPI_PROLONG>(c, A, x, y, b, d, alpha, m); break;
    case EPI_RESTRICT_ZERO: launch_sell_epi<T, L, U, P, EPI_RESTRICT_ZERO>(c, A, x, y, b, d, alpha, m); break;
    default: throw Error(PM_E_INVALID, "unknown SpMV epilogue");
  }
}

// Shapes 442 (FP64) and 482 (FP32): twice the steps in flight where the matrix has
// slices of more than eight steps (a launch of few slices is as long as its longest)
// and the launch few slices (the sums are the same). Four lanes, half / twice the steps:
//   FP64 cycle of 3D Q2 in us: 8^3 49.9 / 43.8, 16^3 135.6 / 101.9 (30 slices per SM
//   in the finest sweep), 24^3 211.5 / 195.9 (97); above 128 slices per SM the finest
//   sweep is no faster (28^3 263 / 271, the SpMV of 32^3 39.2 / 42.8). Product of the
//   combined Stokes matrix of 12^3 20.2 / 13.0.
//   FP32 cycle of 3D Q2: 8^3 31.0 / 29.1, 16^3 61.5 / 56.0, 24^3 105.3 / 103.0; the
//   finest sweep of 32^3 (226) 28.8 / 28.9.
//   Restriction of the 24^3 Stokes levels (5 to 8 steps on average, 37 at most): the
//   mixed request 20.41 / 20.21 ms.
//   Short rows (3D Q1: at most seven steps) lose: FP32 cycle of 32^3 48.3 / 51.3, 48^3
//   66.6 / 76.1; FP64 32^3 88.1 / 89.5, 48^3 127.2 / 140.8. Only FP64 launches of few
//   slices gain (16^3, 4 slices per SM: 53.1 / 49.4).
static bool sell_long_rows(const DevCsr& A) { return A.sell_max_steps > 8; }
static bool sell_deep64(const pm_ctx* c, const DevCsr& A, int ns = 1) {
  const long long slices = (long long)A.n_slices * ns;
  return slices <= (sell_long_rows(A) ? 128ll : 16ll) * c->num_sms;
}
static bool sell_deep32(const pm_ctx* c, const DevCsr& A, int ns = 1) {
  return sell_long_rows(A) && (long long)A.n_slices * ns <= 128ll * c->num_sms;
}

static void launch_sell(pm_ctx* c, const DevCsr& A, int epi, const float* x, float* y, const float* b,
                        const float* d, float alpha) {
  BlockMask mg = A.mask;
  mg.guard = c->guard;
  switch (c->sell_shape) {
    case 140: launch_sell_shape<float, 1, 4, false>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 141: launch_sell_shape<float, 1, 4, true>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 180: launch_sell_shape<float, 1, 8, false>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 240: launch_sell_shape<float, 2, 4, false>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 241: launch_sell_shape<float, 2, 4, true>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 280: launch_sell_shape<float, 2, 8, false>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 440: launch_sell_shape<float, 4, 4, false>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 441: launch_sell_shape<float, 4, 4, true>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 480: launch_sell_shape<float, 4, 8, false>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 481: launch_sell_shape<float, 4, 8, true>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 482:
      if (sell_deep32(c, A)) launch_sell_shape<float, 4, 16, true>(c, A, epi, x, y, b, d, alpha, mg);
      else launch_sell_shape<float, 4, 8, true>(c, A, epi, x, y, b, d, alpha, mg);
      break;
    case 840: launch_sell_shape<float, 8, 4, false>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 841: launch_sell_shape<float, 8, 4, true>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 881: launch_sell_shape<float, 8, 8, true>(c, A, epi, x, y, b, d, alpha, mg); break;
    default: throw Error(PM_E_INVALID, "unknown sliced SpMV shape " + std::to_string(c->sell_shape));
  }
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

static void launch_sell64(pm_ctx* c, const DevCsr& A, int epi, const double* x, double* y, const double* b,
                          const double* d, double alpha) {
  BlockMask mg = A.mask;
  mg.guard = c->guard;
  switch (c->sell_shape64) {
    case 441: launch_sell_shape<double, 4, 4, true>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 442:
      if (sell_deep64(c, A)) launch_sell_shape<double, 4, 8, true>(c, A, epi, x, y, b, d, alpha, mg);
      else launch_sell_shape<double, 4, 4, true>(c, A, epi, x, y, b, d, alpha, mg);
      break;
    case 481: launch_sell_shape<double, 4, 8, true>(c, A, epi, x, y, b, d, alpha, mg); break;
    case 841: launch_sell_shape<double, 8, 4, true>(c, A, epi, x, y, b, d, alpha, mg); break;
    default: throw Error(PM_E_INVALID, "unknown FP64 sliced SpMV shape " + std::to_string(c->sell_shape64));
  }
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

template <class TV, class TX, class TA>
static void csr_dispatch(pm_ctx* c, const DevCsr& A, const TV* vals, const TX* diag, int epi,
                         const TX* x, TX* y, const TX* b, TA alpha, int n) {
  const bool fp32 = sizeof(TV) == 4;
  const int G = fp32 ? A.lanes32 : A.lanes;
  const int U = fp32 ? A.unroll32 : A.unroll;
  const bool use_stream = A.stream && A.n_rblocks > 0 && n == A.n_rows;
  const int* rb = use_stream ? A.rblock.p : nullptr;
  const int nrb = use_stream ? A.n_rblocks : 0;
  const int* rp = A.row_ptr.p;
  const int* ci = A.cols.p;
  const bool probe = c->probe_nnz != 0 && A.nnz == c->probe_nnz &&
                     (c->probe_epilogue < 0 || c->probe_epilogue == (epi == EPI_RESTRICT_ZERO ? EPI_RESTRICT : epi)) &&
                     (c->probe_precision == 0 || c->probe_precision == int(sizeof(TV)));
  if (probe) {
    cudaEvent_t e0 = probe_event(c);
    PM_CUDA(cudaEventRecord(e0, c->stream));
    c->probe_events.push_back(e0);
    c->probe_bytes.push_back(epi_bytes(A, epi, int(sizeof(TV)), n));
  }
  if constexpr (sizeof(TV) == 8) {
    if (c->sell_shape64 > 0 && A.sell64_ok && A.sell_lanes == c->sell_shape64 / 100 && A.n_slices > 0 &&
        n == A.n_rows) {
      launch_sell64(c, A, epi, reinterpret_cast<const double*>(x), reinterpret_cast<double*>(y),
                    reinterpret_cast<const double*>(b), reinterpret_cast<const double*>(diag), double(alpha));
      if (probe) {
        cudaEvent_t e1 = probe_event(c);
        PM_CUDA(cudaEventRecord(e1, c->stream));
        c->probe_events.push_back(e1);
      }
      return;
    }
  }
  if constexpr (sizeof(TV) == 4) {
    if (c->sell_shape > 0 && A.sell_lanes == c->sell_shape / 100 &&
        A.n_slices > 0 && n == A.n_rows) {
      launch_sell(c, A, epi, reinterpret_cast<const float*>(x), reinterpret_cast<float*>(y),
                  reinterpret_cast<const float*>(b), reinterpret_cast<const float*>(diag), float(alpha));
      if (probe) {
        cudaEvent_t e1 = probe_event(c);
        PM_CUDA(cudaEventRecord(e1, c->stream));
        c->probe_events.push_back(e1);
      }
      return;
    }
  }
  switch (epi) {
    case EPI_AXPY: launch_epi<TV, TX, TA, EPI_AXPY>(c, G, U, n, rp, ci, vals, x, y, b, diag, alpha, A.mask, rb, nrb); break;
    case EPI_SET: launch_epi<TV, TX, TA, EPI_SET>(c, G, U, n, rp, ci, vals, x, y, b, diag, alpha, A.mask, rb, nrb); break;
    case EPI_DEFECT: launch_epi<TV, TX, TA, EPI_DEFECT>(c, G, U, n, rp, ci, vals, x, y, b, diag, alpha, A.mask, rb, nrb); break;
    case EPI_JACOBI: launch_epi<TV, TX, TA, EPI_JACOBI>(c, G, U, n, rp, ci, vals, x, y, b, diag, alpha, A.mask, rb, nrb); break;
    case EPI_RESTRICT: launch_epi<TV, TX, TA, EPI_RESTRICT>(c, G, U, n, rp, ci, vals, x, y, b, diag, alpha, A.mask, rb, nrb); break;
    case EPI_PROLONG: launch_epi<TV, TX, TA, EPI_PROLONG>(c, G, U, n, rp, ci, vals, x, y, b, diag, alpha, A.mask, rb, nrb); break;
    case EPI_RESTRICT_ZERO: launch_epi<TV, TX, TA, EPI_RESTRICT_ZERO>(c, G, U, n, rp, ci, vals, x, y, b, diag, alpha, A.mask, rb, nrb); break;
    default: throw Error(PM_E_INVALID, "unknown SpMV epilogue");
  }
  if (probe) {
    cudaEvent_t e1 = probe_event(c);
    PM_CUDA(cudaEventRecord(e1, c->stream));
    c->probe_events.push_back(e1);
  }
}

void probe_reset(pm_ctx* c, int64_t nnz) {
  for (auto e : c->probe_events) c->probe_pool.push_back(e);
  c->probe_events.clear();
  c->probe_bytes.clear();
  c->probe_nnz = nnz;
}

void probe_result(pm_ctx* c, int* count, double* total_ms, double* total_bytes) {
  PM_CUDA(cudaStreamSynchronize(c->stream));
  const int pairs = int(c->probe_events.size() / 2);
  double ms = 0.0, bytes = 0.0;
  for (int i = 0; i < pairs; ++i) {
    float t = 0.0f;
    PM_CUDA(cudaEventElapsedTime(&t, c->probe_events[2 * i], c->probe_events[2 * i + 1]));
    ms += t;
    bytes += c->probe_bytes[i];
  }
  *count = pairs;
  *total_ms = ms;
  *total_bytes = bytes;
}

void csr_apply(pm_ctx* c, const DevCsr& A, int epi, const double* x, double* y, const double* b,
               double alpha, int n_rows_override) {
  if (epi == EPI_JACOBI && !A.diag.p) throw Error(PM_E_INVALID, "Jacobi sweep without diagonal");
  csr_dispatch<double, double, double>(c, A, A.vals.p, A.diag.p, epi, x, y, b, alpha,
                                       n_rows_override >= 0 ? n_rows_override : A.n_rows);
}

void csr_apply32(pm_ctx* c, const DevCsr& A, int epi, const float* x, float* y, const float* b,
                 float alpha, int n_rows_override) {
  if (!A.vals32.p && A.nnz) throw Error(PM_E_INVALID, "matrix has no FP32 copy");
  if (epi == EPI_JACOBI && !A.diag32.p) throw Error(PM_E_INVALID, "Jacobi sweep without FP32 diagonal");
  csr_dispatch<float, float, float>(c, A, A.vals32.p, A.diag32.p, epi, x, y, b, alpha,
                                    n_rows_override >= 0 ? n_rows_override : A.n_rows);
}

void csr_restrict_zero(pm_ctx* c, const DevCsr& R, const double* x, double* y, const double* d, double w, double* x0) {
  csr_dispatch<double, double, double>(c, R, R.vals.p, d, EPI_RESTRICT_ZERO, x, y, (const double*)x0, w, R.n_rows);
}
void csr_restrict_zero32(pm_ctx* c, const DevCsr& R, const float* x, float* y, const float* d, float w, float* x0) {
  if (!R.vals32.p && R.nnz) throw Error(PM_E_INVALID, "matrix has no FP32 copy");
  csr_dispatch<float, float, float>(c, R, R.vals32.p, d, EPI_RESTRICT_ZERO, x, y, (const float*)x0, w, R.n_rows);
}

// ------------------------------------------------------------------ BLAS-1 ---
// block-level sum with a fixed tree (deterministic)
__device__ __forceinline__ double block_sum(double v, double* sh) {
  const int t = threadIdx.x;
  sh[t] = v;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (t < s) sh[t] += sh[t + s];
    __syncthreads();
  }
  double r = sh[0];
  __syncthreads();
  return r;
}

template <class T>
__global__ void __launch_bounds__(256) k_dot_partials(int n, const T* __restrict__ x,
                                                      const T* __restrict__ y,
                                                      double* __restrict__ part) {
  __shared__ double sh[256];
  double s = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    s += double(x[i]) * double(y[i]);
  double r = block_sum(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = r;
}

__global__ void k_finish_sum(const double* __restrict__ part, int np, double* out, int take_sqrt) {
  __shared__ double sh[256];
  double s = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) s += part[i];
  double r = block_sum(s, sh);
  if (threadIdx.x == 0) *out = take_sqrt ? sqrt(r) : r;
}

void dot_partials(pm_ctx* c, int n, const double* x, const double* y, double* partials) {
  k_dot_partials<double><<<red_blocks(n), kRedThreads, 0, c->stream>>>(n, x, y, partials);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

void finish_sum(pm_ctx* c, int n, const double* partials, double* out, bool take_sqrt) {
  k_finish_sum<<<1, 256, 0, c->stream>>>(partials, red_blocks(n), out, take_sqrt ? 1 : 0);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

double dot_host(pm_ctx* c, int n, const double* x, const double* y) {
  dot_partials(c, n, x, y, c->partials.p);
  finish_sum(c, n, c->partials.p, c->dev_scalars.p, false);
  PM_CUDA(cudaMemcpyAsync(c->host_scalars, c->dev_scalars.p, sizeof(double),
                          cudaMemcpyDeviceToHost, c->stream));
  PM_CUDA(cudaStreamSynchronize(c->stream));
  return c->host_scalars[0];
}

template <class T>
__global__ void k_copy(long long n, const T* __restrict__ x, T* __restrict__ y) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] = x[i];
}
__global__ void k_set(long long n, double* __restrict__ y, double v) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] = v;
}
__global__ void k_scale(long long n, double* __restrict__ y, double a) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] *= a;
}
__global__ void k_axpy(long long n, double a, const double* __restrict__ x, double* __restrict__ y) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] += a * x[i];
}
__global__ void k_axpby(long long n, double a, const double* __restrict__ x, double b,
                        double* __restrict__ y) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] = a * x[i] + b * y[i];
}
__global__ void k_div(long long n, const double* __restrict__ d, double* __restrict__ y) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] /= d[i];
}
#define PM_LAUNCH1D(kern, n, ...)                                                     \
  do {                                                                                \
    if ((n) > 0) launch_k(c, kern, dim3(grid_for(c, (n))), dim3(256), 0, __VA_ARGS__); \
  } while (0)

void vcopy(pm_ctx* c, int n, const double* x, double* y) { PM_LAUNCH1D(k_copy<double>, n, n, x, y); }
void vset(pm_ctx* c, int n, double* y, double v) { PM_LAUNCH1D(k_set, n, n, y, v); }
void vscale(pm_ctx* c, int n, double* y, double a) { PM_LAUNCH1D(k_scale, n, n, y, a); }
void vaxpy(pm_ctx* c, int n, double a, const double* x, double* y) { PM_LAUNCH1D(k_axpy, n, n, a, x, y); }
void vaxpby(pm_ctx* c, int n, double a, const double* x, double b, double* y) {
  PM_LAUNCH1D(k_axpby, n, n, a, x, b, y);
}
void vdiv(pm_ctx* c, int n, const double* d, double* y) { PM_LAUNCH1D(k_div, n, n, d, y); }
void vcvt_d2f(pm_ctx* c, int n, const double* x, float* y) { PM_LAUNCH1D(k_d2f, n, n, x, y); }
void vcvt_f2d(pm_ctx* c, int n, const float* x, double* y) { PM_LAUNCH1D(k_f2d, n, n, x, y); }
__global__ void k_copy_nonactive(int n, BlockMask m, const double* __restrict__ src, double* __restrict__ dst) {
  pdl_enter();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (!row_is_active(m, i)) dst[i] = src[i];
}
void copy_nonactive(pm_ctx* c, int n, const BlockMask& m, const double* src, double* dst) {
  PM_LAUNCH1D(k_copy_nonactive, n, n, m, src, dst);
}

// flag := 1 if a non-active entry of x is not zero
__global__ void k_nonactive_nonzero(BlockMask m, const double* __restrict__ x, int* __restrict__ flag) {
  for (int b = 0; b < m.nb; ++b)
    for (int i = m.active_end[b] + blockIdx.x * blockDim.x + threadIdx.x; i < m.end[b];
         i += gridDim.x * blockDim.x)
      if (x[i] != 0.0) *flag = 1;
}
void nonactive_nonzero(pm_ctx* c, const BlockMask& m, const double* x, int* flag) {
  k_nonactive_nonzero<<<kRedBlocks, 256, 0, c->stream>>>(m, x, flag);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

// x = 0 + w ((b - 0) / d) is the damped Jacobi sweep of an exactly zero iterate (the
// sweep's row sums of a_ij * 0 are +0; fma(w, q, +0) rounds like its x + w q with
// x = +0).
// set_finest_rhs and the first step of the cycle in one launch (a conversion, an
// initialisation and, from zero, a diagonal scaling were three)
template <class T>
__global__ void k_cycle_start(int n, BlockMask m, const double* __restrict__ in, T* __restrict__ rhs,
                              T* __restrict__ x, const T* __restrict__ d, T w, int zero) {
  pdl_enter();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const T r = T(in[i]);
    rhs[i] = r;
    x[i] = zero ? fmadd(w, (r - T(0)) / d[i], T(0)) : row_is_active(m, i) ? T(0) : r;
  }
}
template <class T>
void cycle_start(pm_ctx* c, int n, const BlockMask& m, const double* in, T* rhs, T* x, const T* d, T w, bool zero) {
  PM_LAUNCH1D(k_cycle_start<T>, n, n, m, in, rhs, x, d, w, zero ? 1 : 0);
}
template void cycle_start<float>(pm_ctx*, int, const BlockMask&, const double*, float*, float*, const float*, float,
                                 bool);
template void cycle_start<double>(pm_ctx*, int, const BlockMask&, const double*, double*, double*, const double*,
                                  double, bool);
// ------------------------------------------------------------ SOR ----------
void SorColours::build(pm_ctx* c, const DevCsr& A) {
  if (key == A.row_ptr.p && key_nnz == A.nnz) return;
  const int n = A.n_rows;
  if (A.n_cols != n) throw Error(PM_E_INVALID, "SOR needs a square matrix");
  std::vector<int> rp(static_cast<size_t>(n) + 1), ci(static_cast<size_t>(A.nnz));
  PM_CUDA(cudaMemcpyAsync(rp.data(), A.row_ptr.p, rp.size() * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  if (A.nnz)
    PM_CUDA(cudaMemcpyAsync(ci.data(), A.cols.p, ci.size() * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  PM_CUDA(cudaStreamSynchronize(c->stream));
  // the transposed pattern: rows k that store column i
  std::vector<int> tp(static_cast<size_t>(n) + 1, 0), tc(ci.size());
  for (int k : ci) tp[size_t(k) + 1]++;
  for (int i = 0; i < n; ++i) tp[size_t(i) + 1] += tp[size_t(i)];
  std::vector<int> fill(tp.begin(), tp.end() - 1);
  for (int i = 0; i < n; ++i)
    for (int k = rp[size_t(i)]; k < rp[size_t(i) + 1]; ++k) tc[size_t(fill[size_t(ci[size_t(k)])]++)] = i;
  std::vector<int> colour(static_cast<size_t>(n), -1), stamp;
  int n_col = 0;
  for (int i = 0; i < n; ++i) {
    auto mark = [&](int j) {
      if (j < i && j != i) {
        const int cj = colour[size_t(j)];
        if (cj >= int(stamp.size())) stamp.resize(size_t(cj) + 1, -1);
        stamp[size_t(cj)] = i;
      }
    };
    for (int k = rp[size_t(i)]; k < rp[size_t(i) + 1]; ++k) mark(ci[size_t(k)]);
    for (int k = tp[size_t(i)]; k < tp[size_t(i) + 1]; ++k) mark(tc[size_t(k)]);
    int cc = 0;
    while (cc < int(stamp.size()) && stamp[size_t(cc)] == i) ++cc;
    colour[size_t(i)] = cc;
    n_col = std::max(n_col, cc + 1);
  }
  ptr.assign(size_t(n_col) + 1, 0);
  for (int i = 0; i < n; ++i) ptr[size_t(colour[size_t(i)]) + 1]++;
  for (int k = 0; k < n_col; ++k) ptr[size_t(k) + 1] += ptr[size_t(k)];
  std::vector<int> order(static_cast<size_t>(n)), pos(ptr.begin(), ptr.end() - 1);
  for (int i = 0; i < n; ++i) order[size_t(pos[size_t(colour[size_t(i)])]++)] = i;
  rows.upload(order, c->stream);
  PM_CUDA(cudaStreamSynchronize(c->stream));
  key = A.row_ptr.p;
  key_nnz = A.nnz;
}

void sor_check_diagonal(pm_ctx* c, const DevCsr& A) {
  if (!A.diag.p) throw Error(PM_E_INVALID, "SOR check without diagonal");
  std::vector<double> d(static_cast<size_t>(A.n_rows));
  if (!d.empty())
    PM_CUDA(cudaMemcpyAsync(d.data(), A.diag.p, d.size() * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  PM_CUDA(cudaStreamSynchronize(c->stream));
  for (double v : d)
    if (v == 0.0) throw Error(PM_E_INVALID, "There is a zero on the diagonal. You can not use `sor` in this case");
}

// x_row += omega (b_row - sum_k a_row,k x_k) / d_row for the rows of one
// colour, G lanes per row (they do not couple, so x is updated in place)
template <class T, int G>
__global__ void __launch_bounds__(256) k_sor_rows(int cnt, const int* __restrict__ rows, const int* __restrict__ rp,
                                                  const int* __restrict__ ci, const T* __restrict__ v,
                                                  const T* __restrict__ d, const T* __restrict__ b, T* x, T omega,
                                                  const int* __restrict__ guard) {
  if (guarded(guard)) return;  // uniform for the whole grid
  const int lane = threadIdx.x & (G - 1);
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const bool valid = q < cnt;
  const int row = valid ? __ldg(rows + q) : 0;
  const int beg = valid ? __ldg(rp + row) : 0;
  const int end = valid ? __ldg(rp + row + 1) : 0;
  T s = T(0);
  for (int k = beg + lane; k < end; k += G) s += __ldg(v + k) * x[__ldg(ci + k)];
#pragma unroll
  for (int off = G / 2; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off, G);
  if (valid && lane == 0) x[row] = x[row] + omega * (b[row] - s) / d[row];
}

template <class T>
static void sor_sweep_t(pm_ctx* c, const DevCsr& A, const T* vals, const T* diag, const SorColours& col, const T* b,
                        T* x, T omega, bool backward) {
  if (!diag) throw Error(PM_E_INVALID, "SOR sweep without diagonal");
  if (col.ptr.empty() || col.key != A.row_ptr.p) throw Error(PM_E_INVALID, "SOR sweep without the matrix's colours");
  const int nc = int(col.ptr.size()) - 1;
  const bool wide = A.nnz > 16 * int64_t(A.n_rows);
  for (int q = 0; q < nc; ++q) {
    const int k = backward ? nc - 1 - q : q;
    const int cnt = col.ptr[size_t(k) + 1] - col.ptr[size_t(k)];
    if (!cnt) continue;
    const int* rows = col.rows.p + col.ptr[size_t(k)];
    if (wide)
      k_sor_rows<T, 8><<<nblocks((long long)cnt * 8, 256), 256, 0, c->stream>>>(
          cnt, rows, A.row_ptr.p, A.cols.p, vals, diag, b, x, omega, c->guard);
    else
      k_sor_rows<T, 4><<<nblocks((long long)cnt * 4, 256), 256, 0, c->stream>>>(
          cnt, rows, A.row_ptr.p, A.cols.p, vals, diag, b, x, omega, c->guard);
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
  }
}

void sor_sweep(pm_ctx* c, const DevCsr& A, const SorColours& col, const double* b, double* x, double omega,
               bool backward) {
  sor_sweep_t<double>(c, A, A.vals.p, A.diag.p, col, b, x, omega, backward);
}
void sor_sweep32(pm_ctx* c, const DevCsr& A, const SorColours& col, const float* b, float* x, float omega,
                 bool backward) {
  if (!A.vals32.p) throw Error(PM_E_INVALID, "matrix has no FP32 copy");
  sor_sweep_t<float>(c, A, A.vals32.p, A.diag32.p, col, b, x, omega, backward);
}

// ------------------------------------------------------- dense inverse ------
// the active block as a dense row-major matrix, one warp per row
template <class T>
__global__ void __launch_bounds__(256) k_dense_fill(int na, const int* __restrict__ act, const int* __restrict__ pos,
                                                    const int* __restrict__ rp, const int* __restrict__ ci,
                                                    const double* __restrict__ v, T* __restrict__ M) {
  const int ia = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (ia >= na) return;
  const int i = act[ia];
  T* row = M + (size_t)ia * na;
  for (int j = lane; j < na; j += 32) row[j] = T(0);
  __syncwarp();
  for (int k = rp[i] + lane; k < rp[i + 1]; k += 32) {
    const int jp = pos[ci[k]];
    if (jp >= 0) row[jp] = T(v[k]);
  }
}

// pivot search, row swap and pivot-row scaling of Gauss-Jordan step k
__global__ void __launch_bounds__(256) k_gj_pivot(int na, int k, double* __restrict__ M,
                                                  int* __restrict__ perm, double* __restrict__ colk,
                                                  int* __restrict__ flag) {
  __shared__ double sv[256];
  __shared__ int si[256];
  const int t = threadIdx.x;
  double best = -1.0;
  int bi = na;
  for (int i = k + t; i < na; i += blockDim.x) {
    const double a = fabs(M[(size_t)i * na + k]);
    if (a > best) { best = a; bi = i; }
  }
  sv[t] = best;
  si[t] = bi;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (t < s) {
      if (sv[t + s] > sv[t] || (sv[t + s] == sv[t] && si[t + s] < si[t])) {
        sv[t] = sv[t + s];
        si[t] = si[t + s];
      }
    }
    __syncthreads();
  }
  const int p = si[0];
  const bool singular = !(sv[0] > 0.0);
  if (t == 0) {
    perm[k] = singular ? k : p;
    if (singular) *flag = 1;
  }
  if (!singular && p != k)
    for (int j = t; j < na; j += blockDim.x) {
      double a = M[(size_t)k * na + j];
      M[(size_t)k * na + j] = M[(size_t)p * na + j];
      M[(size_t)p * na + j] = a;
    }
  __syncthreads();
  const double piv = singular ? 1.0 : M[(size_t)k * na + k];
  for (int i = t; i < na; i += blockDim.x) {
    colk[i] = (i == k) ? 0.0 : M[(size_t)i * na + k];
  }
  __syncthreads();
  for (int i = t; i < na; i += blockDim.x)
    if (i != k) M[(size_t)i * na + k] = 0.0;
  __syncthreads();
  if (t == 0) M[(size_t)k * na + k] = 1.0;
  __syncthreads();
  for (int j = t; j < na; j += blockDim.x) M[(size_t)k * na + j] /= piv;
}

__global__ void k_gj_update(int na, int k, double* __restrict__ M, const double* __restrict__ colk) {
  const long long total = (long long)na * na;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = int(e / na), j = int(e % na);
    if (i == k) continue;
    const double f = colk[i];
    if (f != 0.0) M[e] -= f * M[(size_t)k * na + j];
  }
}

__global__ void k_gj_unswap(int na, double* __restrict__ M, const int* __restrict__ perm) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= na) return;
  double* row = M + (size_t)i * na;
  for (int k = na - 1; k >= 0; --k) {
    const int p = perm[k];
    if (p != k) {
      double a = row[k];
      row[k] = row[p];
      row[p] = a;
    }
  }
}

// The whole Gauss-Jordan elimination in one cooperative launch (all blocks
// resident; cooperative_groups grid barriers, two per column). Every block owns
// a contiguous range of rows. Step k: every block reduces the per-block
// partial arg-max of column k in the same fixed order (largest magnitude, the
// smallest row on ties: the pivot rule of k_gj_pivot), then writes its share of
// the scaled pivot row, the old row k and the column multipliers; after the
// barrier each block eliminates its own rows and records the partial arg-max
// of column k+1. The values are those of k_gj_pivot + k_gj_update (same
// operations per entry), without 2 launches per column.
__global__ void __launch_bounds__(256) k_gj_coop(int na, double* __restrict__ M, int* __restrict__ perm,
                                                 double* __restrict__ rowk, double* __restrict__ oldk,
                                                 double* __restrict__ colk, double* __restrict__ part_v,
                                                 int* __restrict__ part_i, int* __restrict__ flag) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  __shared__ double sv[256];
  __shared__ int si[256];
  __shared__ int s_p;
  __shared__ double s_pv;
  const int t = threadIdx.x, nb = gridDim.x, b = blockIdx.x;
  const int per = (na + nb - 1) / nb;
  const int r0 = min(na, b * per), r1 = min(na, r0 + per);
  auto block_argmax = [&](int col, int from) {
    double best = -1.0;
    int bi = na;
    for (int i = max(r0, from) + t; i < r1; i += blockDim.x) {
      const double a = fabs(M[(size_t)i * na + col]);
      if (a > best) { best = a; bi = i; }
    }
    sv[t] = best;
    si[t] = bi;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
      if (t < s && (sv[t + s] > sv[t] || (sv[t + s] == sv[t] && si[t + s] < si[t]))) {
        sv[t] = sv[t + s];
        si[t] = si[t + s];
      }
      __syncthreads();
    }
    if (t == 0) {
      part_v[b] = sv[0];
      part_i[b] = si[0];
    }
  };
  block_argmax(0, 0);
  for (int k = 0; k < na; ++k) {
    grid.sync();
    // pivot of column k: the same reduction in every block
    if (t == 0) {
      double best = -1.0;
      int bi = na;
      for (int q = 0; q < nb; ++q)
        if (part_v[q] > best || (part_v[q] == best && part_i[q] < bi)) {
          best = part_v[q];
          bi = part_i[q];
        }
      const bool singular = !(best > 0.0);
      s_p = singular ? k : bi;
      s_pv = singular ? 1.0 : M[(size_t)bi * na + k];
      if (b == 0) {
        perm[k] = s_p;
        if (singular) *flag = 1;
      }
    }
    __syncthreads();
    const int p = s_p;
    const double pv = s_pv;
    // scaled pivot row, old row k and the multipliers (rows after the swap)
    for (int e = b * blockDim.x + t; e < na; e += nb * blockDim.x) {
      rowk[e] = (e == k ? 1.0 : M[(size_t)p * na + e]) / pv;
      oldk[e] = M[(size_t)k * na + e];
      colk[e] = (e == p && p != k) ? M[(size_t)k * na + k] : M[(size_t)e * na + k];
    }
    grid.sync();
    // elimination of this block's rows
    const long long cnt = (long long)(r1 - r0) * na;
    for (long long e = t; e < cnt; e += blockDim.x) {
      const int i = r0 + int(e / na), j = int(e % na);
      double* Mi = M + (size_t)i * na;
      if (i == k) {
        Mi[j] = rowk[j];
      } else {
        const double base = (i == p && p != k) ? oldk[j] : Mi[j];
        const double f = colk[i];
        Mi[j] = (j == k ? 0.0 : base) - f * rowk[j];
      }
    }
    __syncthreads();
    if (k + 1 < na) block_argmax(k + 1, k + 1);
  }
}

// Arg-max with the pivot rule of k_gj_pivot (the largest |a|, the smallest
// position on ties, NaN never) on the bits of |a| as integers: three warp
// reductions of 32-bit words. Compared as FP64 numbers in shuffle steps, the
// search took longer than the elimination step (FP64 compares run on the FP64
// pipe too).
__device__ __forceinline__ unsigned long long gj_key(double a) {
  const unsigned long long k = (unsigned long long)__double_as_longlong(fabs(a));
  return k > 0x7ff0000000000000ull ? 0ull : k;
}
__device__ __forceinline__ unsigned long long gj_key(float a) {
  const unsigned k = __float_as_uint(fabsf(a));
  return k > 0x7f800000u ? 0ull : (unsigned long long)k;
}
template <bool WIDE>  // WIDE: 64-bit keys
__device__ __forceinline__ void gj_warp_best(unsigned long long& key, int& pos, int none) {
  if (WIDE) {
    const unsigned hi = unsigned(key >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? unsigned(key) : 0u);
    const unsigned long long best = ((unsigned long long)mh << 32) | ml;
    pos = __reduce_min_sync(0xffffffffu, key == best ? pos : none);
    key = best;
  } else {
    const unsigned best = __reduce_max_sync(0xffffffffu, unsigned(key));
    pos = __reduce_min_sync(0xffffffffu, unsigned(key) == best ? pos : none);
    key = best;
  }
}

// Blocked Gauss-Jordan inverse with partial pivoting, in panels of NB columns K:
// two launches per panel, the matrix before and after a panel in two buffers.
//
// k_gj_panel: one block runs the NB elimination steps on the panel's columns of
// the rows that can still be pivots (position k0 on). Every thread keeps RPT
// rows of the panel in registers; a step takes two block barriers (the arg-max
// over the warps' candidates; the scaled pivot row and the row it displaces
// through shared memory). It leaves D = P^-1 (P: the pivot rows' block of the
// panel), prm = the row at every position after the panel's swaps, and rowsrc =
// the composition of all swaps so far.
// k_gj_apply, on all SMs: the panel's columns become D in the panel's rows and W
// elsewhere (W = -M_K D, by the panel's elimination steps on every row: formed
// from D itself it loses accuracy with the condition of P), the others src(prm)
// (panel rows: 0) + (D | W) * (pivot rows of src); after the last panel the
// columns go where the row swaps belong in the inverse (out[i][rowsrc[j]]).
//
// Both are launched early and read what the launch before them writes (the matrix,
// D, prm, rowsrc): plain pointers, no trigger before the wait.
//
// The chain of columns bounds it. A thread-block cluster with one cluster
// barrier and one remote row per column took 4 to 8 us per column.
// Update of a two-level solver (the rest of it takes about 85 us), cluster or
// row-resident kernel before and now: 225 rows 1,444 and 496 us in FP64, 901 and
// 304 in FP32; 343 rows 2,977 and 893, 1,763 and 444; 729 rows 6,868 and 3,449
// in FP64; 1,331 rows 20.8 and 13.7 ms; 2,197 rows (column by column) 190 and 48.
constexpr int kGjMaxRows = 4096;

template <class T, int NB, int RPT>
__global__ void __launch_bounds__(1024) k_gj_panel(int n, int k0, int nb, const T* M, T* D, T* steps, int* prm,
                                                   int* rowsrc, int* flag) {
  constexpr bool WIDE = sizeof(T) == 8;
  // by the parity of the step: the warps' candidates (key, position, row) and
  // the row at the step's position
  __shared__ __align__(16) T cand[2][32][NB], orow[2][NB];
  __shared__ unsigned long long wkey[2][32];
  __shared__ int wpos[2][32];
  extern __shared__ int sp[];  // row at each position
  const int t = threadIdx.x, bd = blockDim.x, lane = t & 31, warp = t >> 5, nw = bd >> 5;
  pdl_wait();
  pdl_trigger();
  T row[RPT][NB];
#pragma unroll
  for (int s = 0; s < RPT; ++s) {
    const int r = k0 + t + s * bd;
#pragma unroll
    for (int j = 0; j < NB; ++j) row[s][j] = (r < n && j < nb) ? M[(size_t)r * n + k0 + j] : T(0);
  }
  for (int r = t; r < n; r += bd) sp[r] = r;
  // The columns rotate by one place per step, so that the step's column is
  // always row[s][0] and the loop body stays rolled (unrolled over the steps, the
  // panel took 2 us per column fetching instructions); NB rotations put them back.
#pragma unroll 1
  for (int k = 0; k < NB; ++k) {
    if (k >= nb) {  // uniform: the last panel's missing columns
#pragma unroll
      for (int s = 0; s < RPT; ++s) {
        const T first = row[s][0];
#pragma unroll
        for (int j = 1; j < NB; ++j) row[s][j - 1] = row[s][j];
        row[s][NB - 1] = first;
      }
      continue;
    }
    const int kk = k0 + k, buf = k & 1;
    unsigned long long key = 0;
    int p = n;
#pragma unroll
    for (int s = 0; s < RPT; ++s) {
      const int r = k0 + t + s * bd;
      const unsigned long long a = gj_key(row[s][0]);
      if (r >= kk && r < n && (a > key || p == n)) {  // rows in increasing order: ties keep the smaller
        key = a;
        p = r;
      }
    }
    gj_warp_best<WIDE>(key, p, n);
#pragma unroll
    for (int s = 0; s < RPT; ++s) {
      const int r = k0 + t + s * bd;
      if (r == p) {
        wkey[buf][warp] = key;
        wpos[buf][warp] = p;
#pragma unroll
        for (int j = 0; j < NB; ++j) cand[buf][warp][j] = row[s][j];
      }
      if (r == kk)
#pragma unroll
        for (int j = 0; j < NB; ++j) orow[buf][j] = row[s][j];
    }
    if (p == n && lane == 0) {  // no candidate in this warp
      wkey[buf][warp] = 0;
      wpos[buf][warp] = n;
    }
    // one barrier per step: the buffers of step k are written again at step
    // k + 2, after the barrier of step k + 1, which every thread reaches only
    // when it has read them
    __syncthreads();
    key = lane < nw ? wkey[buf][lane] : 0;
    p = lane < nw ? wpos[buf][lane] : n;
    gj_warp_best<WIDE>(key, p, n);
    const bool singular = key == 0;
    if (singular) p = kk;
    const T* pr = singular ? orow[buf] : cand[buf][((p - k0) % bd) >> 5];
    const T rpv = T(1) / (singular ? T(1) : pr[0]);
    // the step for the other rows: the pivot row, its reciprocal on the diagonal
    if (t < NB) steps[k * NB + (k + t) % NB] = t == 0 ? rpv : pr[t];
    if (t == 0) {
      const int a = sp[kk];
      sp[kk] = sp[p];
      sp[p] = a;
      if (singular) *flag = 1;
    }
#pragma unroll
    for (int s = 0; s < RPT; ++s) {
      const int r = k0 + t + s * bd;
      if (r == p && p != kk)  // the displaced row moves here
#pragma unroll
        for (int j = 0; j < NB; ++j) row[s][j] = orow[buf][j];
      // the pivot row becomes 0 + rpv (pivot row), column k of every row -g
      T g = row[s][0] * rpv;
      if (r == kk) {
        g = -rpv;
#pragma unroll
        for (int j = 1; j < NB; ++j) row[s][j] = T(0);
      }
#pragma unroll
      for (int j = 1; j < NB; ++j) row[s][j - 1] = row[s][j] - g * pr[j];
      row[s][NB - 1] = -g;
    }
  }
  __syncthreads();
  if (t < nb)  // positions k0 .. k0 + nb - 1 belong to the first threads
#pragma unroll
    for (int j = 0; j < NB; ++j) D[t * NB + j] = j < nb ? row[0][j] : T(0);
  // the swaps touch positions from k0 on; every thread reads its old entries
  // before the barrier and writes after it
  int from[RPT];
#pragma unroll
  for (int s = 0; s < RPT; ++s) {
    const int r = k0 + t + s * bd;
    from[s] = r >= n ? 0 : k0 == 0 ? sp[r] : rowsrc[sp[r]];
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < RPT; ++s)
    if (k0 + t + s * bd < n) rowsrc[k0 + t + s * bd] = from[s];
  for (int r = t; r < n; r += bd) prm[r] = sp[r];
}

// TR x 32 tile per block of 32 x 8 threads; cols: the last panel's column map
template <class T, int NB, int TR>
__global__ void __launch_bounds__(256) k_gj_apply(int n, int k0, int nb, const T* src, const T* D, const T* steps,
                                                  const int* prm, const int* cols, T* dst) {
  constexpr int QR = TR / 8;
  static_assert(256 % NB == 0 && NB <= 32 && (TR * NB) % 32 == 0, "one thread per panel entry, rows within a warp");
  __shared__ T w[TR][NB + 1], piv[NB][32], st[NB][NB];
  const int tx = threadIdx.x, ty = threadIdx.y, t = ty * 32 + tx;
  const int i0 = blockIdx.y * TR, j = blockIdx.x * 32 + tx;
  pdl_wait();
  pdl_trigger();
  for (int e = t; e < NB * NB; e += 256) st[e / NB][e % NB] = e / NB < nb ? steps[e] : T(0);
  for (int l = ty; l < NB; l += 8) piv[l][tx] = (l < nb && j < n) ? src[(size_t)prm[k0 + l] * n + j] : T(0);
  T acc[QR];
#pragma unroll
  for (int q = 0; q < QR; ++q) {
    const int i = i0 + ty + 8 * q;
    acc[q] = (i < n && j < n && (i < k0 || i >= k0 + nb)) ? src[(size_t)prm[i] * n + j] : T(0);
  }
  __syncthreads();
  // the panel's steps on the tile's rows, one thread per entry; the panel's own
  // rows come from k_gj_panel
  for (int e = t; e < TR * NB; e += 256) {
    const int r = e / NB, l = e % NB, i = i0 + r;
    T v = (i < n && l < nb) ? src[(size_t)prm[i] * n + k0 + l] : T(0);
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      const T g = __shfl_sync(0xffffffffu, v, k, NB) * st[k][k];
      if (k < nb) v = l == k ? -g : v - g * st[k][l];
    }
    w[r][l] = (i >= k0 && i < k0 + nb) ? D[(i - k0) * NB + l] : v;
  }
  __syncthreads();
  if (j >= n) return;
  const bool own = j >= k0 && j < k0 + nb;  // a column of the panel
  const int jo = cols ? cols[j] : j;
#pragma unroll
  for (int q = 0; q < QR; ++q) {
    const int r = ty + 8 * q, i = i0 + r;
    if (i >= n) continue;
    T s = acc[q];
    if (own) {
      s = w[r][j - k0];
    } else {
#pragma unroll
      for (int l = 0; l < NB; ++l) s += w[r][l] * piv[l][tx];
    }
    dst[(size_t)i * n + jo] = s;
  }
}

// the matrix of gj_panels goes from buffer to buffer, panel by panel, so that the last
// panel writes `out`: where it starts (a third buffer of n x n held 134 MB more at
// 4,096 rows, for the solver's life)
template <class T>
static T* gj_start(int n, int width, T* work, T* out) { return ((n + width - 1) / width) % 2 ? work : out; }

// the matrix in gj_start(n, NB, work, out); d: the panel, behind the n x n of work
template <class T, int NB, int RPT, int TR>
static void gj_panels(pm_ctx* c, int n, T* work, int* prm, int* rowsrc, int* flag, T* out) {
  T *a = gj_start(n, NB, work, out), *b = a == work ? out : work, *d = work + size_t(n) * n;
  const dim3 grid((n + 31) / 32, (n + TR - 1) / TR), block(32, 8);
  const size_t smem = size_t(n) * sizeof(int);
  for (int k0 = 0; k0 < n; k0 += NB) {
    const int nb = std::min(NB, n - k0), rows = n - k0;
    const bool last = k0 + nb == n;
    if (rows <= 1024)
      launch_pdl(c, k_gj_panel<T, NB, 1>, dim3(1), dim3((rows + 31) & ~31), smem, n, k0, nb, a, d, d + NB * NB, prm, rowsrc,
                 flag);
    else if (RPT > 1 && rows <= 2048)
      launch_pdl(c, k_gj_panel<T, NB, (RPT > 1 ? RPT / 2 : 1)>, dim3(1), dim3(1024), smem, n, k0, nb, a, d, d + NB * NB, prm, rowsrc,
                 flag);
    else
      launch_pdl(c, k_gj_panel<T, NB, RPT>, dim3(1), dim3(1024), smem, n, k0, nb, a, d, d + NB * NB, prm, rowsrc,
                 flag);
    launch_pdl(c, k_gj_apply<T, NB, TR>, grid, block, 0, n, k0, nb, a, d, d + NB * NB, prm,
               last ? rowsrc : nullptr, b);
    std::swap(a, b);
  }
}

// Panel widths, by the same update: FP64 343 rows 910 / 822 / 962 us with 4 / 8 /
// 16 columns (a step's FP64 work grows with the width, the launches fall with
// it); FP32 469 / 416 / 459 us with 8 / 16 / 32 (with W formed from D).
constexpr int kGjWidth32 = 16, kGjWidth64 = 8;
static void gj_inverse(pm_ctx* c, int n, float* work, int* prm, int* rowsrc, int* flag, float* out) {
  gj_panels<float, kGjWidth32, 1, 16>(c, n, work, prm, rowsrc, flag, out);
}
static void gj_inverse(pm_ctx* c, int n, double* work, int* prm, int* rowsrc, int* flag, double* out) {
  gj_panels<double, kGjWidth64, 4, 16>(c, n, work, prm, rowsrc, flag, out);
}

__global__ void k_coarse_gemv32(int n, int na, const int* __restrict__ act, const int* __restrict__ pos,
                                const float* __restrict__ inv, const float* __restrict__ b,
                                float* __restrict__ x) {
  pdl_enter();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp < na) {
    const float* row = inv + (size_t)warp * na;
    float s = 0.0f;
    for (int j = lane; j < na; j += 32) s += row[j] * b[act[j]];
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) x[act[warp]] = s;
  } else {
    const int t = (warp - na) * 32 + lane;
    if (t < n && pos[t] < 0) x[t] = b[t];
  }
}

// the mixed cycle's coarse solve with the FP64 inverse: FP32 right-hand
// side and iterate, FP64 inverse entries and FP64 accumulation (the split
// of the outer solve: FP64 for the coarse-grid direct solve)
__global__ void k_coarse_gemv_mixed(int n, int na, const int* __restrict__ act, const int* __restrict__ pos,
                                    const double* __restrict__ inv, const float* __restrict__ b,
                                    float* __restrict__ x) {
  pdl_enter();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp < na) {
    const double* row = inv + (size_t)warp * na;
    double s = 0.0;
    for (int j = lane; j < na; j += 32) s = fma(row[j], double(b[act[j]]), s);
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) x[act[warp]] = float(s);
  } else {
    const int t = (warp - na) * 32 + lane;
    if (t < n && pos[t] < 0) x[t] = b[t];
  }
}

// launches go to another stream for the lifetime of the object
struct StreamSwap {
  pm_ctx* c;
  cudaStream_t saved;
  StreamSwap(pm_ctx* c_, cudaStream_t s_) : c(c_), saved(c_->stream) { c->stream = s_; }
  ~StreamSwap() { c->stream = saved; }
};

void DenseInverse::solve_mixed(pm_ctx* c, const float* b, float* x) {
  if (!has64) throw Error(PM_E_INVALID, "coarse solve before the FP64 inverse was built");
  const long long threads = (long long)na * 32 + n;
  launch_k(c, k_coarse_gemv_mixed, dim3(nblocks(threads, 256)), dim3(256), 0, n, na, (const int*)act.p,
           (const int*)pos.p, (const double*)inv.p, b, x);
}

void DenseInverse::build32(pm_ctx* c, const DevCsr& A) {
  launch32(c, A, c->stream);
  complete32(c, A);
}

// the active rows that the FP32 inverse is computed for in FP32; larger ones
// take the FP64 inverse, rounded
constexpr int kGjRows32 = 640;

void DenseInverse::launch32(pm_ctx* c, const DevCsr& A, cudaStream_t s) {
  pending32 = false;
  set_rows(c, A);
  if (na == 0 || na > kGjRows32) {
    build(c, A);
    inv32.ensure(size_t(na) * na);
    if (na) {
      k_d2f<<<grid_for(c, (long long)na * na), 256, 0, c->stream>>>((long long)na * na, inv.p, inv32.p);
      PM_CHECK_LAUNCH();
      c->kernel_launches++;
    }
    has32 = true;
    return;
  }
  // the preparation and the kernels on stream s (restored on every exit)
  StreamSwap swap(c, s);
  const size_t nn = size_t(na) * na;
  inv32.ensure(nn);
  work32.ensure(nn + 2 * kGjWidth32 * kGjWidth32);
  prepare(c, A, gj_start(na, kGjWidth32, work32.p, inv32.p));
  gj_inverse(c, na, work32.p, perm.p, perm.p + na, flag.p, inv32.p);
  if (!done_event) PM_CUDA(cudaEventCreateWithFlags(&done_event, cudaEventDisableTiming));
  PM_CUDA(cudaEventRecord(done_event, s));
  pending32 = true;
}

void DenseInverse::complete32(pm_ctx* c, const DevCsr& A) {
  if (!pending32) return;  // done at launch (large matrices) or nothing queued
  pending32 = false;
  int h_flag = 0;
  PM_CUDA(cudaStreamWaitEvent(c->stream, done_event, 0));
  PM_CUDA(cudaMemcpyAsync(&h_flag, flag.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  PM_CUDA(cudaStreamSynchronize(c->stream));
  if (h_flag) {
    // no FP32 pivot (a singular matrix, or values beyond the FP32 range): the
    // FP64 inverse decides (and throws if the matrix is singular), rounded
    build(c, A);
    if (na) {
      k_d2f<<<grid_for(c, (long long)na * na), 256, 0, c->stream>>>((long long)na * na, inv.p, inv32.p);
      PM_CHECK_LAUNCH();
      c->kernel_launches++;
    }
    has32 = true;
    return;
  }
  has32 = true;
}

void DenseInverse::solve32(pm_ctx* c, const float* b, float* x) {
  if (!has32) throw Error(PM_E_INVALID, "coarse FP32 inverse used before build32");
  const long long threads = (long long)(na + (n + 31) / 32) * 32;
  launch_k(c, k_coarse_gemv32, dim3(nblocks(threads, 256)), dim3(256), 0, n, na, (const int*)act.p,
             (const int*)pos.p, (const float*)inv32.p, b, x);
}

// the active rows depend on the block layout only; kept until it changes
void DenseInverse::set_rows(pm_ctx* c, const DevCsr& A) {
  bool same = act_set && n == A.n_rows && rows_of.nb == A.mask.nb;
  for (int b = 0; same && b < A.mask.nb; ++b)
    same = rows_of.start[b] == A.mask.start[b] && rows_of.active_end[b] == A.mask.active_end[b] &&
           rows_of.end[b] == A.mask.end[b];
  if (same) return;
  act_set = false;
  n = A.n_rows;
  std::vector<int> h_act, h_pos(n, -1);
  for (int i = 0; i < n; ++i) {
    bool active = false;
    for (int b = 0; b < A.mask.nb; ++b)
      if (i >= A.mask.start[b] && i < A.mask.end[b]) active = i < A.mask.active_end[b];
    if (active) {
      h_pos[i] = int(h_act.size());
      h_act.push_back(i);
    }
  }
  na = int(h_act.size());
  if (na > 20000) throw Error(PM_E_UNSUPPORTED, "coarse direct solve limited to 20000 active rows");
  act.upload(h_act, c->stream);
  pos.upload(h_pos, c->stream);
  tmp.ensure(std::max(na, 1));
  perm.ensure(2 * std::max(na, 1));
  flag.ensure(1);
  PM_CUDA(cudaStreamSynchronize(c->stream));  // the host vectors go out of scope
  rows_of = A.mask;
  rows_of.guard = nullptr;
  act_set = true;
}

template <class T>
void DenseInverse::prepare(pm_ctx* c, const DevCsr& A, T* M) {
  PM_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), c->stream));
  has64 = has32 = false;
  if (na == 0) return;
  k_dense_fill<T><<<nblocks((long long)na * 32, 256), 256, 0, c->stream>>>(na, act.p, pos.p, A.row_ptr.p, A.cols.p,
                                                                         A.vals.p, M);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

void DenseInverse::build(pm_ctx* c, const DevCsr& A) {
  launch64(c, A, c->stream);
  complete64(c);
}

void DenseInverse::complete64(pm_ctx* c) {
  if (!pending64) return;
  pending64 = false;
  int h_flag = 0;
  PM_CUDA(cudaStreamWaitEvent(c->stream, done_event, 0));
  PM_CUDA(cudaMemcpyAsync(&h_flag, flag.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  PM_CUDA(cudaStreamSynchronize(c->stream));
  if (h_flag) throw Error(PM_E_BREAKDOWN, "coarse matrix is singular (zero pivot)");
  has64 = true;
}

void DenseInverse::launch64(pm_ctx* c, const DevCsr& A, cudaStream_t s) {
  pending64 = false;
  set_rows(c, A);
  StreamSwap swap(c, s);
  const size_t nn = size_t(na) * na;
  inv.ensure(nn);
  const bool panels = na <= kGjMaxRows;
  if (panels && na) {
    work.ensure(nn + 2 * kGjWidth64 * kGjWidth64);
    prepare(c, A, gj_start(na, kGjWidth64, work.p, inv.p));
    gj_inverse(c, na, work.p, perm.p, perm.p + na, flag.p, inv.p);
  } else {
    prepare(c, A, inv.p);
    if (na == 0) {
      has64 = true;
      return;
    }
    eliminate_columns(c);
  }
  if (!done_event) PM_CUDA(cudaEventCreateWithFlags(&done_event, cudaEventDisableTiming));
  PM_CUDA(cudaEventRecord(done_event, s));
  pending64 = true;
}

// Column by column, in place: more rows than the panel's block keeps in
// registers
void DenseInverse::eliminate_columns(pm_ctx* c) {
  int coop = 0, per_sm = 0;
  PM_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device));
  PM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gj_coop, 256, 0));
  if (coop && per_sm > 0) {
    // one cooperative launch; at most one block per SM and about 8 rows per block
    int nb = std::min(c->num_sms, std::max(1, (na + 7) / 8));
    rowk.ensure(na);
    oldk.ensure(na);
    part_v.ensure(nb);
    part_i.ensure(nb);
    double* M = inv.p;
    int* pp = perm.p;
    double* rk = rowk.p;
    double* ok = oldk.p;
    double* ck = tmp.p;
    double* pv = part_v.p;
    int* pi = part_i.p;
    int* fl = flag.p;
    int nan_ = na;
    void* args[] = {&nan_, &M, &pp, &rk, &ok, &ck, &pv, &pi, &fl};
    PM_CUDA(cudaLaunchCooperativeKernel((const void*)k_gj_coop, dim3(nb), dim3(256), args, 0, c->stream));
    c->kernel_launches++;
  } else {
    const int ugrid = std::max(1, std::min(nblocks((long long)na * na, 256), c->num_sms * 8));
    for (int k = 0; k < na; ++k) {
      k_gj_pivot<<<1, 256, 0, c->stream>>>(na, k, inv.p, perm.p, tmp.p, flag.p);
      k_gj_update<<<ugrid, 256, 0, c->stream>>>(na, k, inv.p, tmp.p);
      c->kernel_launches += 2;
    }
  }
  PM_CHECK_LAUNCH();
  k_gj_unswap<<<nblocks(na, 128), 128, 0, c->stream>>>(na, inv.p, perm.p);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

// tmp_a = b_a - sum over non-active columns of A_{a,j} b_j
__global__ void k_coarse_rhs(int na, const int* __restrict__ act, const int* __restrict__ pos,
                             const int* __restrict__ rp, const int* __restrict__ ci,
                             const double* __restrict__ v, const double* __restrict__ b,
                             double* __restrict__ tmp) {
  int ia = blockIdx.x * blockDim.x + threadIdx.x;
  if (ia >= na) return;
  const int i = act[ia];
  double r = b[i];
  for (int k = rp[i]; k < rp[i + 1]; ++k)
    if (pos[ci[k]] < 0) r -= v[k] * b[ci[k]];
  tmp[ia] = r;
}

// x_a = inv * tmp (one warp per row), x_n = b_n
__global__ void k_coarse_gemv(int n, int na, const int* __restrict__ act, const int* __restrict__ pos,
                              const double* __restrict__ inv, const double* __restrict__ tmp,
                              const double* __restrict__ b, double* __restrict__ x,
                              const int* __restrict__ gather) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp < na) {
    const double* row = inv + (size_t)warp * na;
    double s = 0.0;
    // gather != null: the right-hand side's non-actives are zero, read b directly
    for (int j = lane; j < na; j += 32) s += row[j] * (gather ? b[gather[j]] : tmp[j]);
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) x[act[warp]] = s;
  } else {
    // remaining threads copy the non-active entries
    const int t = (warp - na) * 32 + lane;
    if (t < n && pos[t] < 0) x[t] = b[t];
  }
}

void DenseInverse::solve(pm_ctx* c, const DevCsr& A, const double* b, double* x, bool rhs_nonactive_zero) {
  if (na > 0 && !rhs_nonactive_zero) {
    k_coarse_rhs<<<nblocks(na, 128), 128, 0, c->stream>>>(na, act.p, pos.p, A.row_ptr.p, A.cols.p,
                                                          A.vals.p, b, tmp.p);
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
  }
  const long long threads = (long long)(na + (n + 31) / 32) * 32;
  k_coarse_gemv<<<nblocks(threads, 256), 256, 0, c->stream>>>(n, na, act.p, pos.p, inv.p, tmp.p, b, x,
                                                              rhs_nonactive_zero ? act.p : nullptr);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

}  // namespace pm

// ---------------------------------------------------------------------------
// Batched launches (pm_batch.h): the same operation for the slots of a batch
// in one launch (the slot is blockIdx.x in the SpMV family, blockIdx.y
// elsewhere). The SpMV family runs csr_body / sell_body,
// the other kernels restate the single-problem loops line for line, so each
// slot gets the bits a lone launch gives.
#include "pm_batch.h"

namespace pm {

// SpMV-family launches: bt.vals holds two pointers per slot, the sliced-ELL
// values [2 s] and the CSR values [2 s + 1]; bt.aux the slot's diagonal
template <class TV, class TX, class TA, int G, int U, int EPI>
__global__ void __launch_bounds__(256)
csr_batch_kernel(int n_rows, const int* __restrict__ row_ptr, const int* __restrict__ cols,
                 const TV* __restrict__ vals, const TX* x, TX* y, const TX* b, const TX* __restrict__ diag,
                 TA alpha, BlockMask mask, Batch bt) {
  const int s = blockIdx.x;
  if (!bt.on[s]) return;
  const TV* v = bt.vals ? static_cast<const TV*>(bt.vals[2 * s + 1]) : vals;
  const TX* d = bt.aux ? static_cast<const TX*>(bt.aux[s]) : diag;
  const TX* xs = slot_ptr(x, bt, s);
  csr_body<TV, TX, TA, G, U, EPI>(n_rows, row_ptr, cols, v, xs, slot_ptr(y, bt, s), slot_ptr(b, bt, s), d, xs,
                                  alpha, mask, blockIdx.y, gridDim.y);
}

template <class T, int L, int U, bool PIPE, int EPI>
__global__ void __launch_bounds__(128)
sell_batch_kernel(int n_slices, const int* __restrict__ perm, const int* __restrict__ soff,
                  const int* __restrict__ scols, const T* __restrict__ svals, const T* x, T* y, const T* b,
                  const T* __restrict__ diag, T alpha, BlockMask mask, Batch bt) {
  const int s = blockIdx.x;
  if (!bt.on[s]) return;
  const T* v = bt.vals ? static_cast<const T*>(bt.vals[2 * s]) : svals;
  const T* d = bt.aux ? static_cast<const T*>(bt.aux[s]) : diag;
  sell_body<T, L, U, PIPE, EPI>(n_slices, perm, soff, scols, v, slot_ptr(x, bt, s), slot_ptr(y, bt, s),
                                slot_ptr(b, bt, s), d, alpha, mask, blockIdx.y);
}

template <class T, int L, int U, bool P, int EPI>
static void launch_sell_batch_epi(pm_ctx* c, const DevCsr& A, int ns, const Batch& bt, const T* x, T* y, const T* b,
                                  const T* d, T alpha, const BlockMask& m) {
  cudaLaunchConfig_t cfg = {};
  if (nblocks(A.n_slices, 4) > 65535) throw Error(PM_E_UNSUPPORTED, "batched launch: too many row blocks");
  cfg.gridDim = dim3(unsigned(ns), unsigned(nblocks(A.n_slices, 4)));
  cfg.blockDim = dim3(128);
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = c->pdl >= 1 ? 1 : 0;
  PM_CUDA(cudaLaunchKernelEx(&cfg, sell_batch_kernel<T, L, U, P, EPI>, A.n_slices, (const int*)A.sell_perm.p,
                             (const int*)A.sell_off.p, (const int*)A.sell_cols.p, sell_values<T>(A), x, y, b, d,
                             alpha, m, bt));
  c->kernel_launches++;
}

template <class T, int L, int U, bool P>
static void launch_sell_batch(pm_ctx* c, const DevCsr& A, int ns, const Batch& bt, int epi, const T* x, T* y,
                              const T* b, const T* d, T alpha, const BlockMask& m) {
  switch (epi) {
    case EPI_AXPY: launch_sell_batch_epi<T, L, U, P, EPI_AXPY>(c, A, ns, bt, x, y, b, d, alpha, m); break;
    case EPI_SET: launch_sell_batch_epi<T, L, U, P, EPI_SET>(c, A, ns, bt, x, y, b, d, alpha, m); break;
    case EPI_DEFECT: launch_sell_batch_epi<T, L, U, P, EPI_DEFECT>(c, A, ns, bt, x, y, b, d, alpha, m); break;
    case EPI_JACOBI: launch_sell_batch_epi<T, L, U, P, EPI_JACOBI>(c, A, ns, bt, x, y, b, d, alpha, m); break;
    case EPI_RESTRICT: launch_sell_batch_epi<T, L, U, P, EPI_RESTRICT>(c, A, ns, bt, x, y, b, d, alpha, m); break;
    case EPI_PROLONG: launch_sell_batch_epi<T, L, U, P, EPI_PROLONG>(c, A, ns, bt, x, y, b, d, alpha, m); break;
    default: throw Error(PM_E_INVALID, "unknown SpMV epilogue");
  }
}

template <class TV, class TX, class TA, int G, int U>
static void launch_csr_batch_gu(pm_ctx* c, int ns, const Batch& bt, int epi, int n, const DevCsr& A, const TV* v,
                                const TX* x, TX* y, const TX* b, const TX* d, TA alpha, const BlockMask& m) {
  if (nblocks((long long)n * G, 256) > 65535) throw Error(PM_E_UNSUPPORTED, "batched launch: too many row blocks");
  const dim3 gr = dim3(unsigned(ns), unsigned(nblocks((long long)n * G, 256))), bl = dim3(256);
  const int* rp = A.row_ptr.p;
  const int* ci = A.cols.p;
  switch (epi) {
    case EPI_AXPY: csr_batch_kernel<TV, TX, TA, G, U, EPI_AXPY><<<gr, bl, 0, c->stream>>>(n, rp, ci, v, x, y, b, d, alpha, m, bt); break;
    case EPI_SET: csr_batch_kernel<TV, TX, TA, G, U, EPI_SET><<<gr, bl, 0, c->stream>>>(n, rp, ci, v, x, y, b, d, alpha, m, bt); break;
    case EPI_DEFECT: csr_batch_kernel<TV, TX, TA, G, U, EPI_DEFECT><<<gr, bl, 0, c->stream>>>(n, rp, ci, v, x, y, b, d, alpha, m, bt); break;
    case EPI_JACOBI: csr_batch_kernel<TV, TX, TA, G, U, EPI_JACOBI><<<gr, bl, 0, c->stream>>>(n, rp, ci, v, x, y, b, d, alpha, m, bt); break;
    case EPI_RESTRICT: csr_batch_kernel<TV, TX, TA, G, U, EPI_RESTRICT><<<gr, bl, 0, c->stream>>>(n, rp, ci, v, x, y, b, d, alpha, m, bt); break;
    case EPI_PROLONG: csr_batch_kernel<TV, TX, TA, G, U, EPI_PROLONG><<<gr, bl, 0, c->stream>>>(n, rp, ci, v, x, y, b, d, alpha, m, bt); break;
    default: throw Error(PM_E_INVALID, "unknown SpMV epilogue");
  }
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

// the launch shapes DevCsr::upload picks: FP64 two or four lanes x eight
// loads, FP32 four x four or eight x sixteen
template <class TV, class TX, class TA>
static void launch_csr_batch(pm_ctx* c, int ns, const Batch& bt, int epi, int n, const DevCsr& A, const TV* v,
                             const TX* x, TX* y, const TX* b, const TX* d, TA alpha, const BlockMask& m) {
  const bool fp32 = sizeof(TV) == 4;
  const int G = fp32 ? A.lanes32 : A.lanes;
  const int U = fp32 ? A.unroll32 : A.unroll;
  if (G == 2 && U == 8) launch_csr_batch_gu<TV, TX, TA, 2, 8>(c, ns, bt, epi, n, A, v, x, y, b, d, alpha, m);
  else if (G == 4 && U == 4) launch_csr_batch_gu<TV, TX, TA, 4, 4>(c, ns, bt, epi, n, A, v, x, y, b, d, alpha, m);
  else if (G == 4 && U == 8) launch_csr_batch_gu<TV, TX, TA, 4, 8>(c, ns, bt, epi, n, A, v, x, y, b, d, alpha, m);
  else if (G == 8 && U == 16) launch_csr_batch_gu<TV, TX, TA, 8, 16>(c, ns, bt, epi, n, A, v, x, y, b, d, alpha, m);
  else throw Error(PM_E_UNSUPPORTED, "batched CSR launch shape " + std::to_string(G) + "x" + std::to_string(U));
}

void csr_apply_batch(pm_ctx* c, const DevCsr& A, int ns, const Batch& bt, int epi, const double* x, double* y,
                     const double* b, double alpha) {
  const int n = A.n_rows;
  if (n <= 0) return;
  if (A.stream && A.n_rblocks > 0) throw Error(PM_E_UNSUPPORTED, "batched launch of the streaming CSR kernel");
  if (c->sell_shape64 > 0 && A.sell64_ok && A.sell_lanes == c->sell_shape64 / 100 && A.n_slices > 0) {
    switch (c->sell_shape64) {
      case 441: launch_sell_batch<double, 4, 4, true>(c, A, ns, bt, epi, x, y, b, A.diag.p, alpha, A.mask); break;
      case 442:
        if (sell_deep64(c, A, ns)) launch_sell_batch<double, 4, 8, true>(c, A, ns, bt, epi, x, y, b, A.diag.p, alpha, A.mask);
        else launch_sell_batch<double, 4, 4, true>(c, A, ns, bt, epi, x, y, b, A.diag.p, alpha, A.mask);
        break;
      case 481: launch_sell_batch<double, 4, 8, true>(c, A, ns, bt, epi, x, y, b, A.diag.p, alpha, A.mask); break;
      case 841: launch_sell_batch<double, 8, 4, true>(c, A, ns, bt, epi, x, y, b, A.diag.p, alpha, A.mask); break;
      default: throw Error(PM_E_INVALID, "unknown FP64 sliced SpMV shape");
    }
    PM_CHECK_LAUNCH();
    return;
  }
  launch_csr_batch<double, double, double>(c, ns, bt, epi, n, A, A.vals.p, x, y, b, A.diag.p, alpha, A.mask);
}

void csr_apply32_batch(pm_ctx* c, const DevCsr& A, int ns, const Batch& bt, int epi, const float* x, float* y,
                       const float* b, float alpha) {
  const int n = A.n_rows;
  if (n <= 0) return;
  if (A.stream && A.n_rblocks > 0) throw Error(PM_E_UNSUPPORTED, "batched launch of the streaming CSR kernel");
  if (c->sell_shape > 0 && A.sell_lanes == c->sell_shape / 100 && A.n_slices > 0) {
    switch (c->sell_shape) {
      case 441: launch_sell_batch<float, 4, 4, true>(c, A, ns, bt, epi, x, y, b, A.diag32.p, alpha, A.mask); break;
      case 481: launch_sell_batch<float, 4, 8, true>(c, A, ns, bt, epi, x, y, b, A.diag32.p, alpha, A.mask); break;
      case 482:
        if (sell_deep32(c, A, ns)) launch_sell_batch<float, 4, 16, true>(c, A, ns, bt, epi, x, y, b, A.diag32.p, alpha, A.mask);
        else launch_sell_batch<float, 4, 8, true>(c, A, ns, bt, epi, x, y, b, A.diag32.p, alpha, A.mask);
        break;
      case 841: launch_sell_batch<float, 8, 4, true>(c, A, ns, bt, epi, x, y, b, A.diag32.p, alpha, A.mask); break;
      case 881: launch_sell_batch<float, 8, 8, true>(c, A, ns, bt, epi, x, y, b, A.diag32.p, alpha, A.mask); break;
      default: throw Error(PM_E_UNSUPPORTED, "batched launch of sliced shape " + std::to_string(c->sell_shape));
    }
    PM_CHECK_LAUNCH();
    return;
  }
  launch_csr_batch<float, float, float>(c, ns, bt, epi, n, A, A.vals32.p, x, y, b, A.diag32.p, alpha, A.mask);
}

__global__ void kb_copy(long long n, const double* __restrict__ x, double* __restrict__ y, Batch bt) {
  if (!bt.on[blockIdx.y]) return;
  x = slot_ptr(x, bt);
  y = slot_ptr(y, bt);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = x[i];
}
__global__ void kb_d2f(long long n, const double* __restrict__ x, float* __restrict__ y, Batch bt) {
  if (!bt.on[blockIdx.y]) return;
  x = slot_ptr(x, bt);
  y = slot_ptr(y, bt);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = float(x[i]);
}
__global__ void kb_f2d(long long n, const float* __restrict__ x, double* __restrict__ y, Batch bt) {
  if (!bt.on[blockIdx.y]) return;
  x = slot_ptr(x, bt);
  y = slot_ptr(y, bt);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = double(x[i]);
}
template <class T>
__global__ void kb_init_sol(int n, BlockMask m, const T* __restrict__ rhs, T* __restrict__ sol, Batch bt) {
  if (!bt.on[blockIdx.y]) return;
  rhs = slot_ptr(rhs, bt);
  sol = slot_ptr(sol, bt);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    sol[i] = row_is_active(m, i) ? T(0) : rhs[i];
}
template <class T>
__global__ void kb_jacobi_zero(int n, const T* __restrict__ b, T w, T* __restrict__ x, Batch bt) {
  const int s = blockIdx.y;
  if (!bt.on[s]) return;
  const T* d = static_cast<const T*>(bt.aux[s]);
  b = slot_ptr(b, bt);
  x = slot_ptr(x, bt);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x[i] = fmadd(w, (b[i] - T(0)) / d[i], T(0));
}

#define PM_LAUNCH_BATCH(kern, ns, n, ...)                                                       \
  do {                                                                                          \
    if ((n) > 0) {                                                                              \
      kern<<<dim3(unsigned(grid_for(c, (n))), unsigned(ns)), 256, 0, c->stream>>>(__VA_ARGS__); \
      PM_CHECK_LAUNCH();                                                                        \
      c->kernel_launches++;                                                                     \
    }                                                                                           \
  } while (0)

void vcopy_batch(pm_ctx* c, int ns, const Batch& bt, int n, const double* x, double* y) {
  PM_LAUNCH_BATCH(kb_copy, ns, n, n, x, y, bt);
}
void vcvt_d2f_batch(pm_ctx* c, int ns, const Batch& bt, int n, const double* x, float* y) {
  PM_LAUNCH_BATCH(kb_d2f, ns, n, n, x, y, bt);
}
void vcvt_f2d_batch(pm_ctx* c, int ns, const Batch& bt, int n, const float* x, double* y) {
  PM_LAUNCH_BATCH(kb_f2d, ns, n, n, x, y, bt);
}
template <class T>
void init_solution_batch(pm_ctx* c, int ns, const Batch& bt, int n, const BlockMask& m, const T* rhs, T* sol) {
  PM_LAUNCH_BATCH(kb_init_sol<T>, ns, n, n, m, rhs, sol, bt);
}
template void init_solution_batch<float>(pm_ctx*, int, const Batch&, int, const BlockMask&, const float*, float*);
template void init_solution_batch<double>(pm_ctx*, int, const Batch&, int, const BlockMask&, const double*, double*);
template <class T>
void jacobi_from_zero_batch(pm_ctx* c, int ns, const Batch& bt, int n, const T* b, T w, T* x) {
  PM_LAUNCH_BATCH(kb_jacobi_zero<T>, ns, n, n, b, w, x, bt);
}
template void jacobi_from_zero_batch<float>(pm_ctx*, int, const Batch&, int, const float*, float, float*);
template void jacobi_from_zero_batch<double>(pm_ctx*, int, const Batch&, int, const double*, double, double*);

// the coarse-grid inverse of slot s is bt.aux[s]; act / pos are the same for
// every slot (one set-up)
__global__ void kb_coarse_gemv32(int n, int na, const int* __restrict__ act, const int* __restrict__ pos,
                                 const float* __restrict__ b, float* __restrict__ x, Batch bt) {
  const int s = blockIdx.y;
  if (!bt.on[s]) return;
  const float* inv = static_cast<const float*>(bt.aux[s]);
  b = slot_ptr(b, bt);
  x = slot_ptr(x, bt);
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp < na) {
    const float* row = inv + (size_t)warp * na;
    float sum = 0.0f;
    for (int j = lane; j < na; j += 32) sum += row[j] * b[act[j]];
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
    if (lane == 0) x[act[warp]] = sum;
  } else {
    const int t = (warp - na) * 32 + lane;
    if (t < n && pos[t] < 0) x[t] = b[t];
  }
}
// the FP64 coarse solve of a right-hand side with zero non-actives (the
// gather form of k_coarse_gemv)
__global__ void kb_coarse_gemv(int n, int na, const int* __restrict__ act, const int* __restrict__ pos,
                               const double* __restrict__ b, double* __restrict__ x, Batch bt) {
  const int s = blockIdx.y;
  if (!bt.on[s]) return;
  const double* inv = static_cast<const double*>(bt.aux[s]);
  b = slot_ptr(b, bt);
  x = slot_ptr(x, bt);
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp < na) {
    const double* row = inv + (size_t)warp * na;
    double sum = 0.0;
    for (int j = lane; j < na; j += 32) sum += row[j] * b[act[j]];
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
    if (lane == 0) x[act[warp]] = sum;
  } else {
    const int t = (warp - na) * 32 + lane;
    if (t < n && pos[t] < 0) x[t] = b[t];
  }
}

void coarse_solve32_batch(pm_ctx* c, int ns, const Batch& bt, const DenseInverse& inv0, const float* b, float* x) {
  const long long threads = (long long)(inv0.na + (inv0.n + 31) / 32) * 32;
  kb_coarse_gemv32<<<dim3(unsigned(nblocks(threads, 256)), unsigned(ns)), 256, 0, c->stream>>>(
      inv0.n, inv0.na, inv0.act.p, inv0.pos.p, b, x, bt);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

void coarse_solve_batch(pm_ctx* c, int ns, const Batch& bt, const DenseInverse& inv0, const double* b, double* x) {
  const long long threads = (long long)(inv0.na + (inv0.n + 31) / 32) * 32;
  kb_coarse_gemv<<<dim3(unsigned(nblocks(threads, 256)), unsigned(ns)), 256, 0, c->stream>>>(
      inv0.n, inv0.na, inv0.act.p, inv0.pos.p, b, x, bt);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

__global__ void __launch_bounds__(256) kb_dot_partials(int n, const double* __restrict__ x,
                                                       const double* __restrict__ y, double* __restrict__ part,
                                                       Batch bt) {
  if (!bt.on[blockIdx.y]) return;
  x = slot_ptr(x, bt);
  y = slot_ptr(y, bt);
  part = slot_ptr(part, bt);
  __shared__ double sh[256];
  double s = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s += x[i] * y[i];
  double r = block_sum(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = r;
}
__global__ void kb_finish_sum(const double* __restrict__ part, int np, double* out, int take_sqrt, Batch bt) {
  if (!bt.on[blockIdx.y]) return;
  part = slot_ptr(part, bt);
  out = slot_ptr(out, bt);
  __shared__ double sh[256];
  double s = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) s += part[i];
  double r = block_sum(s, sh);
  if (threadIdx.x == 0) *out = take_sqrt ? sqrt(r) : r;
}
void dot_partials_batch(pm_ctx* c, int ns, const Batch& bt, int n, const double* x, const double* y, double* part) {
  kb_dot_partials<<<dim3(unsigned(red_blocks(n)), unsigned(ns)), kRedThreads, 0, c->stream>>>(n, x, y, part, bt);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}
void finish_sum_batch(pm_ctx* c, int ns, const Batch& bt, int n, const double* part, double* out, bool take_sqrt) {
  kb_finish_sum<<<dim3(1, unsigned(ns)), 256, 0, c->stream>>>(part, red_blocks(n), out, take_sqrt ? 1 : 0, bt);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}
__global__ void kb_nonactive_nonzero(BlockMask m, const double* __restrict__ x, int* __restrict__ flag, Batch bt) {
  if (!bt.on[blockIdx.y]) return;
  x = slot_ptr(x, bt);
  flag = slot_ptr(flag, bt);
  for (int b = 0; b < m.nb; ++b)
    for (int i = m.active_end[b] + blockIdx.x * blockDim.x + threadIdx.x; i < m.end[b]; i += gridDim.x * blockDim.x)
      if (x[i] != 0.0) *flag = 1;
}
void nonactive_nonzero_batch(pm_ctx* c, int ns, const Batch& bt, const BlockMask& m, const double* x, int* flag) {
  kb_nonactive_nonzero<<<dim3(kRedBlocks, unsigned(ns)), 256, 0, c->stream>>>(m, x, flag, bt);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

}  // namespace pm
