// mtp_kernels.cu - evaluation-kernel instantiations and the supporting kernels:
// incoming-slot lists, deterministic force gather, fixed-order reductions.
#include "mtp_launch.hpp"
#include "mtp_md.hpp"

#include <climits>
#include <type_traits>

namespace mtp {

// ---------------------------------------------------------------------------
// evaluation kernel launch
// ---------------------------------------------------------------------------
template <typename T>
static SmemLayout eval_layout(const DevModel& md, int n_pad, int threads, bool vglobal, int A) {
  auto layout = [&](int qs) {
    return smem_layout<T>(vglobal ? 0 : md.v_size, md.M, md.S, md.R, md.K, md.D, md.P, md.n_list, md.n3_len, n_pad, qs,
                          threads, A);
  };
  return layout(row_stride<T>(n_pad, threads, [&](int qs) { return layout(qs).total; }));
}

namespace {

// The dynamic shared-memory limit of each instantiation only ever grows, so a
// later launch never finds it lowered by an occupancy query for a smaller
// shape, and steady-state launches make no attribute calls (graph capture).
template <typename T, bool G, int A>
cudaError_t ensure_smem_limit(size_t bytes) {
  static size_t granted = 0;
  if (bytes <= granted) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_mtp_eval<T, G, A>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(bytes));
  if (e == cudaSuccess) granted = bytes;
  return e;
}

template <typename T, bool G, int A>
int occupancy_t(size_t bytes, int threads) {
  int nb = 0;
  if (bytes > kMaxSmemPerBlock) return 0;
  if (ensure_smem_limit<T, G, A>(bytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_mtp_eval<T, G, A>, threads, bytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return nb;
}

template <typename T, bool G, int A>
cudaError_t launch_t(const DevModel& md, const DevIO& io, int threads, int blocks, size_t bytes, cudaStream_t st) {
  cudaError_t e = ensure_smem_limit<T, G, A>(bytes);
  if (e != cudaSuccess) return e;
  k_mtp_eval<T, G, A><<<blocks, threads, bytes, st>>>(md, io);
  return cudaGetLastError();
}

}  // namespace

// Supported (precision, placement, atoms per block) combinations.
#define MTP_EVAL_VARIANTS(X) \
  X(double, false, 1) X(double, false, 2) X(double, true, 1) X(double, true, 2) X(float, false, 1) X(float, false, 2) \
  X(float, false, 4) X(float, true, 1)

bool eval_variant_exists(bool fp64, bool vglobal, int A) {
#define X(T, G, AA) \
  if ((fp64 == std::is_same<T, double>::value) && vglobal == G && A == AA) return true;
  MTP_EVAL_VARIANTS(X)
#undef X
  return false;
}

EvalFit eval_fit(const DevModel& md, int n_pad, int threads, bool fp64, bool vglobal, int A) {
  const SmemLayout L = fp64 ? eval_layout<double>(md, n_pad, threads, vglobal, A)
                            : eval_layout<float>(md, n_pad, threads, vglobal, A);
  EvalFit fit;
  fit.qs = L.qs;
  fit.smem = L.total;
#define X(T, G, AA) \
  if ((fp64 == std::is_same<T, double>::value) && vglobal == G && A == AA) \
    fit.per_sm = occupancy_t<T, G, AA>(L.total, threads);
  MTP_EVAL_VARIANTS(X)
#undef X
  return fit;
}

cudaError_t launch_eval(const DevModel& md, const DevIO& io, const EvalFit& fit, int threads, int blocks, bool fp64,
                        bool vglobal, int A, cudaStream_t st) {
  if (io.natoms <= 0) return cudaSuccess;
  DevIO rows = io;
  rows.qs = fit.qs;
#define X(T, G, AA) \
  if ((fp64 == std::is_same<T, double>::value) && vglobal == G && A == AA) \
    return launch_t<T, G, AA>(md, rows, threads, blocks, fit.smem, st);
  MTP_EVAL_VARIANTS(X)
#undef X
  return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// incoming-slot lists
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool scatter_slot(int i, int s, int natoms, int stride, const int* js,
                                             const int* jtypes, const int* counts, int& j) {
  const int cnt = counts ? min(__ldg(counts + i), stride) : stride;
  if (s >= cnt) return false;
  const size_t x = static_cast<size_t>(i) * stride + s;
  if (__ldg(jtypes + x) < 0) return false;
  j = __ldg(js + x);
  return j >= 0 && j < natoms;
}

__global__ void k_count_incoming(int natoms, int stride, const int* js, const int* jtypes, const int* counts,
                                 int* in_cnt) {
  const size_t n = static_cast<size_t>(natoms) * stride;
  for (size_t x = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; x < n;
       x += static_cast<size_t>(gridDim.x) * blockDim.x) {
    int j;
    if (scatter_slot(static_cast<int>(x / stride), static_cast<int>(x % stride), natoms, stride, js, jtypes,
                     counts, j))
      atomicAdd(in_cnt + j, 1);
  }
}

// exclusive scan, three kernels: per-1024 block scans, scan of block totals, offsets
__global__ void k_scan_blocks(int n, const int* in, int* out, int* block_tot) {
  __shared__ int wsum[32];
  const int i = blockIdx.x * 1024 + threadIdx.x;
  int v = i < n ? in[i] : 0;
  const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (l >= o) x += y;
  }
  if (l == 31) wsum[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = wsum[l];
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, s, o);
      if (l >= o) s += y;
    }
    wsum[l] = s;
  }
  __syncthreads();
  const int incl = x + (w > 0 ? wsum[w - 1] : 0);
  if (i < n) out[i] = incl - v;
  if (threadIdx.x == 1023) block_tot[blockIdx.x] = incl;
}

__global__ void k_scan_totals(int nb, int* block_tot, int* total_out) {
  // single block of 1024 threads, sequential over chunks of 1024 totals
  __shared__ int wsum[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nb; base += 1024) {
    const int i = base + threadIdx.x;
    int v = i < nb ? block_tot[i] : 0;
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, x, o);
      if (l >= o) x += y;
    }
    if (l == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
      int s = wsum[l];
      for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, s, o);
        if (l >= o) s += y;
      }
      wsum[l] = s;
    }
    __syncthreads();
    const int incl = x + (w > 0 ? wsum[w - 1] : 0) + carry;
    if (i < nb) block_tot[i] = incl - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry = incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total_out = carry;
}

__global__ void k_scan_add(int n, int* out, const int* block_off) {
  const int i = blockIdx.x * 1024 + threadIdx.x;
  if (i < n) out[i] += block_off[blockIdx.x];
}

// The whole scan in one block: thread t sums the `per` consecutive values it
// owns, the block scans the sums, and the thread writes its prefixes.  For
// small n (a LAMMPS-size call) it replaces three launches.
__global__ void k_scan_one_block(int n, int per, const int* __restrict__ in, int* __restrict__ out) {
  __shared__ int wsum[32];
  const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b = min(n, static_cast<int>(threadIdx.x) * per), e = min(n, b + per);
  int v = 0;
  for (int i = b; i < e; ++i) v += in[i];
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (l >= o) x += y;
  }
  if (l == 31) wsum[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = wsum[l];
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, s, o);
      if (l >= o) s += y;
    }
    wsum[l] = s;
  }
  __syncthreads();
  int run = x - v + (w > 0 ? wsum[w - 1] : 0);
  for (int i = b; i < e; ++i) {
    out[i] = run;
    run += in[i];
  }
  if (threadIdx.x == 1023) out[n] = run;
}

// Up to this many values one block scans all (8 per thread: 4 us at 8,192
// values; the three kernels take 6 us with their gaps).
constexpr int kOneBlockScan = 8192;

// out[0..n) = exclusive prefix sums of in, out[n] = total; blk holds n/1024 + 1 ints.
cudaError_t scan_exclusive(int n, const int* in, int* out, int* blk, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (n <= kOneBlockScan) {
    k_scan_one_block<<<1, 1024, 0, st>>>(n, (n + 1023) / 1024, in, out);
    return cudaGetLastError();
  }
  const int nb = (n + 1023) / 1024;
  k_scan_blocks<<<nb, 1024, 0, st>>>(n, in, out, blk);
  k_scan_totals<<<1, 1024, 0, st>>>(nb, blk, out + n);
  k_scan_add<<<nb, 1024, 0, st>>>(n, out, blk);
  return cudaGetLastError();
}

// Every slot takes a place in its neighbour's list; the counts run down to
// zero as they hand the places out.
__global__ void k_fill_incoming(int natoms, int stride, const int* js, const int* jtypes, const int* counts,
                                const int* in_ptr, int* in_cnt, int* in_slot) {
  const size_t n = static_cast<size_t>(natoms) * stride;
  for (size_t x = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; x < n;
       x += static_cast<size_t>(gridDim.x) * blockDim.x) {
    int j;
    if (scatter_slot(static_cast<int>(x / stride), static_cast<int>(x % stride), natoms, stride, js, jtypes,
                     counts, j)) {
      const int pos = atomicSub(in_cnt + j, 1) - 1;
      in_slot[in_ptr[j] + pos] = static_cast<int>(x);
    }
  }
}

// Sort one atom's incoming list by slot id (one warp): the gather order, and
// so the rounding of the forces, no longer depends on the fill race above.
// Lists of up to 64 slots are ranked in registers (slot ids are distinct, so
// each value's rank is the count of smaller values); longer lists fall back to
// an insertion sort by the warp's first lane.
__device__ __forceinline__ void sort_incoming(int b, int n, int lane, int* in_slot) {
  if (n <= 64) {
    const int v0 = lane < n ? in_slot[b + lane] : INT_MAX;
    const int v1 = lane + 32 < n ? in_slot[b + lane + 32] : INT_MAX;
    int r0 = 0, r1 = 0;
    for (int k = 0; k < 32; ++k) {
      const int u0 = __shfl_sync(0xffffffffu, v0, k), u1 = __shfl_sync(0xffffffffu, v1, k);
      r0 += (u0 < v0) + (u1 < v0);
      r1 += (u0 < v1) + (u1 < v1);
    }
    __syncwarp();
    if (lane < n) in_slot[b + r0] = v0;
    if (lane + 32 < n) in_slot[b + r1] = v1;
  } else if (lane == 0) {
    for (int x = b + 1; x < b + n; ++x) {
      const int v = in_slot[x];
      int y = x - 1;
      while (y >= b && in_slot[y] > v) {
        in_slot[y + 1] = in_slot[y];
        --y;
      }
      in_slot[y + 1] = v;
    }
  }
  __syncwarp();
}

cudaError_t launch_incoming(int natoms, int stride, const int* js, const int* jtypes, const int* counts,
                            int* in_cnt, int* in_ptr, int* in_slot, int* block_tmp, bool counted, cudaStream_t st) {
  if (natoms <= 0) return cudaSuccess;
  const size_t n = static_cast<size_t>(natoms) * stride;
  const int gb = static_cast<int>(std::min<size_t>((n + 255) / 256, 148 * 32));
  cudaError_t e = cudaSuccess;
  if (!counted) {
    // the counts start at zero (the allocation-free path reuses a shared array)
    e = cudaMemsetAsync(in_cnt, 0, sizeof(int) * natoms, st);
    if (e != cudaSuccess) return e;
    k_count_incoming<<<gb, 256, 0, st>>>(natoms, stride, js, jtypes, counts, in_cnt);
  }
  e = scan_exclusive(natoms, in_cnt, in_ptr, block_tmp, st);
  if (e != cudaSuccess) return e;
  k_fill_incoming<<<gb, 256, 0, st>>>(natoms, stride, js, jtypes, counts, in_ptr, in_cnt, in_slot);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// deterministic force gather: one warp per atom
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sym_rg(const double* r, const double* g, double* w, double sgn) {
  w[0] += sgn * r[0] * g[0];
  w[1] += sgn * r[1] * g[1];
  w[2] += sgn * r[2] * g[2];
  w[3] += sgn * 0.5 * (r[0] * g[1] + r[1] * g[0]);
  w[4] += sgn * 0.5 * (r[0] * g[2] + r[2] * g[0]);
  w[5] += sgn * 0.5 * (r[1] * g[2] + r[2] * g[1]);
}

// kSort: the incoming lists are fresh from launch_incoming and this atom's is
// sorted first (here rather than in a launch of its own).
template <bool kSort>
__global__ void k_force_gather(int natoms, int stride, const double* __restrict__ rijs,
                               const int* __restrict__ counts, const double* __restrict__ G,
                               const int* __restrict__ in_ptr, int* in_slot,
                               double* __restrict__ forces, double* __restrict__ wown,
                               double* __restrict__ vatom) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= natoms) return;
  const int i = warp;
  const int cnt = counts ? min(__ldg(counts + i), stride) : stride;
  double F[3] = {0, 0, 0}, Wo[6] = {0, 0, 0, 0, 0, 0}, Wi[6] = {0, 0, 0, 0, 0, 0};
  const size_t row = static_cast<size_t>(i) * stride;
  for (int s = lane; s < cnt; s += 32) {
    const double* g = G + 3 * (row + s);
    const double* r = rijs + 3 * (row + s);
    double gg[3] = {__ldg(g), __ldg(g + 1), __ldg(g + 2)};
    double rr[3] = {__ldg(r), __ldg(r + 1), __ldg(r + 2)};
    F[0] += gg[0];
    F[1] += gg[1];
    F[2] += gg[2];
    sym_rg(rr, gg, Wo, -1.0);
  }
  const int b = __ldg(in_ptr + i), e = __ldg(in_ptr + i + 1);
  if (kSort) sort_incoming(b, e - b, lane, in_slot);
  for (int x = b + lane; x < e; x += 32) {
    const size_t slot = static_cast<size_t>(in_slot[x]);
    const double* g = G + 3 * slot;
    double gg[3] = {__ldg(g), __ldg(g + 1), __ldg(g + 2)};
    F[0] -= gg[0];
    F[1] -= gg[1];
    F[2] -= gg[2];
    if (vatom) {
      const double* r = rijs + 3 * slot;
      double rr[3] = {__ldg(r), __ldg(r + 1), __ldg(r + 2)};
      sym_rg(rr, gg, Wi, -1.0);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    for (int c = 0; c < 3; ++c) F[c] += __shfl_xor_sync(0xffffffffu, F[c], o);
    for (int c = 0; c < 6; ++c) Wo[c] += __shfl_xor_sync(0xffffffffu, Wo[c], o);
    if (vatom)
      for (int c = 0; c < 6; ++c) Wi[c] += __shfl_xor_sync(0xffffffffu, Wi[c], o);
  }
  if (lane == 0) {
    forces[3 * i] = F[0];
    forces[3 * i + 1] = F[1];
    forces[3 * i + 2] = F[2];
    for (int c = 0; c < 6; ++c) wown[6 * i + c] = Wo[c];
    if (vatom)
      for (int c = 0; c < 6; ++c) vatom[6 * i + c] = 0.5 * (Wo[c] + Wi[c]);
  }
}

cudaError_t launch_force_gather(int natoms, int stride, const double* rijs, const int* counts,
                                const double* pair_grad, const int* in_ptr, int* in_slot, bool sort,
                                double* forces, double* wown, double* vatom, cudaStream_t st) {
  if (natoms <= 0) return cudaSuccess;
  const int threads = 256;
  const int blocks = (natoms * 32 + threads - 1) / threads;
  if (sort)
    k_force_gather<true><<<blocks, threads, 0, st>>>(natoms, stride, rijs, counts, pair_grad, in_ptr, in_slot, forces,
                                                     wown, vatom);
  else
    k_force_gather<false><<<blocks, threads, 0, st>>>(natoms, stride, rijs, counts, pair_grad, in_ptr, in_slot, forces,
                                                      wown, vatom);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// fixed-order totals
// ---------------------------------------------------------------------------
__device__ __forceinline__ double block_reduce_256(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < 8; ++w) s += red[w];
  __syncthreads();
  return s;
}

// Totals of the site energies and virials in one launch: every block sums its
// chunk, and the block that finishes last adds the blocks' partials (which
// block that is does not matter: the order is fixed).  One warp per total
// there: lane l adds partials l, l + 32, ... in order, then a fixed butterfly
// over the lanes.  out[0..6] = totals, out[7] = the device error flags so far
// (low 32 bits), so a host call reads both back with one copy; d_energy and
// d_virial, where given, get theirs.  The ticket at out + 8 starts at zero and
// wraps to zero after every grid's worth of blocks, also where launches on the
// same scratch overlap (calls of the allocation-free path may race): such calls
// spoil their own totals, not those of the calls after them.  Two launches and
// two copies took 9 us of a 2,000-atom call.
__global__ void k_totals(int natoms, const double* __restrict__ e, const double* __restrict__ w, double* partials,
                         double* out, const int* err, double* d_energy, double* d_virial) {
  __shared__ double red[7][8];
  __shared__ bool last;
  const int chunk = (natoms + gridDim.x - 1) / gridDim.x;
  const int b = min(natoms, static_cast<int>(blockIdx.x) * chunk), en = min(natoms, b + chunk);
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int i = b + threadIdx.x; i < en; i += blockDim.x) {
    acc[0] += e[i];
    for (int c = 0; c < 6; ++c) acc[1 + c] += w[6 * i + c];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if (lane == 0) red[c][warp] = acc[c];
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    double s = 0.0;
    for (int k = 0; k < 8; ++k) s += red[threadIdx.x][k];
    partials[7 * blockIdx.x + threadIdx.x] = s;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicInc(reinterpret_cast<unsigned*>(out + 8), gridDim.x - 1) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (warp < 7) {
    double s = 0.0;
    for (int k = lane; k < static_cast<int>(gridDim.x); k += 32) s += __ldcg(partials + 7 * k + warp);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      out[warp] = s;
      if (warp == 0 && d_energy) *d_energy = s;
      if (warp > 0 && d_virial) d_virial[warp - 1] = s;
    }
  } else if (lane == 0) {
    out[7] = __hiloint2double(0, *reinterpret_cast<const volatile int*>(err));
  }
}

// Neighbour rows from positions, one warp per local atom: the candidates of
// the atom's list closer than the cutoff are kept in list order (a ballot and
// a prefix count give each kept candidate its slot), with r_ij = x_j - x_i,
// the owner index of j and its species (-1 for a ghost without an owner).  It
// also counts the incoming slots of each owner (in_cnt, zero before).
// This is the host packing loop of the pair style (pair_jax_mtp.cpp:110-167)
// on the device: r^2 is formed with separately rounded products and sums, as
// that loop does, so the same candidates are kept.
__global__ void k_rows_from_positions(int nlocal, int nall, const double* __restrict__ x,
                                      const int* __restrict__ species, const int* __restrict__ owner,
                                      int list_stride, const int* __restrict__ neigh,
                                      const int* __restrict__ numneigh, double cut2, int stride,
                                      double* __restrict__ rijs, int* __restrict__ js, int* __restrict__ jtypes,
                                      int* __restrict__ counts, int* __restrict__ in_cnt, int* __restrict__ err) {
  const int i = static_cast<int>((static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= nlocal) return;   // the warp leaves together
  const double xi = x[3 * i], yi = x[3 * i + 1], zi = x[3 * i + 2];
  const int n = min(max(numneigh[i], 0), list_stride);
  const int* row = neigh + static_cast<size_t>(i) * list_stride;
  int kept = 0;
  for (int c0 = 0; c0 < n; c0 += 32) {
    const int c = c0 + lane;
    bool keep = false;
    double dx = 0.0, dy = 0.0, dz = 0.0;
    int j = -1;
    if (c < n) {
      j = row[c];
      if (j >= 0 && j < nall && j != i) {
        dx = x[3 * j] - xi;
        dy = x[3 * j + 1] - yi;
        dz = x[3 * j + 2] - zi;
        const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        keep = r2 < cut2;
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (keep) {
      const int slot = kept + __popc(m & ((1u << lane) - 1u));
      if (slot < stride) {
        const size_t o = static_cast<size_t>(i) * stride + slot;
        rijs[3 * o] = dx;
        rijs[3 * o + 1] = dy;
        rijs[3 * o + 2] = dz;
        const int own = owner[j];
        const int t = own >= 0 ? species[j] : -1;
        js[o] = own;
        jtypes[o] = t;
        if (t >= 0 && own < nlocal) atomicAdd(in_cnt + own, 1);   // as k_count_incoming
      }
    }
    kept += __popc(m);
  }
  if (lane == 0) {
    counts[i] = min(kept, stride);
    if (kept > stride) atomicOr(err, kErrCapacity);
  }
}

cudaError_t launch_rows_from_positions(int nlocal, int nall, const double* x, const int* species, const int* owner,
                                       int list_stride, const int* neigh, const int* numneigh, double cutoff,
                                       int stride, double* rijs, int* js, int* jtypes, int* counts, int* in_cnt,
                                       int* err, cudaStream_t st) {
  if (nlocal <= 0) return cudaSuccess;
  const cudaError_t e = cudaMemsetAsync(in_cnt, 0, sizeof(int) * nlocal, st);
  if (e != cudaSuccess) return e;
  const size_t threads = static_cast<size_t>(nlocal) * 32;
  k_rows_from_positions<<<static_cast<unsigned>((threads + 255) / 256), 256, 0, st>>>(
      nlocal, nall, x, species, owner, list_stride, neigh, numneigh, cutoff * cutoff, stride, rijs, js, jtypes,
      counts, in_cnt, err);
  return cudaGetLastError();
}

cudaError_t launch_totals(int natoms, const double* site_energy, const double* wown, double* partials,
                          double* out, const int* err, double* d_energy, double* d_virial, cudaStream_t st) {
  k_totals<<<kReduceBlocks, 256, 0, st>>>(natoms, site_energy, wown, partials, out, err, d_energy, d_virial);
  return cudaGetLastError();
}

__global__ void k_config_ptr(int natoms, int nconfig, const int* cfg, int* ptr, int* err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > natoms) return;
  const int c = i < natoms ? cfg[i] : nconfig;
  const int p = i > 0 ? cfg[i - 1] : -1;
  if (c < p || (i < natoms && (c < 0 || c >= nconfig))) {
    atomicOr(err, kErrCapacity);
    return;
  }
  for (int x = p + 1; x <= c; ++x) ptr[x] = i;
}

cudaError_t launch_config_ptr(int natoms, int nconfig, const int* cfg_of_atom, int* cfg_ptr, int* err,
                              cudaStream_t st) {
  cudaMemsetAsync(cfg_ptr, 0, sizeof(int) * (nconfig + 1), st);
  k_config_ptr<<<(natoms + 1 + 255) / 256, 256, 0, st>>>(natoms, nconfig, cfg_of_atom, cfg_ptr, err);
  return cudaGetLastError();
}

__global__ void k_config_totals(int natoms, const int* __restrict__ ptr, const double* __restrict__ e,
                                const double* __restrict__ w, const double* __restrict__ vol,
                                double* __restrict__ energy, double* __restrict__ stress) {
  __shared__ double red[8];
  const int c = blockIdx.x;
  const int b = min(max(ptr[c], 0), natoms), en = min(max(ptr[c + 1], b), natoms);
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int i = b + threadIdx.x; i < en; i += blockDim.x) {
    acc[0] += e[i];
    for (int k = 0; k < 6; ++k) acc[1 + k] += w[6 * i + k];
  }
  double tot[7];
  for (int k = 0; k < 7; ++k) tot[k] = block_reduce_256(acc[k], red);
  if (threadIdx.x == 0) {
    energy[c] = tot[0];
    // wown = -sym(sum r g) in xx,yy,zz,xy,xz,yz; the reference stress is
    // +sym(sum r g)/V in xx,yy,zz,yz,xz,xy
    const double iv = 1.0 / vol[c];
    stress[6 * c + 0] = -tot[1] * iv;
    stress[6 * c + 1] = -tot[2] * iv;
    stress[6 * c + 2] = -tot[3] * iv;
    stress[6 * c + 3] = -tot[6] * iv;
    stress[6 * c + 4] = -tot[5] * iv;
    stress[6 * c + 5] = -tot[4] * iv;
  }
}

cudaError_t launch_config_totals(int natoms, int nconfig, const int* cfg_ptr, const double* site_energy,
                                 const double* wown, const double* volumes, double* energy, double* stress,
                                 cudaStream_t st) {
  if (nconfig <= 0) return cudaSuccess;
  k_config_totals<<<nconfig, 256, 0, st>>>(natoms, cfg_ptr, site_energy, wown, volumes, energy, stress);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// FMA peak probe: 8 independent chains per thread
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_fma_chain(int iters, T seed, T* out) {
  T a0 = seed + threadIdx.x, a1 = a0 + T(1), a2 = a0 + T(2), a3 = a0 + T(3);
  T a4 = a0 + T(4), a5 = a0 + T(5), a6 = a0 + T(6), a7 = a0 + T(7);
  const T m = T(0.999999), c = T(1e-7);
  for (int k = 0; k < iters; ++k) {
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      a0 = a0 * m + c; a1 = a1 * m + c; a2 = a2 * m + c; a3 = a3 * m + c;
      a4 = a4 * m + c; a5 = a5 * m + c; a6 = a6 * m + c; a7 = a7 * m + c;
    }
  }
  const T r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (r == T(-12345.678)) out[0] = r;   // keeps the chains alive
}

template <typename T>
static double time_fma(int sms) {
  T* out = nullptr;
  if (cudaMalloc(&out, sizeof(T)) != cudaSuccess) return 0.0;
  const int threads = 256, blocks = sms * 8, iters = 2048;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  k_fma_chain<T><<<blocks, threads>>>(16, T(1), out);   // warm-up
  cudaEventRecord(a);
  k_fma_chain<T><<<blocks, threads>>>(iters, T(1), out);
  cudaEventRecord(b);
  cudaEventSynchronize(b);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(out);
  const double flops = 2.0 * 8 * 16 * static_cast<double>(iters) * threads * blocks;
  return ms > 0 ? flops / (ms * 1e-3) / 1e12 : 0.0;
}

cudaError_t measure_fma_peak(double* fp64_tflops, double* fp32_tflops) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  double d = 0, f = 0;
  for (int rep = 0; rep < 3; ++rep) {
    d = std::max(d, time_fma<double>(sms));
    f = std::max(f, time_fma<float>(sms));
  }
  *fp64_tflops = d;
  *fp32_tflops = f;
  return cudaGetLastError();
}

}  // namespace mtp
