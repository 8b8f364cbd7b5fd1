// mtp_device.cuh - sm_100a kernels of the MTP evaluator.
//
// One persistent thread block evaluates A centre atoms at a time (a
// grid-stride loop over groups of A atoms):
//
//   N1  neighbour staging: the slots of the atoms' padded rows are read with
//       coalesced loads in one sweep, tested (t_j >= 0, |r| < max_dist),
//       compacted with warp ballots, and each kept neighbour gets its unit
//       vector, distance, radial functions f_mu(d), f'_mu(d) (Chebyshev basis
//       times the smooth cutoff, jax_backend.py:83-95, 108-160) and the powers
//       of its unit vector components, all in shared memory;
//   N2  basic moments m[(mu, a, b, c)] = sum_j f_mu(d_j) u_x^a u_y^b u_z^c
//       (conversion.py:66-81), one thread per (atom, monomial), only the
//       radial functions that have a moment at the monomial's degree;
//   T   contraction tree (conversion.py:95-102) by the lane programs of the
//       schedule, then E_i = xi[t_i] + theta . m[mapping] (jax_backend.py:101-106);
//   R   reverse programs: dE_i/dm for every moment, gathered per source, so
//       no two threads ever add into the same value;
//   N3  per neighbour: dE_i/dr_ij from dE_i/dm of the basic moments by nested
//       Horner over the monomial simplex (the analytic form of
//       jax.value_and_grad at jax_backend.py:56), one neighbour per lane,
//       written to the per-slot gradient array.
//
// The A atoms of a block share every lane-program entry: their values are
// interleaved [slot][atom] so one vector access serves all of them.
//
// Forces then come from a per-atom gather (k_force_gather): the atom's own
// slot gradients minus the gradients of the slots that point at it, in a
// fixed order, so results are bitwise reproducible without atomics
// (jax_backend.py:263-303 uses an atomic segment_sum instead).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "mtp_model.hpp"

namespace mtp {

enum ErrBits : int { kErrNonFinite = 1, kErrSpecies = 2, kErrCapacity = 4 };

struct DevPass {
  int offset;
  int steps;
};

// Everything the evaluation kernel needs about the potential (device pointers).
struct DevModel {
  const uint2* entries;
  DevPass fwd[kMaxPasses];
  DevPass rev[kMaxPasses];
  int nfwd, nrev;
  // steps each warp runs in each pass, [nfwd + nrev][lanes / 32]: a warp
  // stops after its longest lane's program (Pass::wsteps)
  const int* warp_steps;
  const double* radial;     // [S][S][R][K]
  const double* species;    // [S]
  const double* theta;      // [Sa]
  const int* mapping;       // [Sa]
  const int* seed_idx;      // [nseed]
  const double* seed_val;   // [nseed]
  const int* zero_list;     // [nzero]
  const int* mono_word;     // [P] Schedule::mono_word
  const int* mono_list;     // [n_list] Schedule::mono_list
  int n_list;
  const int* dm_zero;       // [ndm_zero] adjoint positions no pass stores and no seed sets
  int nseed, nzero, ndm_zero;
  int S, R, K, M, B, P, D, Sa;
  int chain_mode;           // Schedule::chain_mode
  int n3_len;               // Schedule::n3_len
  const int* n3_src;        // [n3_len] adjoint position of each chain slot, or -1
  // Schedule::n3_words and n3_off, here among the kernel's parameters: read
  // with a warp-uniform index they are uniform values, so the chains' branches
  // are uniform ones (from shared memory, every step of a chain paid for a
  // possibly divergent branch)
  int n3_words[kMaxChains];
  unsigned char n3_off[kMaxRunOffsets];
  int v_m, v_dm, n_dm, v_zero, v_one, v_size;  // n_dm: slots of the adjoint region
  double scaling, rmin, rmax;
};

struct DevIO {
  int natoms;
  int nbr_stride;
  int n_pad;                // slots of a staging row (>= max count, <= nbr_stride rounded)
  int qs;                   // its stride (EvalFit; set by launch_eval)
  const int* itypes;        // [natoms]
  const double* rijs;       // [natoms][nbr_stride][3]
  const int* jtypes;        // [natoms][nbr_stride]
  const int* counts;        // [natoms] or null
  double* site_energy;      // [natoms]
  double* pair_grad;        // [natoms][nbr_stride][3]
  int* err;                 // error bits
  void* vscratch;           // [grid][v_size] value space when it lives in global memory
};

// Lane-program entries requested ahead of use (registers), per thread.
constexpr int kPrefetch = kStepAlign;

// Neighbours (or radial functions) one 16-byte shared-memory access covers.
template <typename T>
constexpr int kVec = 16 / static_cast<int>(sizeof(T));

// Shared-memory carve of the evaluation kernel for A atoms per block.  The
// value space is interleaved [slot][atom] so one vector access serves all A
// atoms.  Neighbour staging is kept per atom as rows over the kept neighbours
// (radial functions f_mu, their derivatives, 1/d, the powers of u_x, u_y and
// u_z), so that the basic moments read several neighbours with one 16-byte
// load and the force phase, whose lanes are neighbours, reads without bank
// conflicts.  The row stride is an odd number of 16-byte words: 8 lanes that read
// 8 rows in turn at the same neighbour hit 8 different bank groups (row_stride).
// The force phase's chain copy of dE/dm ([atom][n3_len])
// and its partial sums take the moment half of the value space (dead once the
// reverse passes are done) when they fit there.
struct SmemLayout {
  int qs;         // stride of a staging row
  int rows;       // staging rows per atom: R (f), R (f'), 1 (1/d), 3 power_rows(D)
  int rp;         // radial functions per coefficient row (R rounded up to kVec)
  int n3s;        // stride of one atom's chain copy
  size_t v, rad, st, slot, mono, dmc, n3p, red, cnt, total;
};

// Force-phase words: one FP64 value or a pair of FP32 ones (struct Force).
constexpr int kForceBytes = 8;

// Powers of a unit vector component in the staging: up to the degree, and the
// first one always (levels 2 and 4 have scalar moments only, but their forces
// point along the unit vector too).
__host__ __device__ inline int power_rows(int D) { return D < 1 ? 2 : D + 1; }

// Warps that share one chunk of neighbours (32 lanes of `items`) in the force
// phase: as few as let every chunk of the block have a group (no partial sums
// to exchange when it is one warp), for rows filled to three quarters.  A rule
// on the launch alone: an atom's rounding must not depend on the atoms beside
// it.
__host__ __device__ inline int n3_group_warps(int NW, int A, int n_pad, int items) {
  const int chunks = (A * n_pad * 3 / 4 + 32 * items - 1) / (32 * items);
  int gw = NW;
  while (gw > 1 && NW / gw < chunks) gw >>= 1;
  return gw;
}

// Shared memory of an SM, what a block takes beside its own, and what one block
// can have.
constexpr size_t kSmemPerSM = 228 * 1024, kSmemReserved = 1024, kMaxSmemPerBlock = 227 * 1024;

// Stride of a staging row of n_pad slots.  An odd number of 16-byte words (see
// SmemLayout); where that is one word more than the slots need and without it
// another block fits on an SM (`total` gives a block's bytes for a stride), the
// slots' own words, whose bank conflicts in the basic moments cost less.
template <typename T, typename Total>
inline int row_stride(int n_pad, int threads, const Total& total) {
  const int words = (n_pad + kVec<T> - 1) / kVec<T>;
  auto blocks = [&](int w) {   // by shared memory and by registers (128 a thread)
    const size_t bytes = total(w * kVec<T>);
    return bytes > kMaxSmemPerBlock ? 0 : std::min<size_t>(512 / threads, kSmemPerSM / (bytes + kSmemReserved));
  };
  return (blocks(words) > blocks(words | 1) ? words : words | 1) * kVec<T>;
}

template <typename T>
__host__ __device__ inline SmemLayout smem_layout(int v_size, int M, int S, int R, int K, int D, int P, int n_list,
                                                  int n3_len, int n_pad, int qs, int threads, int A) {
  SmemLayout L;
  L.qs = qs;
  L.rows = 2 * R + 1 + 3 * power_rows(D);
  L.rp = (R + kVec<T> - 1) / kVec<T> * kVec<T>;
  // an atom's copy starts one 16-byte word further into the banks than the one before
  L.n3s = ((n3_len + 15) & ~15) + 2;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    size_t at = (o + 31) & ~size_t(31);
    o = at + bytes;
    return at;
  };
  L.v = take(sizeof(T) * v_size * A);
  L.rad = take(sizeof(T) * S * S * L.rp * K);
  L.st = take(sizeof(T) * L.rows * L.qs * A);
  L.slot = take(sizeof(int) * n_pad * A);
  // tables that every iteration reads: with most of the SM's memory taken as
  // shared memory there is next to no L1 left, and a load from L2 costs more
  // than a monomial's work
  L.mono = take(sizeof(int) * P + sizeof(uint16_t) * n_list);
  const size_t dmc = kForceBytes * static_cast<size_t>(L.n3s) * A;
  // (G_x, G_y, G_z, S) of each thread, exchanged where several warps share a chunk
  const bool shared = n3_group_warps(threads / 32, A, n_pad, kForceBytes / static_cast<int>(sizeof(T))) > 1;
  const size_t n3p = shared ? kForceBytes * 4 * static_cast<size_t>(threads) : 0;
  const size_t dead = v_size > 0 ? sizeof(T) * M * A : 0;
  L.dmc = dmc <= dead ? L.v : take(dmc);
  L.n3p = L.dmc == L.v && dmc + n3p <= dead ? L.v + dmc : take(n3p);
  L.red = take(sizeof(double) * (threads / 32) * A);
  L.cnt = take(sizeof(int) * (threads / 32 + A));   // per-warp counts, then the atoms' species
  L.total = (o + 31) & ~size_t(31);
  return L;
}

__device__ __forceinline__ double dev_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float dev_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double dev_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float dev_fma(float a, float b, float c) { return fmaf(a, b, c); }

// A values of one value-space slot, loaded/stored as one vector access.
template <typename T, int A>
struct __align__(sizeof(T) * A) Pack {
  T v[A];
};

// Integer multiplicity of an entry (y & kMultMask < 2^14) as T without an
// int-to-float conversion instruction: OR-ing m into the mantissa of 2^23
// (2^52) gives the float (double) 2^23 + m exactly, and subtracting 2^23
// (2^52) leaves m exactly.
template <typename T>
__device__ __forceinline__ T entry_mult(uint32_t y);
template <>
__device__ __forceinline__ float entry_mult<float>(uint32_t y) {
  return __int_as_float(static_cast<int>((y & kMultMask) | 0x4B000000u)) - 8388608.0f;
}
template <>
__device__ __forceinline__ double entry_mult<double>(uint32_t y) {
  return __hiloint2double(0x43300000, static_cast<int>(y & kMultMask)) - 4503599627370496.0;
}

// Stream one lane program pass: every thread walks its column of the
// [steps][LANES] entry array with PF entries in flight (registers), so the L2
// latency of the program overlaps the arithmetic.  LANES is a template
// argument so every request is one load at a constant offset; PF divides
// kStepAlign, so steps is a multiple of PF and the program holds PF rows after
// any pass: nothing is bounds-tested.  Each entry feeds A atoms:
// acc[a] += c * V[x][a] * V[y][a]; STORE/ADD flush into V[d][a].
// Operands are read through Vr and flushes go through V: a pass never reads a
// slot that it writes, so the two views do not alias.  The operand
// gathers of all PF entries in flight are issued before any of their flushes
// (allowed for the same reason); with the value space in global memory this
// overlaps PF gathers' latencies (level-28 FP64 forward 54.1 -> 38.4 ms at
// 32,000 atoms), in shared memory it gains 0.1-0.6 % at the tuned shapes
// (2.5 % at 256 lanes x 1 atom in FP64).
template <typename T, int A, int LANES, int PF>
__device__ __forceinline__ void run_pass(const uint2* __restrict__ ent, int steps, T* __restrict__ V,
                                         const T* __restrict__ Vr) {
  static_assert(PF >= 1 && kStepAlign % PF == 0, "prefetch depth must divide the pass step alignment");
  const uint2* p = ent;
  uint2 buf[PF];
#pragma unroll
  for (int k = 0; k < PF; ++k) buf[k] = __ldg(p + k * LANES);
  T acc[A];
#pragma unroll
  for (int a = 0; a < A; ++a) acc[a] = T(0);
  for (int s0 = 0; s0 < steps; s0 += PF) {
    p += PF * LANES;
    uint2 ek[PF];
    Pack<T, A> va[PF], vb[PF];
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      ek[k] = buf[k];
      va[k] = *reinterpret_cast<const Pack<T, A>*>(Vr + (ek[k].x & 0xFFFFu) * A);
      vb[k] = *reinterpret_cast<const Pack<T, A>*>(Vr + (ek[k].x >> 16) * A);
      buf[k] = __ldg(p + k * LANES);
    }
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      const uint2 e = ek[k];
      const T c = entry_mult<T>(e.y);
#pragma unroll
      for (int a = 0; a < A; ++a) acc[a] = dev_fma(c * va[k].v[a], vb[k].v[a], acc[a]);
      if (e.y & (3u << kOpShift)) {
        Pack<T, A>* dst = reinterpret_cast<Pack<T, A>*>(V + (e.y >> kDstShift) * A);
        Pack<T, A> out;
        if (e.y & (kOpStore << kOpShift)) {
#pragma unroll
          for (int a = 0; a < A; ++a) out.v[a] = acc[a];
        } else {
          out = *dst;
#pragma unroll
          for (int a = 0; a < A; ++a) out.v[a] += acc[a];
        }
        *dst = out;
#pragma unroll
        for (int a = 0; a < A; ++a) acc[a] = T(0);
      }
    }
  }
}

// Lane p of every warp gets its warp's step count of pass p (forward passes,
// then reverse ones; at most 32 passes), so a pass reads its count with a
// shuffle instead of a load.
__device__ __forceinline__ int warp_steps_of_lane(const DevModel& md, int tid, int NT) {
  const int p = tid & 31;
  return p < md.nfwd + md.nrev ? __ldg(md.warp_steps + p * (NT >> 5) + (tid >> 5)) : 0;
}

// Generic lane-program streamer (used by the dual-number kernels): every thread
// walks its column of the [steps][LANES] entries with PF in flight.  PF divides
// kStepAlign, so steps is a multiple of PF and the rows after a pass exist;
// LANES is fixed so every request is one load at a constant offset.  A Body
// has load(e) (the entry's operand gathers) and apply(e, operands) (the
// arithmetic and the flush); with kEarly the gathers of all PF entries are
// issued before the first apply, which a pass allows because it never reads a
// slot that it writes.
template <int LANES, int PF, bool kEarly, typename Body>
__device__ __forceinline__ void stream_entries_t(const uint2* __restrict__ ent, int steps, int tid, Body& body) {
  static_assert(PF >= 1 && kStepAlign % PF == 0, "prefetch depth must divide the pass step alignment");
  const uint2* p = ent + tid;
  uint2 buf[PF];
#pragma unroll
  for (int k = 0; k < PF; ++k) buf[k] = __ldg(p + k * LANES);
  for (int s0 = 0; s0 < steps; s0 += PF) {
    p += PF * LANES;
    uint2 ek[PF];
    typename Body::Operands op[PF];
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      ek[k] = buf[k];
      if (kEarly) op[k] = body.load(ek[k]);
      buf[k] = __ldg(p + k * LANES);
    }
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      if (!kEarly) op[k] = body.load(ek[k]);
      body.apply(ek[k], op[k]);
    }
  }
}

template <int PF, bool kEarly, typename Body>
__device__ __forceinline__ void stream_entries_n(const uint2* __restrict__ ent, int steps, int lanes, int tid,
                                                 Body& body) {
  if (lanes == 512) stream_entries_t<512, PF, kEarly>(ent, steps, tid, body);
  else if (lanes == 256) stream_entries_t<256, PF, kEarly>(ent, steps, tid, body);
  else stream_entries_t<128, PF, kEarly>(ent, steps, tid, body);
}

// Two FP32 values in a 64-bit register (one instruction for two FMAs).
using Two = unsigned long long;
__device__ __forceinline__ Two pack2(float a, float b) {
  Two r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(Two a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ Two mul2(Two a, Two b) {
  Two r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ Two fma2(Two a, Two b, Two c) {
  Two r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// What a lane of the force phase computes with: two neighbours of one atom
// side by side in FP32 (two-wide instructions), one neighbour in FP64.
template <typename T>
struct Force;
template <>
struct Force<float> {
  using P = Two;
  static constexpr int kItems = 2;
  static __device__ __forceinline__ P make(float a, float b) { return pack2(a, b); }
  static __device__ __forceinline__ P fma(P a, P b, P c) { return fma2(a, b, c); }
  static __device__ __forceinline__ P mul(P a, P b) { return mul2(a, b); }
  static __device__ __forceinline__ float get(P a, int i) { return i ? unpack2(a).y : unpack2(a).x; }
};
template <>
struct Force<double> {
  using P = double;
  static constexpr int kItems = 1;
  static __device__ __forceinline__ P make(double a, double) { return a; }
  static __device__ __forceinline__ P fma(P a, P b, P c) { return ::fma(a, b, c); }
  static __device__ __forceinline__ P mul(P a, P b) { return a * b; }
  static __device__ __forceinline__ double get(P a, int) { return a; }
};

// Radial functions at step k of a force-phase chain (k = D - degree) on a
// level-structured basis of offset OFF (Schedule::chain_mode).
template <int R, int OFF>
__host__ __device__ constexpr int chain_nm(int k) {
  return (k + OFF) / 2 + 1 < R ? (k + OFF) / 2 + 1 : R;
}
template <int R, int OFF>
__host__ __device__ constexpr int chain_len(int top) {
  int n = 0;
  for (int k = 0; k <= top; ++k) n += chain_nm<R, OFF>(k);
  return n;
}

// Horner chain in u_z of the monomial pair (a, b): steps k = 0 .. top go from
// u_z^top down, step k adding sum_mu g f_mu (and g f'_mu) over its radial
// functions.  h = sum_c w_c u_z^c, hz its u_z-derivative, hs the same sum with
// f'.  The chain's adjoints g are contiguous (in FP32 each is there twice, for
// the lane's two neighbours), so they come in 16-byte loads, requested kAhead
// words before their use; the last requests may lie past the chain (and are
// not used).  One body serves every length and stops at top: a body per length
// was 10 KB of code that each warp walked through once a chain, and fetching
// it cost more than the arithmetic.
template <typename T, int R, int OFF>
__device__ __forceinline__ void chain(int top, const typename Force<T>::P* __restrict__ g,
                                      const typename Force<T>::P (&f)[R], const typename Force<T>::P (&fp)[R],
                                      typename Force<T>::P uz, typename Force<T>::P& h, typename Force<T>::P& hz,
                                      typename Force<T>::P& hs) {
  using F = Force<T>;
  using P = typename F::P;
  constexpr int N = chain_len<R, OFF>(kMaxDegree), NV = (N + 1) / 2, kAhead = 3;
  struct __align__(16) Word { P v[2]; };
  const Word* gw = reinterpret_cast<const Word*>(g);
  P v[NV * 2];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) *reinterpret_cast<Word*>(v + 2 * i) = gw[i];
  h = hz = hs = F::make(T(0), T(0));
  int at = 0;
#pragma unroll
  for (int k = 0; k <= kMaxDegree; ++k) {
    if (k > top) break;
    P w = F::make(T(0), T(0)), wp = w;
#pragma unroll
    for (int mu = 0; mu < chain_nm<R, OFF>(k); ++mu) {
      if (at % 2 == 0 && at / 2 + kAhead < NV) *reinterpret_cast<Word*>(v + at + 2 * kAhead) = gw[at / 2 + kAhead];
      w = F::fma(v[at], f[mu], w);
      wp = F::fma(v[at], fp[mu], wp);
      ++at;
    }
    hz = F::fma(hz, uz, h);
    h = F::fma(h, uz, w);
    hs = F::fma(hs, uz, wp);
  }
}

// The same chain on a basis without the level structure: every step has all R
// radial functions (zero adjoints where the basis has no moment).
template <typename T, int R>
__device__ __forceinline__ void chain_dense(int top, const typename Force<T>::P* __restrict__ g,
                                            const typename Force<T>::P (&f)[R], const typename Force<T>::P (&fp)[R],
                                            typename Force<T>::P uz, typename Force<T>::P& h,
                                            typename Force<T>::P& hz, typename Force<T>::P& hs) {
  using F = Force<T>;
  using P = typename F::P;
  h = hz = hs = F::make(T(0), T(0));
  for (int k = 0; k <= top; ++k, g += R) {
    P w = F::make(T(0), T(0)), wp = w;
#pragma unroll
    for (int mu = 0; mu < R; ++mu) {
      w = F::fma(g[mu], f[mu], w);
      wp = F::fma(g[mu], fp[mu], wp);
    }
    hz = F::fma(hz, uz, h);
    h = F::fma(h, uz, w);
    hs = F::fma(hs, uz, wp);
  }
}

// Force phase.  A lane takes one kept neighbour (FP64) or two of one atom, q
// and q + ceil(nv / 2) (FP32); chunk c holds the lanes j = 32 c + lane over the
// A atoms' lists in turn.  Groups of GW warps take the chunks in turn; the
// warps of a group split the monomial pairs (a, b), ordered by b and then a
// descending, into runs of about equal cost (Schedule::n3_words).
// Chains of one b are gathered by Horner in u_x as they come, so a pair costs
// four multiply-adds beside its chain; a segment's end (the last pair of one b
// or of the run) applies the powers of u_y and of the x-exponent where the
// segment stopped.  With W_s = sum_mu Dm[s][mu] f_mu(d) over monomials s and
// W'_s the same with f': G = grad_u sum_s W_s u^s and S = sum_s W'_s u^s.
// Partial sums of a group's warps are added in warp order (deterministic).
// Bound by the latency of the chains (two dependent multiply-adds a step): level
// 24 mixed at 512 lanes x 4 atoms, 15,800 cycles an iteration, 18,400 with lanes
// on neighbours but the adjoints read one value per load from the value space.
template <typename T, int A, int R, int MODE>
__device__ __forceinline__ void force_phase(const DevModel& md, const DevIO& io, const SmemLayout& L,
                                            unsigned char* smem, const int (&nv_a)[A], int base, int tid, int NT) {
  using F = Force<T>;
  using P = typename F::P;
  constexpr int kItems = F::kItems;
  const int w = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, NW = NT >> 5;   // known to be warp-uniform
  const int GW = n3_group_warps(NW, A, io.n_pad, kItems), g = w / GW, wg = w - g * GW, NG = NW / GW;
  const int lg = 31 - __clz(GW);
  // offsets of the cut into 2^lg runs follow those of the cuts into fewer
  const int i0 = md.n3_off[GW - 1 + lg + wg], i1 = md.n3_off[GW + lg + wg];
  const int D1 = power_rows(md.D), qs = L.qs, n_pad = io.n_pad;
  P* part = reinterpret_cast<P*>(smem + L.n3p);
  int J = 0;
#pragma unroll
  for (int a = 0; a < A; ++a) J += (nv_a[a] + kItems - 1) / kItems;
  // every group runs the same number of rounds (the block's barriers match)
  for (int r0 = 0; r0 < J; r0 += 32 * NG) {
    const int j = r0 + 32 * g + lane;
    const bool act = j < J;
    int a = 0, q = act ? j : r0, nv = nv_a[0];
#pragma unroll
    for (int aa = 0; aa + 1 < A; ++aa)
      if (a == aa && q >= (nv_a[aa] + kItems - 1) / kItems) {
        q -= (nv_a[aa] + kItems - 1) / kItems;
        a = aa + 1;
        nv = nv_a[aa + 1];
      }
    const int h2 = (nv + 1) / 2;                             // the lane's second neighbour is q + h2
    const int d2 = kItems == 2 && q + h2 < nv ? h2 : 0;      // (an odd list's last lane takes q twice)
    const T* st = reinterpret_cast<const T*>(smem + L.st) + static_cast<size_t>(a) * L.rows * qs + q;
    auto row = [&](int r) { return F::make(st[r * qs], st[r * qs + d2]); };
    const int px = 2 * R + 1, py = px + D1, pz = py + D1;    // rows of the powers
    const P* dmc = reinterpret_cast<const P*>(smem + L.dmc) + static_cast<size_t>(a) * L.n3s;
    P f[R], fp[R];
#pragma unroll
    for (int mu = 0; mu < R; ++mu) {
      f[mu] = row(mu);
      fp[mu] = row(R + mu);
    }
    const P ux = row(px + 1), uz = row(pz + 1), zero = F::make(T(0), T(0));
    P Gx = zero, Gy = zero, Gz = zero, Ss = zero, H = zero, Hx = zero, Hz = zero, Hs = zero;
    const int iend = r0 + 32 * g < J ? i1 : i0;   // a group without a neighbour left has nothing to add
    for (int i = i0; i < iend; ++i) {
      const int word = md.n3_words[i];
      const int top = word & 15;
      P h, hz, hs;
      if (MODE < 0) chain_dense<T, R>(top, dmc + (word >> 16) * 2, f, fp, uz, h, hz, hs);
      else chain<T, R, MODE < 0 ? 0 : MODE>(top, dmc + (word >> 16) * 2, f, fp, uz, h, hz, hs);
      Hx = F::fma(Hx, ux, H);
      H = F::fma(H, ux, h);
      Hz = F::fma(Hz, ux, hz);
      Hs = F::fma(Hs, ux, hs);
      const int ea = (word >> 4) & 15, eb = (word >> 8) & 15;
      if (ea == 0 || i + 1 == iend) {
        const P xa = row(px + ea), yb = row(py + eb);
        const T ca = static_cast<T>(ea), cb = static_cast<T>(eb);
        const P dxa = F::mul(F::make(ca, ca), row(px + max(ea - 1, 0)));   // 0 where the exponent is 0
        const P dyb = F::mul(F::make(cb, cb), row(py + max(eb - 1, 0)));
        const P xy = F::mul(xa, yb);
        Gx = F::fma(yb, F::fma(xa, Hx, F::mul(dxa, H)), Gx);
        Gy = F::fma(F::mul(xa, dyb), H, Gy);
        Gz = F::fma(xy, Hz, Gz);
        Ss = F::fma(xy, Hs, Ss);
        H = Hx = Hz = Hs = zero;
      }
    }
    if (GW > 1) {
      P* mine = part + w * 32 + lane;
      mine[0] = Gx;
      mine[NT] = Gy;
      mine[2 * NT] = Gz;
      mine[3 * NT] = Ss;
      __syncthreads();
      if (wg == 0) {
        const P one = F::make(T(1), T(1));
        for (int x = 1; x < GW; ++x) {
          const P* o = mine + x * 32;
          Gx = F::fma(one, o[0], Gx);
          Gy = F::fma(one, o[NT], Gy);
          Gz = F::fma(one, o[2 * NT], Gz);
          Ss = F::fma(one, o[3 * NT], Ss);
        }
      }
    }
    if (wg == 0 && act) {
#pragma unroll
      for (int k = 0; k < kItems; ++k) {
        if (k == 1 && d2 == 0) break;
        const T uxk = F::get(ux, k), uyk = st[(py + 1) * qs + (k ? d2 : 0)], uzk = F::get(uz, k);
        const T inv_d = st[2 * R * qs + (k ? d2 : 0)];
        const T Gxk = F::get(Gx, k), Gyk = F::get(Gy, k), Gzk = F::get(Gz, k), Sk = F::get(Ss, k);
        const T ug = uxk * Gxk + uyk * Gyk + uzk * Gzk;
        const T gx = uxk * Sk + (Gxk - uxk * ug) * inv_d;
        const T gy = uyk * Sk + (Gyk - uyk * ug) * inv_d;
        const T gz = uzk * Sk + (Gzk - uzk * ug) * inv_d;
        const int slot = reinterpret_cast<const int*>(smem + L.slot)[a * n_pad + q + (k ? d2 : 0)];
        double* grow = io.pair_grad + (static_cast<size_t>(base + a) * io.nbr_stride + slot) * 3;
        grow[0] = static_cast<double>(gx);
        grow[1] = static_cast<double>(gy);
        grow[2] = static_cast<double>(gz);
        if (!(isfinite(static_cast<double>(gx)) && isfinite(static_cast<double>(gy)) &&
              isfinite(static_cast<double>(gz))))
          atomicOr(io.err, kErrNonFinite);
      }
    }
    // the next chunk's partial sums may only overwrite these once they are added
    if (GW > 1 && r0 + 32 * NG < J) __syncthreads();
  }
}

// Basic moments of one (atom, monomial) task for NM radial functions:
// acc[mu] = sum_q f_mu(d_q) u_x^a u_y^b u_z^c over the kept neighbours, kVec
// neighbours per 16-byte load (rows are padded to that with f = 0).  FP32 sums
// the even and the odd neighbours side by side in two-wide instructions.
template <int NM>
__device__ __forceinline__ void moment_task(const float* __restrict__ f, int qs, const float* __restrict__ px,
                                            const float* __restrict__ py, const float* __restrict__ pz, int nv,
                                            float (&acc)[kMaxR]) {
  Two s[NM];
#pragma unroll
  for (int mu = 0; mu < NM; ++mu) s[mu] = pack2(0.f, 0.f);
#pragma unroll 2
  for (int q = 0; q < nv; q += 4) {
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(px + q), y = *reinterpret_cast<const ulonglong2*>(py + q),
                     z = *reinterpret_cast<const ulonglong2*>(pz + q);
    const Two m0 = mul2(mul2(x.x, y.x), z.x), m1 = mul2(mul2(x.y, y.y), z.y);
#pragma unroll
    for (int mu = 0; mu < NM; ++mu) {
      const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(f + mu * qs + q);
      s[mu] = fma2(g.x, m0, s[mu]);
      s[mu] = fma2(g.y, m1, s[mu]);
    }
  }
#pragma unroll
  for (int mu = 0; mu < NM; ++mu) acc[mu] = unpack2(s[mu]).x + unpack2(s[mu]).y;
}

template <int NM>
__device__ __forceinline__ void moment_task(const double* __restrict__ f, int qs, const double* __restrict__ px,
                                            const double* __restrict__ py, const double* __restrict__ pz, int nv,
                                            double (&acc)[kMaxR]) {
#pragma unroll 2
  for (int q = 0; q < nv; q += 2) {
    const double2 x = *reinterpret_cast<const double2*>(px + q), y = *reinterpret_cast<const double2*>(py + q),
                  z = *reinterpret_cast<const double2*>(pz + q);
    const double m0 = x.x * y.x * z.x, m1 = x.y * y.y * z.y;
#pragma unroll
    for (int mu = 0; mu < NM; ++mu) {
      const double2 g = *reinterpret_cast<const double2*>(f + mu * qs + q);
      acc[mu] = fma(g.x, m0, acc[mu]);
      acc[mu] = fma(g.y, m1, acc[mu]);
    }
  }
}

// Per-warp sums of A doubles per thread: lane 0 of warp w writes atom a's
// sum to red[a * warps + w] (summed later in warp order: deterministic).
template <int A>
__device__ __forceinline__ void warp_partials(double (&v)[A], double* red) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
  for (int a = 0; a < A; ++a) {
    for (int o = 16; o > 0; o >>= 1) v[a] += __shfl_xor_sync(0xffffffffu, v[a], o);
    if (l == 0) red[a * nw + w] = v[a];
  }
}

// ---------------------------------------------------------------------------
// evaluation kernel
// ---------------------------------------------------------------------------
// A atoms per block share every lane-program entry.  kVGlobal: the value
// space (moments, adjoints, partials) is a private slice of global memory
// (L1/L2-resident) instead of shared memory; used when it does not fit in
// shared memory (level 28 in FP64).
//
// What bounds it: shared-memory wavefronts.  Level 24 mixed at 512 lanes x 4
// atoms keeps 16 warps and all of an SM's shared memory busy with one block; the
// tree takes about three fifths of an iteration, most of it 16-byte gathers at
// four cycles a warp, and the rest is the latency of N1 to N3 with 16 warps.
// With the value space in global memory it is the L1 data pipe and the program
// stream from L2.  Staging rows, 16-byte basic moments and neighbours on lanes
// in the force phase, one launch, before -> after: level 24 mixed 512 x 4,
// 55,296 atoms 4.74 -> 4.15 ms; level 20 mixed 256 x 4, 16,000 atoms 0.553 ->
// 0.450; level 16 mixed 128 x 4, 27,648 atoms 0.435 -> 0.356, FP64 128 x 2 0.672
// -> 0.565; level 24 FP64 512 x 2, 16,384 atoms 2.41 -> 2.32.
//
// One block's rows of a staging task (atom, slot), as they lie in memory.
struct RowSlot {
  double x, y, z;
  int jt, it, cnt;
};

// Contraction tree of one block iteration: forward passes, the warps' parts of
// the site energies (jax_backend.py:101-106), reverse passes.  Ends with a
// barrier.
template <typename T, int A, int LANES>
__device__ __forceinline__ void run_tree(const DevModel& md, T* V, double* sRed, int my_wsteps, int tid) {
  const uint2* ent = md.entries + tid;
  // energy terms of this thread, requested before the last forward pass
  double th[2] = {0.0, 0.0};
  int at[2] = {0, 0};
  auto request = [&]() {
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (tid + k * LANES < md.Sa) {
        th[k] = __ldg(md.theta + tid + k * LANES);
        at[k] = __ldg(md.mapping + tid + k * LANES);
      }
  };
  if (md.nfwd == 0) request();
  __syncthreads();   // basic moments and adjoint seeds are in place
  for (int ps = 0; ps < md.nfwd; ++ps) {
    if (ps == md.nfwd - 1) request();
    run_pass<T, A, LANES, kPrefetch>(ent + md.fwd[ps].offset, __shfl_sync(0xFFFFFFFFu, my_wsteps, ps), V, V);
    __syncthreads();
  }
  // energy: E_i = xi[t_i] + sum_alpha theta_alpha m[map_alpha] in FP64: warp
  // sums now, the block sum after the reverse passes' barriers (no barrier of
  // its own on the critical path)
  {
    double ep[A];
#pragma unroll
    for (int a = 0; a < A; ++a) ep[a] = 0.0;
    auto add = [&](double t, int k) {
      const Pack<T, A> m = *reinterpret_cast<const Pack<T, A>*>(V + (md.v_m + k) * A);
#pragma unroll
      for (int a = 0; a < A; ++a) ep[a] = fma(t, static_cast<double>(m.v[a]), ep[a]);
    };
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (tid + k * LANES < md.Sa) add(th[k], at[k]);
    for (int al = tid + 2 * LANES; al < md.Sa; al += LANES) add(__ldg(md.theta + al), __ldg(md.mapping + al));
    warp_partials<A>(ep, sRed);
  }
  for (int ps = 0; ps < md.nrev; ++ps) {
    run_pass<T, A, LANES, kPrefetch>(ent + md.rev[ps].offset, __shfl_sync(0xFFFFFFFFu, my_wsteps, md.nfwd + ps), V,
                                     V);
    __syncthreads();
  }
  if (md.nrev == 0) __syncthreads();
}

template <typename T, bool kVGlobal, int A>
__global__ void __launch_bounds__(512) k_mtp_eval(DevModel md, DevIO io) {
  extern __shared__ __align__(32) unsigned char smem[];
  const int NT = blockDim.x;
  const int tid = threadIdx.x;
  // this warp's step count of pass p (forward passes, then reverse ones) is
  // held by lane p and shuffled out at the pass: no load before a pass
  const int my_wsteps = warp_steps_of_lane(md, tid, NT);
  const SmemLayout L = smem_layout<T>(kVGlobal ? 0 : md.v_size, md.M, md.S, md.R, md.K, md.D, md.P, md.n_list, md.n3_len,
                                      io.n_pad, io.qs, NT, A);
  T* V = kVGlobal ? reinterpret_cast<T*>(io.vscratch) + static_cast<size_t>(blockIdx.x) * md.v_size * A
                  : reinterpret_cast<T*>(smem + L.v);
  T* sRad = reinterpret_cast<T*>(smem + L.rad);
  T* sSt = reinterpret_cast<T*>(smem + L.st);
  double* sRed = reinterpret_cast<double*>(smem + L.red);
  int* sCnt = reinterpret_cast<int*>(smem + L.cnt);
  int* sType = sCnt + (NT >> 5);
  const int n_pad = io.n_pad, qs = L.qs;
  constexpr int VW = kVec<T>;

  const int S = md.S, R = md.R, K = md.K, P = md.P, D1 = power_rows(md.D);
  // per-block constants; radial coefficients as [pair][n][mu], rows padded to whole 16-byte words
  for (int x = tid; x < S * S * K * L.rp; x += NT) {
    const int mu = x % L.rp, n = x / L.rp % K, st = x / (L.rp * K);
    sRad[x] = mu < R ? static_cast<T>(md.radial[(st * R + mu) * K + n]) : T(0);
  }
  for (int a = tid; a < A; a += NT) {
    V[md.v_zero * A + a] = T(0);
    V[md.v_one * A + a] = T(1);
  }
  int* sMono = reinterpret_cast<int*>(smem + L.mono);
  uint16_t* sList = reinterpret_cast<uint16_t*>(sMono + P);
  for (int x = tid; x < P; x += NT) sMono[x] = md.mono_word[x];
  for (int x = tid; x < md.n_list; x += NT) sList[x] = static_cast<uint16_t>(md.mono_list[x]);
  const T rmax = static_cast<T>(md.rmax);
  const T inv_range = static_cast<T>(1.0 / (md.rmax - md.rmin));
  const T rsum = static_cast<T>(md.rmin + md.rmax);
  const T scal = static_cast<T>(md.scaling);

  // staging tasks (atom, slot) with each atom's slots padded to whole warps,
  // so a warp's ballot covers one atom.  When the block has twice as many
  // threads as tasks, every task has two threads (role 0: tid < NV, role 1:
  // the thread NV above it): both load and test the slot (the same ballot),
  // role 0 stores 1/d and the radial functions, role 1 the powers
  const int S32 = (io.nbr_stride + 31) & ~31;
  const int NV = A * S32;
  const bool split = 2 * NV <= NT;
  const int span = split ? NV : NT;   // tasks per sweep
  const int role = split ? (tid < NV ? 0 : tid < 2 * NV ? 1 : 2) : 0;
  auto load_slot = [&](int at, int v0) {
    RowSlot r{0.0, 0.0, 0.0, -1, 0, 0};
    const int v = v0 + (split ? tid - role * NV : tid);
    const int a = (role < 2 && v < NV) ? v / S32 : A;
    const int s = v - a * S32, atom = at + a;
    if (a < A && atom < io.natoms) {
      r.it = __ldg(io.itypes + atom);
      r.cnt = io.counts ? __ldg(io.counts + atom) : io.nbr_stride;
      if (s < io.nbr_stride) {
        const size_t x = static_cast<size_t>(atom) * io.nbr_stride + s;
        r.jt = __ldg(io.jtypes + x);
        r.x = __ldg(io.rijs + 3 * x);
        r.y = __ldg(io.rijs + 3 * x + 1);
        r.z = __ldg(io.rijs + 3 * x + 2);
      }
    }
    return r;
  };
  __syncthreads();

  // the first sweep's rows of the next atoms are loaded before the force
  // phase of the current ones
  RowSlot ahead = load_slot(blockIdx.x * A, 0);
  for (int base = blockIdx.x * A; base < io.natoms; base += gridDim.x * A) {
    // ask L2 for the rows of this block's next atoms now, so their staging
    // loads find them there instead of in DRAM (a hint; nothing waits on it)
    {
      const int next = base + gridDim.x * A;
      if (next < io.natoms) {
        const int na = min(A, io.natoms - next);
        const char* r0 = reinterpret_cast<const char*>(io.rijs + static_cast<size_t>(next) * io.nbr_stride * 3);
        const char* t0 = reinterpret_cast<const char*>(io.jtypes + static_cast<size_t>(next) * io.nbr_stride);
        const int rl = (na * io.nbr_stride * 24 + 127) >> 7, tl = (na * io.nbr_stride * 4 + 127) >> 7;
        for (int x = tid; x < rl + tl; x += NT) {
          const char* a = x < rl ? r0 + 128 * static_cast<size_t>(x) : t0 + 128 * static_cast<size_t>(x - rl);
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
        }
      }
    }
    // moments that are read but never written (the force phase of the
    // previous atom may have reused their slots), adjoints that no pass stores
    // and the adjoint seeds
    for (int x = tid; x < md.nzero * A; x += NT) V[(md.v_m + md.zero_list[x / A]) * A + x % A] = T(0);
    for (int x = tid; x < md.ndm_zero * A; x += NT) V[(md.v_dm + md.dm_zero[x / A]) * A + x % A] = T(0);
    // (requested here, stored after the staging, which hides their latency)
    int seed_at[2];
    double seed_v[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int x = tid + k * NT;
      seed_at[k] = x < md.nseed ? __ldg(md.seed_idx + x) : -1;
      seed_v[k] = x < md.nseed ? __ldg(md.seed_val + x) : 0.0;
    }
    auto put_seed = [&](int at, double v) {
      Pack<T, A> p;
#pragma unroll
      for (int a = 0; a < A; ++a) p.v[a] = static_cast<T>(v);
      *reinterpret_cast<Pack<T, A>*>(V + (md.v_dm + at) * A) = p;
    };
    int nv_a[A];
#pragma unroll
    for (int a = 0; a < A; ++a) nv_a[a] = 0;
    // ---- N1: staging of every atom of the block ---------------------------
    for (int v0 = 0; v0 < NV; v0 += span) {
      const RowSlot row = v0 == 0 ? ahead : load_slot(base, v0);
      const int v = v0 + (split ? tid - role * NV : tid);
      const int a = (role < 2 && v < NV) ? v / S32 : A;
      const int s = v - a * S32, atom = base + a;
      const bool real = a < A && atom < io.natoms;
      int it = row.it, cnt = row.cnt;
      if (real && (it < 0 || it >= S)) {
        if (s == 0) atomicOr(io.err, kErrSpecies);
        it = 0;
      }
      if (real && (cnt > n_pad || cnt < 0)) {
        if (s == 0) atomicOr(io.err, kErrCapacity);
        cnt = cnt < 0 ? 0 : n_pad;
      }
      if (a < A && s == 0) sType[a] = it;
      bool valid = false;
      T rx = T(0), ry = T(0), rz = T(0), d = T(0);
      int jt = -1;
      if (real && s < io.nbr_stride) {
        if (s < cnt) {
          jt = row.jt;
          rx = static_cast<T>(row.x);
          ry = static_cast<T>(row.y);
          rz = static_cast<T>(row.z);
          if (jt >= S) {
            atomicOr(io.err, kErrSpecies);
            jt = -1;
          }
          const T r2 = rx * rx + ry * ry + rz * rz;
          d = dev_sqrt(r2);
          valid = (jt >= 0) && (r2 > T(0)) && (d < rmax);
        }
        if (!valid && role == 0) {
          double* grow = io.pair_grad + (static_cast<size_t>(atom) * io.nbr_stride + s) * 3;
          grow[0] = 0.0;
          grow[1] = 0.0;
          grow[2] = 0.0;
        }
      }
      const unsigned bal = __ballot_sync(0xffffffffu, valid);
      const int w = tid >> 5, l = tid & 31;
      const int wt = w - role * (NV >> 5);   // the role-0 warp of these tasks
      if (l == 0 && role == 0) sCnt[w] = __popc(bal);
      __syncthreads();
      // lane l looks at the count of warp l: sums over the warps of an atom,
      // and over those before this one
      const int nws = span >> 5;   // at most 16
      const int wa = l < nws ? (v0 + 32 * l) / S32 : A;
      const int wc = l < nws ? sCnt[l] : 0;
      const int before = __reduce_add_sync(0xffffffffu, wa == a && l < wt ? wc : 0);
      int nv = 0;
#pragma unroll
      for (int aa = 0; aa < A; ++aa)
        if (aa == a) nv = nv_a[aa];
#pragma unroll
      for (int aa = 0; aa < A; ++aa) nv_a[aa] += __reduce_add_sync(0xffffffffu, wa == aa ? wc : 0);
      if (valid) {
        const int q = nv + before + __popc(bal & ((1u << l) - 1u));
        T* st = sSt + static_cast<size_t>(a) * L.rows * qs + q;
        const T inv_d = T(1) / d;
        if (role == 0) {
          st[2 * R * qs] = inv_d;
          reinterpret_cast<int*>(smem + L.slot)[a * n_pad + q] = s;
          // Chebyshev T_n(x) and dT_n/dx by their recurrences, folded into
          // sum_n c[t_i, t_j, mu, n] T_n for every mu as the terms appear
          const T x = (T(2) * d - rsum) * inv_range;
          const T dxdd = T(2) * inv_range;
          struct __align__(16) Word { T v[VW]; };
          const Word* c = reinterpret_cast<const Word*>(sRad + (static_cast<size_t>(it) * S + jt) * K * L.rp);
          const int nw = L.rp / VW;
          T bas[kMaxR], dbas[kMaxR];
#pragma unroll
          for (int mu = 0; mu < kMaxR; ++mu) bas[mu] = dbas[mu] = T(0);
          T t_prev = T(0), t_cur = T(1), dt_prev = T(0), dt_cur = T(0);   // T_0 = 1, T_0' = 0
          for (int n = 0; n < K; ++n) {
#pragma unroll
            for (int i = 0; i < kMaxR / VW; ++i) {
              if (i < nw) {
                const Word cw = c[n * nw + i];
#pragma unroll
                for (int k = 0; k < VW; ++k) {
                  bas[i * VW + k] = dev_fma(cw.v[k], t_cur, bas[i * VW + k]);
                  dbas[i * VW + k] = dev_fma(cw.v[k], dt_cur, dbas[i * VW + k]);
                }
              }
            }
            const T t_next = n == 0 ? x : T(2) * x * t_cur - t_prev;
            const T dt_next = n == 0 ? T(1) : T(2) * t_cur + T(2) * x * dt_cur - dt_prev;
            t_prev = t_cur;
            t_cur = t_next;
            dt_prev = dt_cur;
            dt_cur = dt_next;
          }
          const T gap = rmax - d;
          const T smooth = gap * gap;
#pragma unroll
          for (int mu = 0; mu < kMaxR; ++mu) {
            if (mu < R) {
              st[mu * qs] = scal * smooth * bas[mu];
              st[(R + mu) * qs] = scal * (T(-2) * gap * bas[mu] + smooth * dbas[mu] * dxdd);
            }
          }
        }
        if (role == 1 || !split) {
          const T ux = rx * inv_d, uy = ry * inv_d, uz = rz * inv_d;
          T* pw = st + (2 * R + 1) * qs;
          T px = T(1), py = T(1), pz = T(1);
          for (int e = 0; e < D1; ++e) {
            pw[e * qs] = px;
            pw[(D1 + e) * qs] = py;
            pw[(2 * D1 + e) * qs] = pz;
            px *= ux;
            py *= uy;
            pz *= uz;
          }
        }
      }
      if (v0 + span < NV) __syncthreads();   // the next sweep overwrites the counts
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (seed_at[k] >= 0) put_seed(seed_at[k], seed_v[k]);
    for (int x = tid + 2 * NT; x < md.nseed; x += NT) put_seed(__ldg(md.seed_idx + x), __ldg(md.seed_val + x));
    // rows end at a whole 16-byte word: the slots past the last neighbour
    // count nothing (f = 0, finite powers)
    for (int x = tid; x < A * L.rows * VW; x += NT) {
      const int k = x % VW, a = x / (L.rows * VW), r = x / VW % L.rows;
      int nv = 0;
#pragma unroll
      for (int aa = 0; aa < A; ++aa)
        if (aa == a) nv = nv_a[aa];
      if (k >= nv % VW && nv % VW) sSt[(static_cast<size_t>(a) * L.rows + r) * qs + nv / VW * VW + k] = T(0);
    }
    __syncthreads();
    // ---- N2: basic moments m[(mu, a, b, c)] of every atom of the block ------
    // tasks (atom, monomial), most radial functions first: monomials are
    // sorted by degree (descending), so monomial P-1-j has the j-th most.  A
    // warp takes 32 consecutive monomials of one atom (one radial-function
    // count and one neighbour list per warp; the warp's largest count is
    // used), warp slots go round-robin over the atoms, and the rounds after
    // the first run the slots in reverse, so each warp's rounds add up to
    // about the same cost and the last, partial round goes to the warps that
    // have the least.
    const int P32 = (P + 31) & ~31;
    for (int t0 = 0; t0 < A * P32; t0 += NT) {
      const int pos = t0 + (t0 ? NT - 1 - tid : tid);
      const int blk = pos >> 5, j = (blk / A) * 32 + (pos & 31);
      const bool act = pos < A * P32 && j < P;
      const int a = act ? blk % A : 0, p = act ? P - 1 - j : 0;
      const int word = sMono[p];   // exponents, radial functions, first entry of sList
      int nv = 0;
#pragma unroll
      for (int aa = 0; aa < A; ++aa)
        if (act && aa == a) nv = nv_a[aa];
      const int nm = __reduce_max_sync(0xffffffffu, act ? word >> 12 & 15 : 0);
      const T* f = sSt + static_cast<size_t>(a) * L.rows * qs;
      const T* px = f + (2 * R + 1 + (word & 15)) * qs;
      const T* py = f + (2 * R + 1 + D1 + (word >> 4 & 15)) * qs;
      const T* pz = f + (2 * R + 1 + 2 * D1 + (word >> 8 & 15)) * qs;
      T acc[kMaxR];
#pragma unroll
      for (int mu = 0; mu < kMaxR; ++mu) acc[mu] = T(0);
      switch (nm) {
        case 0: break;
#define MTP_MOMENTS(NM) \
  case NM: moment_task<NM>(f, qs, px, py, pz, nv, acc); break;
        MTP_MOMENTS(1) MTP_MOMENTS(2) MTP_MOMENTS(3) MTP_MOMENTS(4) MTP_MOMENTS(5) MTP_MOMENTS(6) MTP_MOMENTS(7)
        default: moment_task<8>(f, qs, px, py, pz, nv, acc); break;
#undef MTP_MOMENTS
      }
      if (act) {
        const uint16_t* k = sList + (static_cast<unsigned>(word) >> 16);
#pragma unroll
        for (int mu = 0; mu < kMaxR; ++mu)
          if (mu < (word >> 12 & 15) && k[mu] != 0xFFFFu) V[(md.v_m + k[mu]) * A + a] = acc[mu];
      }
    }

    // ---- T, R: contraction passes and their reverse -----------------------
    if (NT == 512) run_tree<T, A, 512>(md, V, sRed, my_wsteps, tid);
    else if (NT == 256) run_tree<T, A, 256>(md, V, sRed, my_wsteps, tid);
    else run_tree<T, A, 128>(md, V, sRed, my_wsteps, tid);

    // site energies: thread a adds atom a's warp sums in warp order
    if (tid < A && base + tid < io.natoms) {
      double ep = 0.0;
      for (int i = 0; i < (NT >> 5); ++i) ep += sRed[tid * (NT >> 5) + i];
      const double e = __ldg(md.species + sType[tid]) + ep;
      io.site_energy[base + tid] = e;
      if (!isfinite(e)) atomicOr(io.err, kErrNonFinite);
    }

    // ---- N3: dE_i/dr_ij per kept neighbour -------------------------------
    // adjoints of the basic moments, each atom's in chain order
    for (int x = tid; x < md.n3_len; x += NT) {
      const int k = md.chain_mode >= 0 ? x : __ldg(md.n3_src + x);   // structured: placed in chain order
      Pack<T, A> p;
      if (k >= 0) {
        p = *reinterpret_cast<const Pack<T, A>*>(V + (md.v_dm + k) * A);
      } else {
#pragma unroll
        for (int a = 0; a < A; ++a) p.v[a] = T(0);
      }
      typename Force<T>::P* o = reinterpret_cast<typename Force<T>::P*>(smem + L.dmc) + x;
#pragma unroll
      for (int a = 0; a < A; ++a) o[a * L.n3s] = Force<T>::make(p.v[a], p.v[a]);
    }
    ahead = load_slot(base + gridDim.x * A, 0);
    __syncthreads();
#define MTP_FORCES(RR, MODE) \
  case RR: force_phase<T, A, RR, MODE>(md, io, L, smem, nv_a, base, tid, NT); break;
    if (md.chain_mode == 0) {
      switch (R) {
        MTP_FORCES(1, 0) MTP_FORCES(2, 0) MTP_FORCES(3, 0) MTP_FORCES(4, 0)
        MTP_FORCES(5, 0) MTP_FORCES(6, 0) MTP_FORCES(7, 0) MTP_FORCES(8, 0)
        default: break;
      }
    } else if (md.chain_mode == 1) {
      force_phase<T, A, 6, 1>(md, io, L, smem, nv_a, base, tid, NT);
    } else if (md.chain_mode == 2) {
      force_phase<T, A, 6, 2>(md, io, L, smem, nv_a, base, tid, NT);
    } else {
      switch (R) {
        MTP_FORCES(1, -1) MTP_FORCES(2, -1) MTP_FORCES(3, -1) MTP_FORCES(4, -1)
        MTP_FORCES(5, -1) MTP_FORCES(6, -1) MTP_FORCES(7, -1) MTP_FORCES(8, -1)
        default: break;
      }
    }
#undef MTP_FORCES
    __syncthreads();
  }
}

}  // namespace mtp
