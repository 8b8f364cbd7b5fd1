// mtp_train.cu - dual-number adjoint kernel for the coefficient gradient.
#include <algorithm>

#include "mtp_train.hpp"

namespace mtp {

// Warps that share one chunk of neighbours in the last phase (one, with no
// exchange, for long rows: their staging needs the room).
__host__ __device__ inline int train_group_warps(int NW, int n_pad) {
  return n_pad > 192 ? 1 : n3_group_warps(NW, 1, n_pad, 1);
}

// Shared-memory carve of the adjoint block (one atom).  Staging is rows over the
// kept neighbours, as in the evaluation kernel: f_mu, f'_mu, phi_n, phi'_n, the
// powers of u_x, u_y, u_z and the tangents of u and d; the radial sensitivities
// of the last phase take the rows of f and f', which are dead by then.  The
// exchange of that phase's partial sums takes the moment half of a value space
// in shared memory (dead as well) where it fits there, and its adjoints are
// read in place there (structured bases); otherwise they have their own
// regions.
struct TrainSmem {
  int qs, rows;
  int f, fp, phi, phip, pw, du, A, B;   // first row of each field (du: du_x, du_y, du_z, dd)
  size_t v, rad, st, jt, mono, chain, part, gxi, grad, cnt, total;
};

__host__ __device__ inline TrainSmem train_layout(const DevModel& md, bool vglobal, int n_pad, int qs, int threads) {
  const int S = md.S, R = md.R, K = md.K, D = md.D;
  TrainSmem L;
  L.qs = qs;
  L.f = 0;
  L.fp = R;
  L.phi = 2 * R;
  L.phip = 2 * R + K;
  L.pw = 2 * R + 2 * K;
  L.du = L.pw + 3 * (D + 1);
  L.rows = L.du + 4;
  L.A = L.f;
  L.B = L.fp;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    size_t at = (o + 15) & ~size_t(15);
    o = at + bytes;
    return at;
  };
  L.v = take(vglobal ? 0 : sizeof(double) * 2 * md.v_size);
  L.rad = take(sizeof(double) * S * S * R * K);
  L.st = take(sizeof(double) * L.rows * L.qs);
  L.jt = take(sizeof(int) * L.qs);
  L.mono = take(sizeof(int) * md.P + sizeof(uint16_t) * md.n_list);
  L.chain = !vglobal && md.chain_mode >= 0 ? L.v + sizeof(double) * 2 * md.v_dm : take(2 * sizeof(double) * md.n3_len);
  const size_t part = train_group_warps(threads / 32, n_pad) > 1 ? sizeof(double) * 2 * threads : 0;
  L.part = !vglobal && part <= sizeof(double) * 2 * md.M ? L.v : take(part);
  L.gxi = take(sizeof(double) * S);
  L.grad = take(sizeof(double) * S * S * R * K);
  L.cnt = take(sizeof(int) * (threads / 32 + 1));
  L.total = (o + 15) & ~size_t(15);
  return L;
}

// Forward pass on duals: (m3, dm3) += c * (m1 m2, dm1 m2 + m1 dm2).
// Operands are read through Vr and flushes go through V: a pass never reads
// a slot that it writes, so the two views do not alias (which lets the loads
// of later entries move ahead of earlier flushes).
// A value and its tangent sit side by side, so one 16-byte access serves both.
struct DualOperands {
  double2 a, b;
};

struct DualFwdBody {
  using Operands = DualOperands;
  double2* __restrict__ V;
  const double2* __restrict__ Vr;
  double acc, tac;
  __device__ __forceinline__ Operands load(const uint2 e) const { return {Vr[e.x & 0xFFFFu], Vr[e.x >> 16]}; }
  __device__ __forceinline__ void apply(const uint2 e, const Operands& o) {
    const double c = entry_mult<double>(e.y);
    const auto A = o.a, B = o.b;
    acc = dev_fma(c * A.x, B.x, acc);
    tac = dev_fma(c, dev_fma(A.y, B.x, A.x * B.y), tac);
    const uint32_t op = (e.y >> kOpShift) & 3u;
    if (op) {
      const uint32_t d = e.y >> kDstShift;
      if (op == kOpStore) {
        V[d] = make_double2(acc, tac);
      } else {
        const auto o = V[d];
        V[d] = make_double2(o.x + acc, o.y + tac);
      }
      acc = 0.0;
      tac = 0.0;
    }
  }
};

// Reverse pass on duals (entries dst = adj[s], a = adj[t], b = m[o]):
//   lambda_s += c (lambda_t m_o + tau_t dm_o),  tau_s += c tau_t m_o.
struct DualRevBody {
  using Operands = DualOperands;
  double2* __restrict__ V;
  const double2* __restrict__ Vr;
  double acc, tac;
  __device__ __forceinline__ Operands load(const uint2 e) const { return {Vr[e.x & 0xFFFFu], Vr[e.x >> 16]}; }
  __device__ __forceinline__ void apply(const uint2 e, const Operands& o) {
    const double c = entry_mult<double>(e.y);
    const auto A = o.a, B = o.b;   // (lambda_t, tau_t), (m_o, dm_o)
    acc = dev_fma(c, dev_fma(A.x, B.x, A.y * B.y), acc);
    tac = dev_fma(c * A.y, B.x, tac);
    const uint32_t op = (e.y >> kOpShift) & 3u;
    if (op) {
      const uint32_t d = e.y >> kDstShift;
      if (op == kOpStore) {
        V[d] = make_double2(acc, tac);
      } else {
        const auto o = V[d];
        V[d] = make_double2(o.x + acc, o.y + tac);
      }
      acc = 0.0;
      tac = 0.0;
    }
  }
};

// Basic moments and their tangents of one monomial for NM radial functions,
// kVec neighbours per 16-byte load (rows are padded to that with f = f' = 0).
template <int NM>
__device__ __forceinline__ void dual_moments(const double* __restrict__ f, const double* __restrict__ fp, int qs,
                                             const double* __restrict__ px, const double* __restrict__ py,
                                             const double* __restrict__ pz, int ea, int eb, int ec,
                                             const double* __restrict__ du, int nv, double (&acc)[kMaxR],
                                             double (&tac)[kMaxR]) {
  const double am = ea, bm = eb, cm = ec;
  const double *px1 = px - (ea > 0 ? qs : 0), *py1 = py - (eb > 0 ? qs : 0), *pz1 = pz - (ec > 0 ? qs : 0);
  auto two = [](const double* p) { return *reinterpret_cast<const double2*>(p); };
  for (int q = 0; q < nv; q += 2) {
    const double2 x = two(px + q), y = two(py + q), z = two(pz + q), x1 = two(px1 + q), y1 = two(py1 + q),
                  z1 = two(pz1 + q);
    const double2 dx = two(du + q), dy = two(du + qs + q), dz = two(du + 2 * qs + q), dd = two(du + 3 * qs + q);
    const double xy0 = x.x * y.x, xy1 = x.y * y.y, m0 = xy0 * z.x, m1 = xy1 * z.y;
    const double dm0 = fma(am * x1.x * dx.x, y.x * z.x, fma(bm * y1.x * dy.x, x.x * z.x, cm * z1.x * dz.x * xy0));
    const double dm1 = fma(am * x1.y * dx.y, y.y * z.y, fma(bm * y1.y * dy.y, x.y * z.y, cm * z1.y * dz.y * xy1));
    const double e0 = dd.x * m0, e1 = dd.y * m1;
#pragma unroll
    for (int mu = 0; mu < NM; ++mu) {
      const double2 g = two(f + mu * qs + q), gp = two(fp + mu * qs + q);
      acc[mu] = fma(g.x, m0, acc[mu]);
      tac[mu] = fma(gp.x, e0, fma(g.x, dm0, tac[mu]));
      acc[mu] = fma(g.y, m1, acc[mu]);
      tac[mu] = fma(gp.y, e1, fma(g.y, dm1, tac[mu]));
    }
  }
}

// Radial sensitivities of the kept neighbours: with (lambda, tau) the dual
// adjoints of the basic moments, GA_mu = sum_s lambda u^s + tau d(u^s) and
// GB_mu = sum_s tau u^s over the monomials s of mu.  Lanes are neighbours and
// the warps of a group split the monomial chains, as in the evaluation
// kernel's force phase; a step reads its radial functions' (lambda, tau) one
// after the other from the chain-ordered copy, 16 bytes each, the same for all
// lanes.  (One thread per neighbour and share of the monomials, with the
// tables and moment positions read from L2, took 30,000 of 76,000 cycles an
// atom at level 20.)
template <int R, int MODE>
__device__ __forceinline__ void sensitivities(const DevModel& md, const TrainSmem& L, unsigned char* smem, int nv,
                                              int n_pad, int tid, int NT) {
  const int w = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, NW = NT >> 5;   // known to be warp-uniform
  const int GW = train_group_warps(NW, n_pad), g = w / GW, wg = w - g * GW, NG = NW / GW;
  const int lg = 31 - __clz(GW);
  const int i0 = md.n3_off[GW - 1 + lg + wg], i1 = md.n3_off[GW + lg + wg];
  const int D1 = md.D + 1, qs = L.qs;
  double* part = reinterpret_cast<double*>(smem + L.part);
  for (int r0 = 0; r0 < nv; r0 += 32 * NG) {
    const int j = r0 + 32 * g + lane;
    const bool act = j < nv;
    double* st = reinterpret_cast<double*>(smem + L.st) + (act ? j : r0);
    const double *px = st + L.pw * qs, *py = px + D1 * qs, *pz = py + D1 * qs, *du = st + L.du * qs;
    const double dux = du[0], duy = du[qs], duz = du[2 * qs];
    double GA[R], GB[R];
#pragma unroll
    for (int mu = 0; mu < R; ++mu) GA[mu] = GB[mu] = 0.0;
    const int iend = r0 + 32 * g < nv ? i1 : i0;
    for (int i = i0; i < iend; ++i) {
      const int word = md.n3_words[i];
      const int top = word & 15, ea = (word >> 4) & 15, eb = (word >> 8) & 15;
      const double2* lt = reinterpret_cast<const double2*>(smem + L.chain) + (word >> 16) * 2;
      const double xa = px[ea * qs], yb = py[eb * qs], xy = xa * yb;
      const double dxy = ea * px[max(ea - 1, 0) * qs] * dux * yb + eb * py[max(eb - 1, 0) * qs] * duy * xa;
      double cd = top;
#pragma unroll
      for (int k = 0; k <= kMaxDegree; ++k) {
        if (k > top) break;
        const double zc = pz[(top - k) * qs], zc1 = pz[max(top - k - 1, 0) * qs];
        const double m = xy * zc, dm = fma(dxy, zc, xy * (cd * zc1) * duz);
        cd -= 1.0;
#pragma unroll
        for (int mu = 0; mu < (MODE < 0 ? R : chain_nm<R, MODE < 0 ? 0 : MODE>(k)); ++mu) {
          const double2 v = *lt++;
          GA[mu] = fma(v.x, m, fma(v.y, dm, GA[mu]));
          GB[mu] = fma(v.y, m, GB[mu]);
        }
      }
    }
    if (GW > 1) {
      // one radial function at a time: with the value space in global memory,
      // shared memory taken here is L1 taken from its gathers
      double* mine = part + w * 32 + lane;
#pragma unroll
      for (int mu = 0; mu < R; ++mu) {
        mine[0] = GA[mu];
        mine[NT] = GB[mu];
        __syncthreads();
        if (wg == 0) {
          for (int x = 1; x < GW; ++x) {
            GA[mu] += mine[x * 32];
            GB[mu] += mine[NT + x * 32];
          }
        }
        __syncthreads();
      }
    }
    if (wg == 0 && act) {
      const double dd = du[3 * qs];
#pragma unroll
      for (int mu = 0; mu < R; ++mu) {
        st[(L.A + mu) * qs] = GA[mu];
        st[(L.B + mu) * qs] = dd * GB[mu];
      }
    }
  }
}

// One thread's neighbour slot of an atom and the atom's own values.
struct TrainSlot {
  double x, y, z;
  int jt, j, it, cfg, cnt;
};

// Training gradient of one atom per block iteration.  The dual trees bound it: 16
// bytes per operand through the L1 data pipe, from shared memory (level 20) or
// from the block's slice of global memory (level 28).  Adjoint and reduction,
// FP64, with the layout of the evaluation's phases: level 20, 4,968 atoms 0.77
// -> 0.51 ms; level 28, 18,515 atoms 35.8 -> 31.0 ms.
template <bool kVGlobal>
__global__ void __launch_bounds__(512) k_mtp_adjoint(DevModel md, TrainIO io, int n_pad, void* vscratch,
                                                     double* partials) {
  extern __shared__ __align__(32) unsigned char smem[];
  const int NT = blockDim.x, tid = threadIdx.x;
  const int my_wsteps = warp_steps_of_lane(md, tid, NT);
  const int S = md.S, R = md.R, K = md.K, P = md.P, D1 = md.D + 1;
  const TrainSmem L = train_layout(md, kVGlobal, n_pad, io.qs, NT);
  // program entries in flight per thread; with the value space in global
  // memory their operand gathers are issued before any of their flushes
  // (level 28, 32 configurations: 26.1 ms with two entries in flight and
  // gathers at use -> 19.0 ms)
  constexpr int kStreamDepth = kPrefetch;
  double2* V = kVGlobal ? reinterpret_cast<double2*>(vscratch) + static_cast<size_t>(blockIdx.x) * md.v_size
                        : reinterpret_cast<double2*>(smem + L.v);
  double* sRad = reinterpret_cast<double*>(smem + L.rad);
  double* sSt = reinterpret_cast<double*>(smem + L.st);
  int* sJt = reinterpret_cast<int*>(smem + L.jt);
  int* sMono = reinterpret_cast<int*>(smem + L.mono);
  uint16_t* sList = reinterpret_cast<uint16_t*>(sMono + P);
  double2* sChain = reinterpret_cast<double2*>(smem + L.chain);
  double* gXi = reinterpret_cast<double*>(smem + L.gxi);
  double* gRad = reinterpret_cast<double*>(smem + L.grad);
  int* sCnt = reinterpret_cast<int*>(smem + L.cnt);
  const int qs = L.qs;
  const int nrad = S * S * R * K;
  // this block's partial gradients [Sa | S | S*S*R*K]; the moment part is
  // accumulated here directly (each thread owns the same coefficients for
  // every atom), species and radial parts in shared memory
  double* out = partials + static_cast<size_t>(blockIdx.x) * (md.Sa + S + nrad);

  for (int x = tid; x < nrad; x += NT) {
    sRad[x] = md.radial[x];
    gRad[x] = 0.0;
  }
  for (int x = tid; x < P; x += NT) sMono[x] = md.mono_word[x];
  for (int x = tid; x < md.n_list; x += NT) sList[x] = static_cast<uint16_t>(md.mono_list[x]);
  for (int x = tid; x < md.Sa; x += NT) out[x] = 0.0;
  for (int x = tid; x < S; x += NT) gXi[x] = 0.0;
  for (int x = tid; x < md.ndm_zero; x += NT) V[md.v_dm + md.dm_zero[x]] = make_double2(0.0, 0.0);
  if (tid == 0) {
    V[md.v_zero] = make_double2(0.0, 0.0);
    V[md.v_one] = make_double2(1.0, 0.0);
  }
  const double rmax = md.rmax;
  const double inv_range = 1.0 / (md.rmax - md.rmin);
  const double rsum = md.rmin + md.rmax;
  const double scal = md.scaling;
  auto load_slot = [&](int atom, int s) {
    TrainSlot r{0.0, 0.0, 0.0, -1, -1, 0, 0, 0};
    if (atom < io.natoms) {
      r.it = __ldg(io.itypes + atom);
      r.cfg = __ldg(io.cfg + atom);
      r.cnt = io.counts ? __ldg(io.counts + atom) : io.nbr_stride;
      if (s < io.nbr_stride) {
        const size_t x = static_cast<size_t>(atom) * io.nbr_stride + s;
        r.jt = __ldg(io.jtypes + x);
        r.j = __ldg(io.js + x);
        r.x = __ldg(io.rijs + 3 * x);
        r.y = __ldg(io.rijs + 3 * x + 1);
        r.z = __ldg(io.rijs + 3 * x + 2);
      }
    }
    return r;
  };
  __syncthreads();

  // the next atom's slots are loaded before the last phases of this one
  TrainSlot ahead = load_slot(blockIdx.x, tid);
  for (int atom = blockIdx.x; atom < io.natoms; atom += gridDim.x) {
    int it = ahead.it;
    if (it < 0 || it >= S) {
      if (tid == 0) atomicOr(io.err, kErrSpecies);
      it = 0;
    }
    int cfg = ahead.cfg;
    if (cfg < 0 || cfg >= io.nconfig) {
      if (tid == 0) atomicOr(io.err, kErrCapacity);
      cfg = 0;
    }
    const double a_i = __ldg(io.gE + cfg);
    // C maps r onto the stress-loss direction: sum_v gS_v sigma_v = sum_s (C r_s) . g_s
    const double iv = 1.0 / __ldg(io.volumes + cfg);
    const double* gs = io.gS + 6 * cfg;
    const double c00 = gs[0] * iv, c11 = gs[1] * iv, c22 = gs[2] * iv;
    const double c12 = 0.5 * gs[3] * iv, c02 = 0.5 * gs[4] * iv;
    const double c01 = 0.5 * gs[5] * iv;
    const double gfx = __ldg(io.gF + 3 * atom), gfy = __ldg(io.gF + 3 * atom + 1),
            gfz = __ldg(io.gF + 3 * atom + 2);
    int cnt = ahead.cnt;
    if (cnt > n_pad || cnt < 0) {
      if (tid == 0) atomicOr(io.err, kErrCapacity);
      cnt = cnt < 0 ? 0 : n_pad;
    }
    // (the exchange of the last phase may have used these slots)
    for (int x = tid; x < md.nzero; x += NT) V[md.v_m + md.zero_list[x]] = make_double2(0.0, 0.0);
    for (int x = tid; x < md.nseed; x += NT) {
      const double sv = md.seed_val[x];
      V[md.v_dm + md.seed_idx[x]] = make_double2(a_i * sv, sv);
    }

    // ---- N1: stage neighbours with their tangents -------------------------
    int nv = 0;
    for (int s0 = 0; s0 < io.nbr_stride; s0 += NT) {
      const int s = s0 + tid;
      const TrainSlot row = s0 == 0 ? ahead : load_slot(atom, s);
      bool valid = false;
      double rx = 0.0, ry = 0.0, rz = 0.0, d = 0.0;
      int jt = -1, j = -1;
      if (s < io.nbr_stride && s < cnt) {
        jt = row.jt;
        j = row.j;
        rx = row.x;
        ry = row.y;
        rz = row.z;
        if (jt >= S) {
          atomicOr(io.err, kErrSpecies);
          jt = -1;
        }
        const double r2 = rx * rx + ry * ry + rz * rz;
        d = dev_sqrt(r2);
        valid = (jt >= 0) && (r2 > 0.0) && (d < rmax);
      }
      const unsigned bal = __ballot_sync(0xffffffffu, valid);
      const int w = tid >> 5, l = tid & 31;
      if (l == 0) sCnt[w] = __popc(bal);
      __syncthreads();
      const int wc = l < (NT >> 5) ? sCnt[l] : 0;
      const int before = __reduce_add_sync(0xffffffffu, l < w ? wc : 0);
      const int all = __reduce_add_sync(0xffffffffu, wc);
      if (valid) {
        const int q = nv + before + __popc(bal & ((1u << l) - 1u));
        double* st = sSt + q;
        const double inv_d = 1.0 / d;
        const double ux = rx * inv_d, uy = ry * inv_d, uz = rz * inv_d;
        // direction of the neighbour vector: force part + stress part
        double drx = gfx, dry = gfy, drz = gfz;
        if (j >= 0 && j < io.natoms) {
          drx -= __ldg(io.gF + 3 * j);
          dry -= __ldg(io.gF + 3 * j + 1);
          drz -= __ldg(io.gF + 3 * j + 2);
        }
        drx += c00 * rx + c01 * ry + c02 * rz;
        dry += c01 * rx + c11 * ry + c12 * rz;
        drz += c02 * rx + c12 * ry + c22 * rz;
        const double dd = ux * drx + uy * dry + uz * drz;
        st[L.du * qs] = (drx - ux * dd) * inv_d;
        st[(L.du + 1) * qs] = (dry - uy * dd) * inv_d;
        st[(L.du + 2) * qs] = (drz - uz * dd) * inv_d;
        st[(L.du + 3) * qs] = dd;
        sJt[q] = jt;
        const double x = (2.0 * d - rsum) * inv_range;
        const double dxdd = 2.0 * inv_range;
        const double gap = rmax - d;
        const double smooth = gap * gap;
        const double* c = sRad + (static_cast<size_t>(it) * S + jt) * R * K;
        double base[kMaxR], dbase[kMaxR];
#pragma unroll
        for (int mu = 0; mu < kMaxR; ++mu) {
          base[mu] = 0.0;
          dbase[mu] = 0.0;
        }
        double t_prev = 0.0, t_cur = 1.0, dt_prev = 0.0, dt_cur = 0.0;
        for (int n = 0; n < K; ++n) {
          st[(L.phi + n) * qs] = scal * smooth * t_cur;
          st[(L.phip + n) * qs] = scal * (-2.0 * gap * t_cur + smooth * dt_cur * dxdd);
#pragma unroll
          for (int mu = 0; mu < kMaxR; ++mu) {
            if (mu < R) {
              base[mu] = dev_fma(c[mu * K + n], t_cur, base[mu]);
              dbase[mu] = dev_fma(c[mu * K + n], dt_cur, dbase[mu]);
            }
          }
          double t_next, dt_next;
          if (n == 0) {
            t_next = x;
            dt_next = 1.0;
          } else {
            t_next = 2.0 * x * t_cur - t_prev;
            dt_next = 2.0 * t_cur + 2.0 * x * dt_cur - dt_prev;
          }
          t_prev = t_cur;
          t_cur = t_next;
          dt_prev = dt_cur;
          dt_cur = dt_next;
        }
#pragma unroll
        for (int mu = 0; mu < kMaxR; ++mu) {
          if (mu < R) {
            st[(L.f + mu) * qs] = scal * smooth * base[mu];
            st[(L.fp + mu) * qs] = scal * (-2.0 * gap * base[mu] + smooth * dbase[mu] * dxdd);
          }
        }
        double* pw = st + L.pw * qs;
        double px = 1.0, py = 1.0, pz = 1.0;
        for (int e = 0; e < D1; ++e) {
          pw[e * qs] = px;
          pw[(D1 + e) * qs] = py;
          pw[(2 * D1 + e) * qs] = pz;
          px *= ux;
          py *= uy;
          pz *= uz;
        }
      }
      nv += all;
      if (s0 + NT < io.nbr_stride) __syncthreads();   // the next sweep overwrites the counts
    }
    // rows end at a whole 16-byte word: the slot past an odd count adds nothing
    // (all rows zero, the species one that no gradient matches)
    if (nv & 1) {
      for (int r = tid; r < L.rows; r += NT) sSt[r * qs + nv] = 0.0;
      if (tid == 0) sJt[nv] = -1;
    }
    __syncthreads();

    // ---- N2: basic moments and their tangents ------------------------------
    // most radial functions first, one count per warp (Schedule::mono_word)
    for (int t0 = 0; t0 < P; t0 += NT) {
      const bool act = t0 + tid < P;
      const int word = sMono[act ? P - 1 - (t0 + tid) : 0];
      const int nm = __reduce_max_sync(0xffffffffu, act ? word >> 12 & 15 : 0);
      const int ea = word & 15, eb = word >> 4 & 15, ec = word >> 8 & 15;
      const double* px = sSt + (L.pw + ea) * qs;
      const double* py = sSt + (L.pw + D1 + eb) * qs;
      const double* pz = sSt + (L.pw + 2 * D1 + ec) * qs;
      double acc[kMaxR], tac[kMaxR];
#pragma unroll
      for (int mu = 0; mu < kMaxR; ++mu) acc[mu] = tac[mu] = 0.0;
      switch (nm) {
        case 0: break;
#define MTP_DUAL(NM) \
  case NM: dual_moments<NM>(sSt + L.f * qs, sSt + L.fp * qs, qs, px, py, pz, ea, eb, ec, sSt + L.du * qs, nv, acc, tac); break;
        MTP_DUAL(1) MTP_DUAL(2) MTP_DUAL(3) MTP_DUAL(4) MTP_DUAL(5) MTP_DUAL(6) MTP_DUAL(7) MTP_DUAL(8)
#undef MTP_DUAL
        default: break;
      }
      if (act) {
        const uint16_t* k = sList + (static_cast<unsigned>(word) >> 16);
#pragma unroll
        for (int mu = 0; mu < kMaxR; ++mu)
          if (mu < (word >> 12 & 15) && k[mu] != 0xFFFFu) V[md.v_m + k[mu]] = make_double2(acc[mu], tac[mu]);
      }
    }
    __syncthreads();

    // ---- dual forward tree --------------------------------------------------
    for (int ps = 0; ps < md.nfwd; ++ps) {
      DualFwdBody body{V, V, 0.0, 0.0};
      stream_entries_n<kStreamDepth, kVGlobal>(md.entries + md.fwd[ps].offset,
                                               __shfl_sync(0xFFFFFFFFu, my_wsteps, ps), NT, tid, body);
      __syncthreads();
    }
    // four coefficients at a time, so that their loads overlap
    for (int a0 = tid; a0 < md.Sa; a0 += 4 * NT) {
      double2 v[4];
      double o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (a0 + k * NT < md.Sa) {
          v[k] = V[md.v_m + __ldg(md.mapping + a0 + k * NT)];
          o[k] = out[a0 + k * NT];
        }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (a0 + k * NT < md.Sa)
          out[a0 + k * NT] = o[k] + (a_i * v[k].x + v[k].y);
    }
    if (tid == 0) gXi[it] += a_i;

    // ---- dual reverse tree ---------------------------------------------------
    for (int ps = 0; ps < md.nrev; ++ps) {
      DualRevBody body{V, V, 0.0, 0.0};
      stream_entries_n<kStreamDepth, kVGlobal>(md.entries + md.rev[ps].offset,
                                               __shfl_sync(0xFFFFFFFFu, my_wsteps, md.nfwd + ps), NT, tid, body);
      __syncthreads();
    }

    // ---- N3: per-neighbour radial sensitivities ------------------------------
    const bool in_place = !kVGlobal && md.chain_mode >= 0;
    for (int x = tid; x < (in_place ? 0 : md.n3_len); x += NT) {
      const int k = md.chain_mode >= 0 ? x : __ldg(md.n3_src + x);   // structured: placed in chain order
      sChain[x] = k >= 0 ? V[md.v_dm + k] : make_double2(0.0, 0.0);
    }
    ahead = load_slot(atom + gridDim.x, tid);
    __syncthreads();
#define MTP_SENS(RR, MODE) \
  case RR: sensitivities<RR, MODE>(md, L, smem, nv, n_pad, tid, NT); break;
    if (md.chain_mode == 0) {
      switch (R) {
        MTP_SENS(1, 0) MTP_SENS(2, 0) MTP_SENS(3, 0) MTP_SENS(4, 0) MTP_SENS(5, 0) MTP_SENS(6, 0) MTP_SENS(7, 0)
        MTP_SENS(8, 0)
        default: break;
      }
    } else if (md.chain_mode == 1) {
      sensitivities<6, 1>(md, L, smem, nv, n_pad, tid, NT);
    } else if (md.chain_mode == 2) {
      sensitivities<6, 2>(md, L, smem, nv, n_pad, tid, NT);
    } else {
      switch (R) {
        MTP_SENS(1, -1) MTP_SENS(2, -1) MTP_SENS(3, -1) MTP_SENS(4, -1) MTP_SENS(5, -1) MTP_SENS(6, -1)
        MTP_SENS(7, -1) MTP_SENS(8, -1)
        default: break;
      }
    }
#undef MTP_SENS
    __syncthreads();
    // ---- N4: radial coefficient gradient, one thread per (species, mu, n) ----
    for (int x = tid; x < S * R * K; x += NT) {
      const int jt = x / (R * K), mu = x / K % R, n = x % K;
      const double *pa = sSt + (L.A + mu) * qs, *pb = sSt + (L.B + mu) * qs, *pf = sSt + (L.phi + n) * qs,
              *pg = sSt + (L.phip + n) * qs;
      double g = 0.0;
      for (int q = 0; q < nv; q += 2) {
        const double2 a = *reinterpret_cast<const double2*>(pa + q), b = *reinterpret_cast<const double2*>(pb + q),
                      f = *reinterpret_cast<const double2*>(pf + q), h = *reinterpret_cast<const double2*>(pg + q);
        const int2 t = *reinterpret_cast<const int2*>(sJt + q);
        if (t.x == jt) g += a.x * f.x + b.x * h.x;
        if (t.y == jt) g += a.y * f.y + b.y * h.y;
      }
      gRad[((it * S + jt) * R + mu) * K + n] += g;
    }
    __syncthreads();
  }
  // per-block partials: [Sa | S | S*S*R*K] (the moment part is already there)
  for (int x = tid; x < S; x += NT) out[md.Sa + x] = gXi[x];
  for (int x = tid; x < nrad; x += NT) out[md.Sa + S + x] = gRad[x];
}

// Sum of the blocks' partials in a fixed order: a block takes 32 gradients,
// its warp w adds the partials of blocks w, w + 8, .. and the eight sums are
// added in warp order (one thread walking all blocks' partials was a chain of
// a few hundred L2 loads).
__global__ void k_adjoint_reduce(int nblocks, int Sa, int S, int nrad, const double* __restrict__ partials,
                                 double* __restrict__ gmoment, double* __restrict__ gspecies,
                                 double* __restrict__ gradial) {
  __shared__ double sum[8][32];
  const int np = Sa + S + nrad, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int x = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (x < np)
#pragma unroll 8
    for (int b = w; b < nblocks; b += 8) s += partials[static_cast<size_t>(b) * np + x];
  sum[w][lane] = s;
  __syncthreads();
  if (w > 0 || x >= np) return;
  for (int k = 1; k < 8; ++k) s += sum[k][lane];
  if (x < Sa) gmoment[x] = s;
  else if (x < Sa + S) gspecies[x - Sa] = s;
  else gradial[x - Sa - S] = s;
}

void train_free(TrainWorkspace& w) {
  if (w.partials) cudaFree(w.partials);
  if (w.vscratch) cudaFree(w.vscratch);
  w = TrainWorkspace();
}

template <bool G>
static cudaError_t adjoint_smem_limit(size_t bytes) {
  static size_t granted = 0;
  if (bytes <= granted) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_mtp_adjoint<G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(bytes));
  if (e == cudaSuccess) granted = bytes;
  return e;
}

template <bool G>
static int adjoint_occupancy(size_t bytes, int threads) {
  if (bytes > kMaxSmemPerBlock) return 0;
  int nb = 0;
  if (adjoint_smem_limit<G>(bytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_mtp_adjoint<G>, threads, bytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return nb;
}

static TrainSmem adjoint_layout_of(const DevModel& md, bool vglobal, int n_pad, int threads) {
  const int qs = row_stride<double>(
      n_pad, threads, [&](int q) { return train_layout(md, vglobal, n_pad, q, threads).total; });
  return train_layout(md, vglobal, n_pad, qs, threads);
}

bool adjoint_fits_shared(const DevModel& md, int n_pad, int threads) {
  const TrainSmem L = adjoint_layout_of(md, false, n_pad, threads);
  return adjoint_occupancy<false>(L.total, threads) > 0;
}

cudaError_t launch_adjoint(const DevModel& md, const TrainIO& in, int threads, int sm_count, TrainWorkspace& ws,
                           double* gspecies, double* gmoment, double* gradial, cudaStream_t st, std::string& err) {
  const int n_pad = in.nbr_stride;
  const int nrad = md.S * md.S * md.R * md.K;
  const int np = md.Sa + md.S + nrad;
  bool vglobal = false;
  TrainSmem L = adjoint_layout_of(md, false, n_pad, threads);
  int bps = adjoint_occupancy<false>(L.total, threads);
  if (bps <= 0) {
    vglobal = true;
    L = adjoint_layout_of(md, true, n_pad, threads);
    bps = adjoint_occupancy<true>(L.total, threads);
  }
  if (bps <= 0) {
    err = "the adjoint block does not fit in shared memory for this basis and nbr_stride";
    return cudaSuccess;
  }
  TrainIO io = in;
  io.qs = L.qs;
  int blocks = std::max(1, std::min(io.natoms, bps * sm_count));
  if (vglobal) {
    // the blocks' global value spaces should stay resident in L2: cap their
    // total at 5/8 of it (but keep one block per SM)
    int dev = 0, l2 = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev);
    const size_t per = static_cast<size_t>(2) * md.v_size * sizeof(double);
    const int cap = static_cast<int>(std::max<size_t>(sm_count, (static_cast<size_t>(l2) * 5 / 8) / per));
    blocks = std::max(1, std::min(blocks, cap));
  }
  const size_t need_p = static_cast<size_t>(blocks) * np;
  if (need_p > ws.partials_cap) {
    if (ws.partials) cudaFree(ws.partials);
    ws.partials = nullptr;
    cudaError_t e = cudaMalloc(&ws.partials, need_p * sizeof(double));
    if (e != cudaSuccess) return e;
    ws.partials_cap = need_p;
  }
  if (vglobal) {
    const size_t need_v = static_cast<size_t>(blocks) * 2 * md.v_size * sizeof(double);
    if (need_v > ws.vscratch_cap) {
      if (ws.vscratch) cudaFree(ws.vscratch);
      ws.vscratch = nullptr;
      cudaError_t e = cudaMalloc(&ws.vscratch, need_v);
      if (e != cudaSuccess) return e;
      ws.vscratch_cap = need_v;
    }
  }
  if (io.natoms > 0) {
    if (vglobal)
      k_mtp_adjoint<true><<<blocks, threads, L.total, st>>>(md, io, n_pad, ws.vscratch, ws.partials);
    else
      k_mtp_adjoint<false><<<blocks, threads, L.total, st>>>(md, io, n_pad, ws.vscratch, ws.partials);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_adjoint_reduce<<<(np + 31) / 32, 256, 0, st>>>(blocks, md.Sa, md.S, nrad, ws.partials, gmoment, gspecies,
                                                      gradial);
  } else {
    cudaMemsetAsync(gmoment, 0, md.Sa * sizeof(double), st);
    cudaMemsetAsync(gspecies, 0, md.S * sizeof(double), st);
    cudaMemsetAsync(gradial, 0, nrad * sizeof(double), st);
  }
  return cudaGetLastError();
}

}  // namespace mtp
