// mtp_abi.cu - the C ABI (include/mtp_b200.h): handles, device buffers, calls.
//
// Replaces the reference bridge pair_style_files/zero_overhead.cpp: instead
// of refilling NumPy buffers with sentinels and calling a deserialised JAX
// executable through CPython every step (zero_overhead.cpp:61-117, 171-272),
// a handle owns device buffers sized by the pair style's capacities and
// launches the sm_100a kernels directly.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/mtp_b200.h"
#include "mtp_launch.hpp"
#include "mtp_md.hpp"
#include "mtp_model.hpp"
#include "mtp_train.hpp"

using namespace mtp;

namespace {

std::string g_create_error;

struct DeviceSchedule {
  Schedule sched;
  uint2* d_entries = nullptr;
  int* d_warp_steps = nullptr;  // [forward passes, reverse passes][lanes / 32] (Pass::wsteps)
};

// Arguments of a host-buffer call that a cached CUDA graph replays.  The graph
// holds the host and device addresses, the sizes and the launch shapes, so it
// is valid for exactly these and for one generation of the handle's device
// state (bumped whenever coefficients, launch settings or scratch change).
struct HostCallKey {
  int kind = -1;   // 0: mtp_compute, 1: mtp_compute_positions
  int natoms = -1, stride = 0, flags = 0, extra = 0;
  long long gen = -1;
  const void* p[8] = {};
  bool operator==(const HostCallKey& o) const {
    if (kind != o.kind || natoms != o.natoms || stride != o.stride || flags != o.flags || extra != o.extra ||
        gen != o.gen)
      return false;
    for (int k = 0; k < 8; ++k)
      if (p[k] != o.p[k]) return false;
    return true;
  }
};

template <typename T>
cudaError_t dalloc(T** p, size_t n) {
  *p = nullptr;
  if (n == 0) n = 1;
  return cudaMalloc(reinterpret_cast<void**>(p), n * sizeof(T));
}

}  // namespace

// One launch shape that fits, and what the choice goes by: the least of the
// expected times or, with the value space in global memory, of the expected
// one-atom rounds.  A request (mtp_set_launch) goes by a rank that does not
// depend on the number of atoms, so that an atom's rounding does not either: the
// threads asked for, or else the next fewer that fit; of several atoms per block
// the one with the most atoms in flight per SM, then the most warps.
struct Shape {
  int lanes = 0, A = 1;
  EvalFit fit;
  double cost = 0.0;
  bool vglobal = false;
};

struct mtp_handle {
  Potential pot;
  int max_atoms = 0, max_nbr = 0, debug = 0, precision = 0;
  double cutoff = 0.0;
  int device = 0, sm_count = 0;
  size_t l2_bytes = 0;
  cudaStream_t own_stream = nullptr, stream = nullptr;
  int threads = 0, blocks_per_sm = 0;   // requested launch (mtp_set_launch); 0 threads: automatic
  void* d_vscratch = nullptr;   // value spaces in global memory, allocated once (pick_launch)
  std::map<int, DeviceSchedule> scheds;
  std::map<int, DeviceSchedule> sizes;   // by lanes: schedules without programs, to size launches
  // potential tables on the device
  // coefficients: radial, species, theta and the seeds' values in one buffer,
  // sent by one copy from its page-locked image
  double *d_coef = nullptr, *h_coef = nullptr;
  double *d_radial = nullptr, *d_species = nullptr, *d_theta = nullptr, *d_seed_val = nullptr;   // parts of d_coef
  std::vector<int> seed_of;    // [Sa] seed that each mapped moment adds to
  int *d_mapping = nullptr, *d_seed_idx = nullptr;
  // tables that are the same for every schedule of the potential, and the buffer
  // that holds them (upload_tables)
  int *d_tables = nullptr, *d_zero = nullptr, *d_dm_zero = nullptr, *d_n3_src = nullptr;
  int *d_mono_word = nullptr, *d_mono_list = nullptr;
  int nseed = 0;
  // input / output / scratch buffers sized by the capacities
  int *d_itypes = nullptr, *d_js = nullptr, *d_jtypes = nullptr, *d_counts = nullptr;
  double* d_rijs = nullptr;
  double *d_G = nullptr, *d_E = nullptr, *d_F = nullptr, *d_wown = nullptr, *d_vatom = nullptr;
  int *d_in_cnt = nullptr, *d_in_ptr = nullptr, *d_in_slot = nullptr, *d_blk = nullptr;
  bool lists_sorted = true;   // false from building the incoming lists to the force gather that sorts them
  double *d_partials = nullptr, *d_tot = nullptr;
  int* d_err = nullptr;
  int* d_cfg_ptr = nullptr;
  int cfg_cap = 0;
  double* h_tot = nullptr;   // pinned [8]: totals, error flags
  int* h_err = nullptr;      // the flags' word of h_tot
  TrainWorkspace train;
  CellScratch cells;
  int apb = 0;          // requested atoms per block (0: chosen by occupancy)
  Shape last;           // the last evaluation's launch
  int last_blocks = 0;
  // how a (lanes, atoms per block, stride, precision, value-space placement)
  // fits: worked out and asked once, so later calls can be graph-captured
  std::map<long long, EvalFit> fits;
  // profiling of the evaluation kernel
  bool profiling = false;
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> prof_events;
  // host-buffer calls (mtp_compute) on large systems copy the inputs in atom
  // chunks on copy_stream while the evaluation kernel runs on earlier chunks
  cudaStream_t copy_stream = nullptr;
  // set while a host call is captured: its graph forks (run_device)
  bool fork = false;
  cudaEvent_t fork_event = nullptr, join_event = nullptr;
  std::vector<cudaEvent_t> chunk_events;
  int prof_used = 0;
  // mtp_execute_potential: page-locked staging of the per-atom rows
  // (allocated on first use, max_atoms x max_nbr)
  double *hp_rij = nullptr, *hp_F = nullptr;
  int *hp_js = nullptr, *hp_jt = nullptr, *hp_cnt = nullptr, *hp_types = nullptr;
  // mtp_compute below kPipelineMinAtoms with page-locked buffers: the call's
  // copies, kernels and read-backs become one CUDA graph, captured on the
  // second consecutive call with the same arguments and replayed while they
  // repeat (a pair style calls with the same buffers every step)
  long long gen = 0;
  HostCallKey graph_key, seen_key;
  cudaGraphExec_t graph_exec = nullptr;
  bool seen_uncapturable = false;
  long long graph_captures = 0, graph_replays = 0;
  // mtp_compute_positions: positions, species and owners of local and ghost
  // atoms [all_cap], candidate lists [neigh_cap], list lengths [max_atoms]
  double* d_xall = nullptr;
  int *d_spall = nullptr, *d_owner = nullptr, *d_neigh = nullptr, *d_numneigh = nullptr;
  size_t all_cap = 0, neigh_cap = 0;
  // statistics
  long long calls = 0;
  double total_ms = 0.0;
  std::string err;
};

namespace {

int fail(mtp_handle* h, int code, const std::string& msg) {
  if (h) h->err = msg;
  else g_create_error = msg;
  return code;
}

// A CUDA call failed: record it, and let work already queued on the handle's
// streams (copies from or to the caller's host buffers among it) finish
// before the error returns, so the caller may reuse or free those buffers.
int cuda_fail(mtp_handle* h, cudaError_t e, const char* what) {
  const int st = fail(h, MTP_E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  if (h) {
    cudaStreamSynchronize(h->stream);
    if (h->copy_stream) cudaStreamSynchronize(h->copy_stream);
    cudaGetLastError();
  }
  return st;
}

#define MTP_CUDA(h, call)                                  \
  do {                                                     \
    cudaError_t e_ = (call);                               \
    if (e_ != cudaSuccess) return cuda_fail((h), e_, #call); \
  } while (0)

DevModel make_model(mtp_handle* h, const DeviceSchedule& ds) {
  DevModel md{};
  const Schedule& s = ds.sched;
  md.entries = ds.d_entries;
  md.nfwd = static_cast<int>(s.fwd.size());
  md.nrev = static_cast<int>(s.rev.size());
  for (int i = 0; i < md.nfwd; ++i) md.fwd[i] = DevPass{s.fwd[i].offset, s.fwd[i].steps};
  for (int i = 0; i < md.nrev; ++i) md.rev[i] = DevPass{s.rev[i].offset, s.rev[i].steps};
  md.radial = h->d_radial;
  md.species = h->d_species;
  md.theta = h->d_theta;
  md.mapping = h->d_mapping;
  md.seed_idx = h->d_seed_idx;
  md.seed_val = h->d_seed_val;
  md.nseed = h->nseed;
  md.zero_list = h->d_zero;
  md.nzero = static_cast<int>(s.zero_list.size());
  md.mono_word = h->d_mono_word;
  md.mono_list = h->d_mono_list;
  md.n_list = static_cast<int>(s.mono_list.size());
  md.dm_zero = h->d_dm_zero;
  md.ndm_zero = static_cast<int>(s.dm_zero.size());
  md.chain_mode = s.chain_mode;
  md.n3_len = s.n3_len;
  md.n3_src = h->d_n3_src;
  std::copy(s.n3_words.begin(), s.n3_words.end(), md.n3_words);
  std::copy(s.n3_off.begin(), s.n3_off.end(), md.n3_off);
  md.warp_steps = ds.d_warp_steps;
  md.S = h->pot.S;
  md.R = h->pot.R;
  md.K = h->pot.K;
  md.M = h->pot.M;
  md.B = h->pot.B;
  md.P = s.P;
  md.D = s.D;
  md.Sa = h->pot.Sa;
  md.v_m = s.v_m;
  md.v_dm = s.v_dm;
  md.n_dm = s.v_part - s.v_dm;
  md.v_zero = s.v_zero;
  md.v_one = s.v_one;
  md.v_size = s.v_size;
  md.scaling = h->pot.scaling;
  md.rmin = h->pot.min_dist;
  md.rmax = h->pot.max_dist;
  return md;
}

// Bytes of one operand access of the evaluation kernel (sets the bank model
// the schedule's entry order is tuned for).
inline int access_width(bool fp64, int atoms_per_block) { return (fp64 ? 8 : 4) * atoms_per_block; }

// Schedule without programs for `lanes` threads: what a launch needs to be sized.
int get_sizes(mtp_handle* h, int lanes, const DeviceSchedule** out) {
  auto it = h->sizes.find(lanes);
  if (it == h->sizes.end()) {
    DeviceSchedule ds;
    std::string err;
    if (!build_schedule(h->pot, lanes, ds.sched, err, 4, false)) return fail(h, MTP_E_FORMAT, err);
    it = h->sizes.emplace(lanes, std::move(ds)).first;
  }
  *out = &it->second;
  return MTP_OK;
}

// The tables that are the same for every schedule of the potential, in one
// buffer: on the device as a whole or, after a failure, not at all.
int upload_tables(mtp_handle* h, const Schedule& t) {
  const std::pair<int**, const std::vector<int>*> tables[] = {
      {&h->d_zero, &t.zero_list}, {&h->d_dm_zero, &t.dm_zero}, {&h->d_n3_src, &t.n3_src},
      {&h->d_mono_word, &t.mono_word}, {&h->d_mono_list, &t.mono_list}};
  std::vector<int> all;
  std::vector<size_t> at;
  for (const auto& x : tables) {
    at.push_back(all.size());
    all.insert(all.end(), x.second->begin(), x.second->end());
    all.resize((all.size() + 63) / 64 * 64);   // each at a 256-byte boundary
  }
  int* d = nullptr;
  MTP_CUDA(h, dalloc(&d, all.size()));
  const cudaError_t e = cudaMemcpy(d, all.data(), all.size() * sizeof(int), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(d);
    return cuda_fail(h, e, "upload tables");
  }
  h->d_tables = d;
  for (size_t k = 0; k < at.size(); ++k) *tables[k].first = d + at[k];
  return MTP_OK;
}

// Schedule for `lanes` threads and `width`-byte operand accesses, built and
// uploaded on first use; refine_schedule runs where the value space can sit in
// shared memory (bank order matters only there).
int get_schedule(mtp_handle* h, int lanes, int width, const DeviceSchedule** out) {
  const int key = lanes * 64 + width;
  auto it = h->scheds.find(key);
  if (it == h->scheds.end()) {
    DeviceSchedule ds;
    std::string err;
    if (!build_schedule(h->pot, lanes, ds.sched, err, width)) return fail(h, MTP_E_FORMAT, err);
    if (static_cast<size_t>(ds.sched.v_size) * width <= kMaxSmemPerBlock) refine_schedule(ds.sched);
    if (h->d_tables == nullptr) {
      const int st = upload_tables(h, ds.sched);
      if (st != MTP_OK) return st;
    }
    const auto& ent = ds.sched.entries;
    std::vector<int> ws;
    for (const Pass& p : ds.sched.fwd) ws.insert(ws.end(), p.wsteps.begin(), p.wsteps.end());
    for (const Pass& p : ds.sched.rev) ws.insert(ws.end(), p.wsteps.begin(), p.wsteps.end());
    cudaError_t e = dalloc(&ds.d_entries, ent.size() / 2);
    if (e == cudaSuccess)
      e = cudaMemcpy(ds.d_entries, ent.data(), ent.size() * sizeof(uint32_t), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = dalloc(&ds.d_warp_steps, ws.size());
    if (e == cudaSuccess) e = cudaMemcpy(ds.d_warp_steps, ws.data(), ws.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
      cudaFree(ds.d_entries);
      cudaFree(ds.d_warp_steps);
      return cuda_fail(h, e, "upload schedule");
    }
    it = h->scheds.emplace(key, std::move(ds)).first;
  }
  *out = &it->second;
  return MTP_OK;
}

// Send the coefficients, after the work on the handle's stream, by a copy on the
// legacy default stream: it also comes after the work of blocking streams that
// the handle used before (kernels there may still read the old values).  The
// copy is waited for: later work sees the new values on any stream, graph
// replays included.
int upload_coeffs(mtp_handle* h) {
  const Potential& p = h->pot;
  double* o = h->h_coef;
  o = std::copy(p.radial.begin(), p.radial.end(), o);
  o = std::copy(p.species.begin(), p.species.end(), o);
  o = std::copy(p.moment.begin(), p.moment.end(), o);
  std::fill(o, o + h->nseed, 0.0);
  for (int a = 0; a < p.Sa; ++a) o[h->seed_of[a]] += p.moment[a];
  const size_t n = (o - h->h_coef) + h->nseed;
  MTP_CUDA(h, cudaMemcpyAsync(h->d_coef, h->h_coef, n * sizeof(double), cudaMemcpyHostToDevice, nullptr));
  MTP_CUDA(h, cudaStreamSynchronize(nullptr));
  return MTP_OK;
}

void free_handle(mtp_handle* h) {
  if (!h) return;
  auto F = [](void* p) { if (p) cudaFree(p); };
  for (auto& kv : h->scheds) {
    F(kv.second.d_entries);
    F(kv.second.d_warp_steps);
  }
  F(h->d_coef);
  if (h->h_coef) cudaFreeHost(h->h_coef);
  F(h->d_mapping); F(h->d_seed_idx); F(h->d_tables);
  F(h->d_itypes); F(h->d_js); F(h->d_jtypes); F(h->d_counts); F(h->d_rijs);
  F(h->d_G); F(h->d_E); F(h->d_F); F(h->d_wown); F(h->d_vatom);
  F(h->d_in_cnt); F(h->d_in_ptr); F(h->d_in_slot); F(h->d_blk);
  F(h->d_partials); F(h->d_tot); F(h->d_err); F(h->d_cfg_ptr); F(h->d_vscratch);
  F(h->d_xall); F(h->d_spall); F(h->d_owner); F(h->d_neigh); F(h->d_numneigh);
  train_free(h->train);
  F(h->cells.cell); F(h->cells.img); F(h->cells.cnt); F(h->cells.ptr); F(h->cells.cursor); F(h->cells.atoms);
  F(h->cells.blk);
  for (auto& ev : h->prof_events) {
    cudaEventDestroy(ev.first);
    cudaEventDestroy(ev.second);
  }
  if (h->h_tot) cudaFreeHost(h->h_tot);
  for (auto ev : h->chunk_events) cudaEventDestroy(ev);
  if (h->copy_stream) cudaStreamDestroy(h->copy_stream);
  if (h->fork_event) cudaEventDestroy(h->fork_event);
  if (h->join_event) cudaEventDestroy(h->join_event);
  if (h->graph_exec) cudaGraphExecDestroy(h->graph_exec);
  for (void* q : {static_cast<void*>(h->hp_rij), static_cast<void*>(h->hp_F), static_cast<void*>(h->hp_js),
                  static_cast<void*>(h->hp_jt), static_cast<void*>(h->hp_cnt), static_cast<void*>(h->hp_types)})
    if (q) cudaFreeHost(q);
  if (h->own_stream) cudaStreamDestroy(h->own_stream);
  delete h;
}

// How one launch shape fits, within the handle's blocks per SM.
int launch_fit(mtp_handle* h, int lanes, int stride, bool fp64, bool vglobal, int A, EvalFit* fit) {
  const long long key = (static_cast<long long>(stride) << 20) | (lanes << 4) | (A << 2) | (vglobal ? 2 : 0) | (fp64 ? 1 : 0);
  auto it = h->fits.find(key);
  if (it == h->fits.end()) {
    const DeviceSchedule* ds = nullptr;
    int st = get_sizes(h, lanes, &ds);
    if (st != MTP_OK) return st;
    it = h->fits.emplace(key, eval_fit(make_model(h, *ds), stride, lanes, fp64, vglobal, A)).first;
  }
  *fit = it->second;
  if (h->blocks_per_sm > 0) fit->per_sm = std::min(fit->per_sm, h->blocks_per_sm);
  return MTP_OK;
}

// Expected time (us) of an evaluation of natoms in rows of `slots` with `bps`
// blocks of `lanes` threads and A atoms per SM; the blocks run an iteration once
// per round.  An iteration has a latency (each lane walks T / lanes of the T
// products three times over, and its share of the slots and basic moments B),
// and the atoms on an SM take their share of its throughput (products, whose
// program entries a block's atoms share, and slots times moments).  One block's
// phases add the two up; several blocks fill each other's waits.
// The constants are fitted to all shapes of levels 16 to 28 (T = 969 to 133,000,
// B = 130 to 800) on 16 to 300 slots and 16 to 16,000 atoms: the shape taken is
// within 0.5 % of the best on average, 14 % at worst (a call of 19 us).  Without
// the slots it was within 2 % and 37 %: level 16 mixed, 4,000 atoms of 200 slots
// 226 us (128 x 4), now 165 (128 x 1); level 20 FP64, 300 atoms of 200 slots 84 us
// (512 x 2), now 71 (256 x 1); and the same within 6 % elsewhere.
double launch_estimate(const Potential& pot, bool fp64, int lanes, int A, int bps, int sms, long long natoms,
                       int slots) {
  const long long groups = (natoms + A - 1) / A;
  const long long rounds = std::max(1LL, (groups + static_cast<long long>(bps) * sms - 1) / (static_cast<long long>(bps) * sms));
  const double blocks = static_cast<double>(std::max(1LL, std::min<long long>(bps, (groups + sms - 1) / sms)));
  const double T = pot.T, B = pot.B, share = static_cast<double>(A) * slots / lanes;
  const double latency = fp64 ? 14.0 + 0.19 * T / lanes + share * (3.4 + 0.023 * B)
                              : 12.0 + 0.19 * T / lanes + share * (2.2 + 0.013 * B);
  const double work = fp64 ? blocks * A * (1.0 + 6.7e-5 * T + slots * (2.2e-3 + 8.8e-5 * B))
                           : blocks * (A * (1.4 + 2.2e-5 * T + slots * (1.7e-3 + 3.4e-5 * B)) + 3e-5 * T);
  return rounds * (latency + work - (1.0 - 1.0 / blocks) * std::min(latency, work));
}

// Value spaces in global memory, one slice of A atoms per SM, and the most atoms
// that may share a block there: two as long as the slices stay in L2.
size_t global_space_bytes(const mtp_handle* h, const DeviceSchedule& ds, int A, bool fp64) {
  return static_cast<size_t>(h->sm_count) * ds.sched.v_size * A * (fp64 ? sizeof(double) : sizeof(float));
}

int global_atoms(const mtp_handle* h, const DeviceSchedule& ds, bool fp64) {
  return eval_variant_exists(fp64, true, 2) && global_space_bytes(h, ds, 2, fp64) <= h->l2_bytes / 4 * 3 ? 2 : 1;
}

// The shapes of the handle's request that fit for natoms, with the value space
// in shared memory.
int shared_shapes(mtp_handle* h, long long natoms, int stride, bool fp64, std::vector<Shape>* out) {
  for (int lanes : {512, 256, 128}) {
    if (h->threads > 0 && lanes > h->threads) continue;
    for (int A : {4, 2, 1}) {
      if (h->apb > 0 && A != h->apb) continue;
      if (!eval_variant_exists(fp64, false, A)) continue;
      EvalFit fit;
      const int st = launch_fit(h, lanes, stride, fp64, false, A, &fit);
      if (st != MTP_OK) return st;
      const int bps = fit.per_sm;
      if (bps <= 0) continue;
      const double rank = 1e5 * (512 / lanes) - (1024 * A * bps + bps * lanes / 32);   // at most 16 atoms in flight
      out->push_back({lanes, A, fit,
                      h->threads > 0 ? rank : launch_estimate(h->pot, fp64, lanes, A, bps, h->sm_count, natoms, stride),
                      false});
    }
  }
  return MTP_OK;
}

// The same with the value space in global memory: 512 lanes give an SM 16 warps
// with one block, so the blocks' value spaces stay within L2.  In FP64 two atoms
// share every program entry (4.5 MB an iteration at level 28, as much L2 traffic
// as the operands) and fill more of each 32-byte sector a gather touches: an
// iteration takes 1.45x one atom's time on 64 slots and 1.87x on 200 (1.78 stands
// for all; 1,200 atoms of 64 slots 1.39 -> 1.11 ms), so they win where that saves
// a round, as long as the value spaces stay in L2 (four atoms' do not: 2,048
// atoms 3.47 ms, two 1.96).  FP32 gets here with rows too long for shared
// memory, whose staging leaves little L1 to the gathers: two atoms take 2.3x one
// atom's time (level 28, 148 / 296 atoms of 500 slots 180 / 402 us), so there is
// no such kernel.
int global_shapes(mtp_handle* h, long long natoms, int stride, bool fp64, std::vector<Shape>* out) {
  const DeviceSchedule* sz = nullptr;
  int st = get_sizes(h, 512, &sz);
  if (st != MTP_OK) return st;
  for (int A : {1, 2}) {
    if (h->apb > 0 && A > h->apb) continue;
    if (A > global_atoms(h, *sz, fp64)) continue;
    EvalFit fit;
    st = launch_fit(h, 512, stride, fp64, true, A, &fit);
    if (st != MTP_OK) return st;
    if (fit.per_sm <= 0) continue;
    fit.per_sm = 1;
    const long long per = static_cast<long long>(A) * h->sm_count;
    const double rounds = static_cast<double>((natoms + per - 1) / per) * (A == 1 ? 1.0 : 1.78);
    const double rank = A == (h->apb == 2 ? 2 : 1) ? 0.0 : 1.0;
    out->push_back({512, A, fit, h->threads > 0 ? rank : rounds, true});
  }
  return MTP_OK;
}

// Programs on the device for `lanes` threads: those whose entry order was tuned
// for `width`-byte operands or, with `any_order`, others (every order computes
// the same sums; the bank conflicts and the order of the terms differ).
const DeviceSchedule* programs_on_device(const mtp_handle* h, int lanes, int width, bool any_order) {
  const auto it = h->scheds.find(lanes * 64 + width);
  if (it != h->scheds.end()) return &it->second;
  if (any_order)
    for (const auto& kv : h->scheds)
      if (kv.second.sched.lanes == lanes) return &kv.second;
  return nullptr;
}

// The shape of the least cost (the first of equal ones).
const Shape& best_shape(const std::vector<Shape>& shapes) {
  return *std::min_element(shapes.begin(), shapes.end(), [](const Shape& a, const Shape& b) { return a.cost < b.cost; });
}

// The same for calls that can upload nothing: of the shapes whose programs are
// on the device or, where there are none, of those that can run with programs
// of another entry order.  Null *ds: there are none of these either.
Shape best_uploaded_shape(const mtp_handle* h, const std::vector<Shape>& shapes, bool fp64, const DeviceSchedule** ds) {
  Shape best;
  *ds = nullptr;
  for (const bool any_order : {false, true}) {
    for (const Shape& c : shapes) {
      const DeviceSchedule* p = programs_on_device(h, c.lanes, access_width(fp64, c.A), any_order);
      if (!p || (*ds && c.cost >= best.cost)) continue;
      best = c;
      *ds = p;
    }
    if (*ds) break;
  }
  return best;
}

// Launch shape for the evaluation kernel on natoms: the (lanes, atoms per
// block) of the least cost (Shape) among those whose value space fits in shared
// memory; when none fits, the value space moves to global memory.  While the stream is being captured nothing can be
// uploaded, so a shape whose programs are not on the device yet gives way to
// the best one whose are.
int pick_launch(mtp_handle* h, long long natoms, int stride, bool fp64, Shape* shape, const DeviceSchedule** ds) {
  std::vector<Shape> shapes;
  shapes.reserve(9);
  int st = shared_shapes(h, natoms, stride, fp64, &shapes);
  if (st != MTP_OK) return st;
  if (shapes.empty() && (st = global_shapes(h, natoms, stride, fp64, &shapes)) != MTP_OK) return st;
  if (shapes.empty())
    return fail(h, MTP_E_CAPACITY, "the evaluation block does not fit in shared memory for this basis and max_nbr");
  Shape best = best_shape(shapes);
  *ds = programs_on_device(h, best.lanes, access_width(fp64, best.A), false);
  if (!*ds) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(h->stream, &cs) != cudaSuccess) cudaGetLastError();
    if (cs != cudaStreamCaptureStatusNone) {
      const Shape ready = best_uploaded_shape(h, shapes, fp64, ds);
      if (*ds) best = ready;
    }
  }
  if (!*ds && (st = get_schedule(h, best.lanes, access_width(fp64, best.A), ds)) != MTP_OK) return st;
  if (best.vglobal && !h->d_vscratch) {
    // for the largest launch any call of this handle can take (one block per SM
    // with the most atoms), once: a graph that a caller captured holds the
    // address, so the buffer must not move when a later call needs more of it
    const size_t bytes = global_space_bytes(h, **ds, global_atoms(h, **ds, fp64), fp64);
    MTP_CUDA(h, cudaMalloc(&h->d_vscratch, bytes));
    ++h->gen;
  }
  *shape = best;
  return MTP_OK;
}

// Blocks of a launch on natoms: every SM full, or one group of atoms each.
int launch_blocks(const mtp_handle* h, const Shape& s, long long natoms) {
  const long long most = static_cast<long long>(s.fit.per_sm) * h->sm_count;
  return static_cast<int>(std::max(1LL, std::min(most, (natoms + s.A - 1) / s.A)));
}

// Evaluation kernel on atoms [lo, lo + n) of a system of `natoms` in device
// rows (site energies and per-slot gradients of those atoms).  The launch
// shape is that of the whole system, so the parts round as one launch would.
int eval_range(mtp_handle* h, int natoms, int lo, int n, int stride, const int* itypes, const double* rijs, const int* jtypes,
               const int* counts) {
  const bool fp64 = h->precision == MTP_PRECISION_FP64;
  const DeviceSchedule* ds = nullptr;
  const int st = pick_launch(h, natoms, stride, fp64, &h->last, &ds);
  if (st != MTP_OK) return st;
  h->last_blocks = launch_blocks(h, h->last, natoms);
  const DevModel md = make_model(h, *ds);
  const size_t rows = static_cast<size_t>(lo) * stride;
  DevIO io{};
  io.natoms = n;
  io.nbr_stride = stride;
  io.n_pad = stride;
  io.itypes = itypes + lo;
  io.rijs = rijs + 3 * rows;
  io.jtypes = jtypes + rows;
  io.counts = counts ? counts + lo : nullptr;
  io.site_energy = h->d_E + lo;
  io.pair_grad = h->d_G + 3 * rows;
  io.err = h->d_err;
  io.vscratch = h->d_vscratch;
  MTP_CUDA(h, launch_eval(md, io, h->last.fit, h->last.lanes, launch_blocks(h, h->last, n), fp64, h->last.vglobal,
                          h->last.A, h->stream));
  return MTP_OK;
}

// Profiling events around the evaluation launches of one call (mtp_profile).
int prof_begin(mtp_handle* h, cudaEvent_t* e1) {
  *e1 = nullptr;
  if (!h->profiling) return MTP_OK;
  if (h->prof_used == static_cast<int>(h->prof_events.size())) {
    cudaEvent_t a, b;
    MTP_CUDA(h, cudaEventCreate(&a));
    MTP_CUDA(h, cudaEventCreate(&b));
    h->prof_events.push_back({a, b});
  }
  const cudaEvent_t e0 = h->prof_events[h->prof_used].first;
  *e1 = h->prof_events[h->prof_used].second;
  ++h->prof_used;
  MTP_CUDA(h, cudaEventRecord(e0, h->stream));
  return MTP_OK;
}

// Evaluate site energies and per-slot gradients, then forces and virials.
// `counted`: the incoming slots were counted with the rows.  While a call is
// captured (h->fork) the incoming lists, which only the force gather needs,
// become a branch of the graph beside the evaluation.
int run_device(mtp_handle* h, int natoms, int stride, const int* itypes, const double* rijs, const int* js,
               const int* jtypes, const int* counts, bool rebuild_incoming, bool counted, double* forces,
               double* vatom) {
  const bool fork = rebuild_incoming && h->fork;
  if (rebuild_incoming) {
    const cudaStream_t s = fork ? h->copy_stream : h->stream;
    if (fork) {
      MTP_CUDA(h, cudaEventRecord(h->fork_event, h->stream));
      MTP_CUDA(h, cudaStreamWaitEvent(s, h->fork_event, 0));
    }
    h->lists_sorted = false;
    MTP_CUDA(h, launch_incoming(natoms, stride, js, jtypes, counts, h->d_in_cnt, h->d_in_ptr, h->d_in_slot,
                                h->d_blk, counted, s));
    if (fork) MTP_CUDA(h, cudaEventRecord(h->join_event, s));
  }
  cudaEvent_t e1 = nullptr;
  int st = prof_begin(h, &e1);
  if (st != MTP_OK) return st;
  st = eval_range(h, natoms, 0, natoms, stride, itypes, rijs, jtypes, counts);
  if (st != MTP_OK) return st;
  if (e1) MTP_CUDA(h, cudaEventRecord(e1, h->stream));
  if (fork) MTP_CUDA(h, cudaStreamWaitEvent(h->stream, h->join_event, 0));
  MTP_CUDA(h, launch_force_gather(natoms, stride, rijs, counts, h->d_G, h->d_in_ptr, h->d_in_slot,
                                  !h->lists_sorted, forces, h->d_wown, vatom, h->stream));
  h->lists_sorted = true;
  return MTP_OK;
}

// True where this device's kernels can store doubles at p: aligned, and memory
// of this device, managed or page-locked host memory (a peer's memory may not be
// mapped here; a copy reaches it all the same).
bool device_writable(const mtp_handle* h, const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (reinterpret_cast<uintptr_t>(p) % alignof(double) != 0 || a.devicePointer != p) return false;
  return a.type == cudaMemoryTypeDevice ? a.device == h->device : a.type != cudaMemoryTypeUnregistered;
}

// Totals into the caller's device buffers (null: not asked for), by the kernel
// itself or, where it cannot write there, by copies that report the error.
int write_totals(mtp_handle* h, int natoms, const double* site_energy, const double* wown, double* partials,
                 double* tot, double* d_energy, double* d_virial) {
  const bool e = d_energy && device_writable(h, d_energy), v = d_virial && device_writable(h, d_virial);
  MTP_CUDA(h, launch_totals(natoms, site_energy, wown, partials, tot, h->d_err, e ? d_energy : nullptr,
                            v ? d_virial : nullptr, h->stream));
  if (d_energy && !e)
    MTP_CUDA(h, cudaMemcpyAsync(d_energy, tot, sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  if (d_virial && !v)
    MTP_CUDA(h, cudaMemcpyAsync(d_virial, tot + 1, 6 * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  return MTP_OK;
}

// Systems from this size on are copied in chunks that overlap the evaluation.
constexpr int kPipelineMinAtoms = 65536;
constexpr int kPipelineChunks = 16;

// run_device for host input buffers: the inputs of chunk k go up on the copy
// stream while the evaluation kernel works on chunk k-1 (events order each
// chunk's kernel after its copies); the incoming lists and the force gather
// need every row and follow the last chunk.  With pinned host buffers the
// copies overlap the kernels; pageable ones are still correct.
int run_host_pipelined_body(mtp_handle* h, int natoms, int stride, const int* itypes, const double* rijs,
                            const int* js, const int* jtypes, const int* counts, double* vatom) {
  const cudaStream_t s = h->stream;
  if (!h->copy_stream) MTP_CUDA(h, cudaStreamCreateWithFlags(&h->copy_stream, cudaStreamNonBlocking));
  // About 8 chunks of at least 8,192 atoms, 16 on large systems: what follows
  // the last copy is one chunk's evaluation (level 16 FP64, 107,550 atoms, three
  // chunks: 4.99 ms, eight: 4.67; level 20, 91,446 atoms, two: 6.37, eight: 5.25)
  const int nch = std::max({1, std::min(kPipelineChunks / 2, natoms / 8192), std::min(kPipelineChunks, natoms / 32768)});
  while (static_cast<int>(h->chunk_events.size()) < nch + 1) {
    cudaEvent_t ev;
    MTP_CUDA(h, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    h->chunk_events.push_back(ev);
  }
  // the copies may only overwrite the device rows once earlier work on the
  // compute stream is done with them
  MTP_CUDA(h, cudaEventRecord(h->chunk_events[nch], s));
  MTP_CUDA(h, cudaStreamWaitEvent(h->copy_stream, h->chunk_events[nch], 0));
  for (int k = 0; k < nch; ++k) {
    const size_t lo = static_cast<size_t>(natoms) * k / nch, hi = static_cast<size_t>(natoms) * (k + 1) / nch;
    const size_t n = hi - lo, r0 = lo * stride, nr = n * stride;
    const cudaStream_t c = h->copy_stream;
    MTP_CUDA(h, cudaMemcpyAsync(h->d_itypes + lo, itypes + lo, n * sizeof(int), cudaMemcpyHostToDevice, c));
    MTP_CUDA(h, cudaMemcpyAsync(h->d_rijs + 3 * r0, rijs + 3 * r0, 3 * nr * sizeof(double), cudaMemcpyHostToDevice, c));
    MTP_CUDA(h, cudaMemcpyAsync(h->d_js + r0, js + r0, nr * sizeof(int), cudaMemcpyHostToDevice, c));
    MTP_CUDA(h, cudaMemcpyAsync(h->d_jtypes + r0, jtypes + r0, nr * sizeof(int), cudaMemcpyHostToDevice, c));
    if (counts) MTP_CUDA(h, cudaMemcpyAsync(h->d_counts + lo, counts + lo, n * sizeof(int), cudaMemcpyHostToDevice, c));
    MTP_CUDA(h, cudaEventRecord(h->chunk_events[k], c));
  }
  cudaEvent_t e1 = nullptr;
  for (int k = 0; k < nch; ++k) {
    const int lo = static_cast<int>(static_cast<size_t>(natoms) * k / nch);
    const int hi = static_cast<int>(static_cast<size_t>(natoms) * (k + 1) / nch);
    MTP_CUDA(h, cudaStreamWaitEvent(s, h->chunk_events[k], 0));
    if (k == 0) {
      int st = prof_begin(h, &e1);
      if (st != MTP_OK) return st;
    }
    int st = eval_range(h, natoms, lo, hi - lo, stride, h->d_itypes, h->d_rijs, h->d_jtypes, counts ? h->d_counts : nullptr);
    if (st != MTP_OK) return st;
  }
  if (e1) MTP_CUDA(h, cudaEventRecord(e1, s));
  h->lists_sorted = false;
  MTP_CUDA(h, launch_incoming(natoms, stride, h->d_js, h->d_jtypes, counts ? h->d_counts : nullptr, h->d_in_cnt,
                              h->d_in_ptr, h->d_in_slot, h->d_blk, false, s));
  MTP_CUDA(h, launch_force_gather(natoms, stride, h->d_rijs, counts ? h->d_counts : nullptr, h->d_G, h->d_in_ptr,
                                  h->d_in_slot, true, h->d_F, h->d_wown, vatom, s));
  h->lists_sorted = true;
  return MTP_OK;
}

// A failure part-way leaves copies from the caller's host buffers in flight:
// they finish before the call returns, so the caller may free the buffers.
int run_host_pipelined(mtp_handle* h, int natoms, int stride, const int* itypes, const double* rijs, const int* js,
                       const int* jtypes, const int* counts, double* vatom) {
  const int st = run_host_pipelined_body(h, natoms, stride, itypes, rijs, js, jtypes, counts, vatom);
  if (st != MTP_OK && h->copy_stream) cudaStreamSynchronize(h->copy_stream);
  return st;
}

// Status from the device error flags already copied to h_err by finished work
// (the flags are cleared on the device when set).
int take_err_flags(mtp_handle* h) {
  const int f = *h->h_err;
  if (f) MTP_CUDA(h, cudaMemsetAsync(h->d_err, 0, sizeof(int), h->stream));
  if (f & kErrSpecies) return fail(h, MTP_E_SPECIES, "a species index is outside [0, species_count)");
  if (f & kErrCapacity) return fail(h, MTP_E_CAPACITY, "a neighbour count exceeds the row length");
  if (f & kErrNonFinite) return fail(h, MTP_E_NONFINITE, "non-finite energy or force produced on the device");
  return MTP_OK;
}

int read_err_flags(mtp_handle* h) {
  MTP_CUDA(h, cudaMemcpyAsync(h->h_err, h->d_err, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  MTP_CUDA(h, cudaStreamSynchronize(h->stream));
  return take_err_flags(h);
}

// True when [p, p + bytes) is page-locked host memory (cudaHostAlloc or
// cudaHostRegister): its first and last byte are checked on every call, so a
// buffer freed and replaced by pageable memory at the same address is seen.
bool host_pinned(const void* p, size_t bytes) {
  if (!p || bytes == 0) return true;
  const char* c = static_cast<const char*>(p);
  for (const char* q : {c, c + bytes - 1}) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, q) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    if (a.type != cudaMemoryTypeHost) return false;
  }
  return true;
}

// Enqueue one host-buffer call below kPipelineMinAtoms on the handle's stream:
// input copies, evaluation, totals, and the copies of the results and of the
// device error flags back to the host.  Nothing here synchronises or
// allocates, so it can be captured into a graph.
int enqueue_small_call(mtp_handle* h, int natoms, int stride, const int* itypes, const double* rijs, const int* js,
                       const int* jtypes, const int* counts, int flags, double* forces, double* eatom,
                       double* vatom) {
  const cudaStream_t s = h->stream;
  const size_t N = natoms, NS = N * stride;
  if (natoms > 0) {
    MTP_CUDA(h, cudaMemcpyAsync(h->d_itypes, itypes, N * sizeof(int), cudaMemcpyHostToDevice, s));
    MTP_CUDA(h, cudaMemcpyAsync(h->d_rijs, rijs, 3 * NS * sizeof(double), cudaMemcpyHostToDevice, s));
    MTP_CUDA(h, cudaMemcpyAsync(h->d_js, js, NS * sizeof(int), cudaMemcpyHostToDevice, s));
    MTP_CUDA(h, cudaMemcpyAsync(h->d_jtypes, jtypes, NS * sizeof(int), cudaMemcpyHostToDevice, s));
    if (counts) MTP_CUDA(h, cudaMemcpyAsync(h->d_counts, counts, N * sizeof(int), cudaMemcpyHostToDevice, s));
  }
  int st = run_device(h, natoms, stride, h->d_itypes, h->d_rijs, h->d_js, h->d_jtypes, counts ? h->d_counts : nullptr,
                      true, false, h->d_F, (flags & MTP_VATOM) ? h->d_vatom : nullptr);
  if (st != MTP_OK) return st;
  MTP_CUDA(h, launch_totals(natoms, h->d_E, h->d_wown, h->d_partials, h->d_tot, h->d_err, nullptr, nullptr, s));
  if (natoms > 0) {
    MTP_CUDA(h, cudaMemcpyAsync(forces, h->d_F, 3 * N * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (flags & MTP_EATOM) MTP_CUDA(h, cudaMemcpyAsync(eatom, h->d_E, N * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (flags & MTP_VATOM)
      MTP_CUDA(h, cudaMemcpyAsync(vatom, h->d_vatom, 6 * N * sizeof(double), cudaMemcpyDeviceToHost, s));
  }
  MTP_CUDA(h, cudaMemcpyAsync(h->h_tot, h->d_tot, 8 * sizeof(double), cudaMemcpyDeviceToHost, s));   // flags in the last
  return MTP_OK;
}

// Run one synchronous host-buffer call.  With every host buffer page-locked
// (pinned), the second consecutive call with the same key is captured into a
// graph and later ones replay it (one launch instead of about twenty copies
// and kernels); otherwise enqueue() runs directly.  The results are the same
// either way: the graph holds the same operations.
template <typename Enqueue>
int run_graphable(mtp_handle* h, const HostCallKey& key, bool pinned, Enqueue&& enqueue) {
  const cudaStream_t s = h->stream;
  bool launched = false;
  if (pinned && h->graph_exec && key == h->graph_key) {
    MTP_CUDA(h, cudaGraphLaunch(h->graph_exec, s));
    launched = true;
    ++h->graph_replays;
  } else if (pinned && key == h->seen_key && !h->seen_uncapturable) {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t ex = nullptr;
    if (!h->copy_stream) MTP_CUDA(h, cudaStreamCreateWithFlags(&h->copy_stream, cudaStreamNonBlocking));
    if (!h->fork_event) MTP_CUDA(h, cudaEventCreateWithFlags(&h->fork_event, cudaEventDisableTiming));
    if (!h->join_event) MTP_CUDA(h, cudaEventCreateWithFlags(&h->join_event, cudaEventDisableTiming));
    bool ok = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
    if (ok) {
      h->fork = true;
      const int cst = enqueue();
      h->fork = false;
      const cudaError_t ce = cudaStreamEndCapture(s, &g);
      ok = cst == MTP_OK && ce == cudaSuccess && g != nullptr;
    }
    if (ok) ok = cudaGraphInstantiate(&ex, g, 0) == cudaSuccess;
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    if (ok) {
      if (h->graph_exec) cudaGraphExecDestroy(h->graph_exec);
      h->graph_exec = ex;
      h->graph_key = key;
      MTP_CUDA(h, cudaGraphLaunch(ex, s));
      launched = true;
      ++h->graph_captures;
    } else {
      h->seen_uncapturable = true;
    }
  } else if (pinned) {
    h->seen_key = key;
    h->seen_uncapturable = false;
  }
  if (!launched) {
    const int st = enqueue();
    if (st != MTP_OK) {
      cudaStreamSynchronize(s);   // copies from the caller's buffers complete before the error returns
      return st;
    }
  }
  MTP_CUDA(h, cudaStreamSynchronize(s));
  return take_err_flags(h);
}

// One host-buffer call of mtp_compute below kPipelineMinAtoms (run_graphable).
int run_small_call(mtp_handle* h, int natoms, int stride, const int* itypes, const double* rijs, const int* js,
                   const int* jtypes, const int* counts, int flags, double* forces, double* eatom, double* vatom) {
  const size_t N = natoms, NS = N * stride;
  HostCallKey key;
  key.kind = 0;
  key.natoms = natoms;
  key.stride = stride;
  key.flags = flags & (MTP_EATOM | MTP_VATOM);
  key.gen = h->gen;
  const void* ptrs[8] = {itypes, rijs, js, jtypes, counts, forces,
                         (flags & MTP_EATOM) ? eatom : nullptr, (flags & MTP_VATOM) ? vatom : nullptr};
  for (int k = 0; k < 8; ++k) key.p[k] = ptrs[k];
  const bool pinned = natoms > 0 && !h->profiling && host_pinned(itypes, N * sizeof(int)) &&
                      host_pinned(rijs, 3 * NS * sizeof(double)) && host_pinned(js, NS * sizeof(int)) &&
                      host_pinned(jtypes, NS * sizeof(int)) && host_pinned(counts, counts ? N * sizeof(int) : 0) &&
                      host_pinned(forces, 3 * N * sizeof(double)) &&
                      host_pinned(key.p[6], (flags & MTP_EATOM) ? N * sizeof(double) : 0) &&
                      host_pinned(key.p[7], (flags & MTP_VATOM) ? 6 * N * sizeof(double) : 0);
  return run_graphable(h, key, pinned, [&]() {
    return enqueue_small_call(h, natoms, stride, itypes, rijs, js, jtypes, counts, flags, forces, eatom, vatom);
  });
}

bool ends_with(const std::string& s, const std::string& suf) {
  return s.size() >= suf.size() && s.compare(s.size() - suf.size(), suf.size(), suf) == 0;
}

}  // namespace

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

int mtp_abi_version(void) { return MTP_B200_ABI_VERSION; }

int mtp_parse_info(const char* path, int* out8, char* errbuf, int err_len) {
  if (!path || !out8) return MTP_E_INVALID;
  Potential pot;
  std::string err;
  if (!parse_mtp_file(path, pot, err)) {
    if (errbuf && err_len > 0) std::snprintf(errbuf, err_len, "%s", err.c_str());
    return MTP_E_FORMAT;
  }
  int D = 0;
  for (int k = 0; k < pot.B; ++k) D = std::max(D, pot.basic[4 * k + 1] + pot.basic[4 * k + 2] + pot.basic[4 * k + 3]);
  const int v[8] = {pot.S, pot.R, pot.K, pot.M, pot.B, pot.T, pot.Sa, D};
  std::memcpy(out8, v, sizeof(v));
  return MTP_OK;
}

int mtp_schedule_emulate(const char* path, int lanes, int width, const double* basic, double* moments,
                         double* dmoments, double* energy_part) {
  if (!path || !basic || !moments || !dmoments) return MTP_E_INVALID;
  if (width != 4 && width != 8 && width != 16) return MTP_E_INVALID;
  Potential pot;
  std::string err;
  if (!parse_mtp_file(path, pot, err)) return MTP_E_FORMAT;
  Schedule s;
  if (!build_schedule(pot, lanes, s, err, width)) return MTP_E_FORMAT;
  refine_schedule(s);
  std::vector<double> V(s.v_size, 0.0);
  for (int k = 0; k < pot.B; ++k) V[s.v_m + k] = basic[k];
  double e = emulate_schedule(pot, s, V);
  for (int k = 0; k < pot.M; ++k) {
    moments[k] = V[s.v_m + k];
    dmoments[k] = V[s.v_dm + s.dm_pos[k]];
  }
  if (energy_part) *energy_part = e;
  return MTP_OK;
}

int mtp_create(const char* mtp_path, int max_atoms, int max_nbr, double cutoff, int debug_level, int precision,
               mtp_handle** out) {
  if (!out) return fail(nullptr, MTP_E_INVALID, "out is null");
  *out = nullptr;
  if (!mtp_path) return fail(nullptr, MTP_E_INVALID, "mtp_path is null");
  if (max_atoms <= 0 || max_nbr <= 0 || !(cutoff > 0.0))
    return fail(nullptr, MTP_E_INVALID, "max_atoms, max_nbr and cutoff must be positive");
  if (precision != MTP_PRECISION_FP64 && precision != MTP_PRECISION_MIXED)
    return fail(nullptr, MTP_E_INVALID, "precision must be MTP_PRECISION_FP64 or MTP_PRECISION_MIXED");
  if (max_nbr > 1024) return fail(nullptr, MTP_E_CAPACITY, "max_nbr above the supported 1024");
  if (static_cast<long long>(max_atoms) * max_nbr >= (1LL << 31))
    return fail(nullptr, MTP_E_CAPACITY, "max_atoms * max_nbr must stay below 2^31");
  std::string path(mtp_path);
  if (ends_with(path, ".bin"))
    return fail(nullptr, MTP_E_FORMAT,
                "'" + path + "' looks like a jax.export .bin; this engine reads the .mtp potential file itself");
  auto* h = new mtp_handle();
  h->max_atoms = max_atoms;
  h->max_nbr = max_nbr;
  h->cutoff = cutoff;
  h->debug = debug_level;
  h->precision = precision;
  std::string err;
  if (!parse_mtp_file(path, h->pot, err)) {
    delete h;
    return fail(nullptr, MTP_E_FORMAT, err);
  }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    delete h;
    return fail(nullptr, MTP_E_NODEVICE, "no CUDA device");
  }
  auto bail = [&](int code) {
    g_create_error = h->err;
    free_handle(h);
    return code;
  };
  if (cudaGetDevice(&h->device) != cudaSuccess) return bail(cuda_fail(h, cudaGetLastError(), "cudaGetDevice"));
  cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, h->device);
  int l2 = 0;
  cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, h->device);
  h->l2_bytes = static_cast<size_t>(l2);
  if (cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking) != cudaSuccess)
    return bail(cuda_fail(h, cudaGetLastError(), "cudaStreamCreate"));
  h->stream = h->own_stream;
  const Potential& p = h->pot;
  const size_t N = static_cast<size_t>(max_atoms), NS = N * max_nbr;
  const size_t ncoef = p.radial.size() + p.S + 2 * static_cast<size_t>(p.Sa);
  bool ok = dalloc(&h->d_coef, ncoef) == cudaSuccess && dalloc(&h->d_mapping, p.Sa) == cudaSuccess &&
            dalloc(&h->d_seed_idx, p.Sa) == cudaSuccess &&
            dalloc(&h->d_itypes, N) == cudaSuccess && dalloc(&h->d_js, NS) == cudaSuccess &&
            dalloc(&h->d_jtypes, NS) == cudaSuccess && dalloc(&h->d_counts, N) == cudaSuccess &&
            dalloc(&h->d_rijs, 3 * NS) == cudaSuccess && dalloc(&h->d_G, 3 * NS) == cudaSuccess &&
            dalloc(&h->d_E, N) == cudaSuccess && dalloc(&h->d_F, 3 * N) == cudaSuccess &&
            dalloc(&h->d_wown, 6 * N) == cudaSuccess && dalloc(&h->d_vatom, 6 * N) == cudaSuccess &&
            dalloc(&h->d_in_cnt, N) == cudaSuccess && dalloc(&h->d_in_ptr, N + 1) == cudaSuccess &&
            dalloc(&h->d_in_slot, NS) == cudaSuccess &&
            dalloc(&h->d_blk, (N + 1023) / 1024 + 1) == cudaSuccess &&
            dalloc(&h->d_partials, 7 * kReduceBlocks) == cudaSuccess && dalloc(&h->d_tot, kTotals) == cudaSuccess &&
            dalloc(&h->d_err, 1) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    h->err = "device allocation failed for the requested capacities";
    return bail(MTP_E_OOM);
  }
  if (cudaMallocHost(&h->h_tot, 8 * sizeof(double)) != cudaSuccess ||
      cudaMallocHost(&h->h_coef, std::max<size_t>(ncoef, 1) * sizeof(double)) != cudaSuccess) {
    h->err = "pinned host allocation failed";
    return bail(MTP_E_OOM);
  }
  h->h_err = reinterpret_cast<int*>(h->h_tot + 7);
  cudaMemset(h->d_err, 0, sizeof(int));
  cudaMemset(h->d_tot, 0, kTotals * sizeof(double));
  if (cudaMemcpy(h->d_mapping, p.mapping.data(), p.Sa * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess)
    return bail(cuda_fail(h, cudaGetLastError(), "upload mapping"));
  h->d_radial = h->d_coef;
  h->d_species = h->d_radial + p.radial.size();
  h->d_theta = h->d_species + p.S;
  h->d_seed_val = h->d_theta + p.Sa;
  {
    // seeds of the reverse pass: the mapped moments, at their adjoint positions
    std::vector<int> si, dm_pos;
    std::vector<double> sv;
    seed_list(p, si, sv);
    adjoint_layout(p, dm_pos);
    h->nseed = static_cast<int>(si.size());
    std::map<int, int> seed;
    for (int k = 0; k < h->nseed; ++k) seed[si[k]] = k;
    for (int m : p.mapping) h->seed_of.push_back(seed[m]);
    for (int& k : si) k = dm_pos[k];
    if (cudaMemcpy(h->d_seed_idx, si.data(), si.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess)
      return bail(cuda_fail(h, cudaGetLastError(), "upload seeds"));
  }
  int st = upload_coeffs(h);
  if (st != MTP_OK) return bail(st);
  const DeviceSchedule* ds = nullptr;
  st = get_sizes(h, 256, &ds);   // checks the tables
  if (st != MTP_OK) return bail(st);
  if (h->debug >= 1) {
    std::fprintf(stderr, "[mtp_b200] %s: S=%d R=%d K=%d M=%d B=%d T=%d Sa=%d; %d fwd + %d rev passes, %d value slots\n",
                 path.c_str(), p.S, p.R, p.K, p.M, p.B, p.T, p.Sa, static_cast<int>(ds->sched.fwd.size()),
                 static_cast<int>(ds->sched.rev.size()), ds->sched.v_size);
  }
  *out = h;
  return MTP_OK;
}

void mtp_destroy(mtp_handle* h) {
  if (!h) return;
  if (h->debug >= 1 && h->calls > 0)
    std::fprintf(stderr, "[mtp_b200] %lld calls, %.3f ms total, %.3f ms/call\n", h->calls, h->total_ms,
                 h->total_ms / h->calls);
  if (h->stream) cudaStreamSynchronize(h->stream);
  free_handle(h);
}

const char* mtp_last_error(const mtp_handle* h) { return h ? h->err.c_str() : g_create_error.c_str(); }

int mtp_set_stream(mtp_handle* h, void* s) {
  if (!h) return MTP_E_INVALID;
  h->stream = static_cast<cudaStream_t>(s);
  return MTP_OK;
}

int mtp_use_own_stream(mtp_handle* h) {
  if (!h) return MTP_E_INVALID;
  h->stream = h->own_stream;
  return MTP_OK;
}

int mtp_get_info(const mtp_handle* h, int* out8) {
  if (!h || !out8) return MTP_E_INVALID;
  const Potential& p = h->pot;
  int D = 0;
  for (int k = 0; k < p.B; ++k) D = std::max(D, p.basic[4 * k + 1] + p.basic[4 * k + 2] + p.basic[4 * k + 3]);
  const int v[8] = {p.S, p.R, p.K, p.M, p.B, p.T, p.Sa, D};
  std::memcpy(out8, v, sizeof(v));
  return MTP_OK;
}

int mtp_get_stats(const mtp_handle* h, double* out4) {
  if (!h || !out4) return MTP_E_INVALID;
  out4[0] = static_cast<double>(h->calls);
  out4[1] = h->total_ms;
  out4[2] = static_cast<double>(h->graph_captures);
  out4[3] = static_cast<double>(h->graph_replays);
  return MTP_OK;
}

int mtp_set_coeffs(mtp_handle* h, const double* species, const double* moment, const double* radial) {
  if (!h) return MTP_E_INVALID;
  // (refused inside a stream capture, before the host's values change; the
  // legacy default stream cannot be captured and is the copy's own)
  if (h->stream) MTP_CUDA(h, cudaStreamSynchronize(h->stream));
  Potential& p = h->pot;
  if (species) std::copy(species, species + p.S, p.species.begin());
  if (moment) std::copy(moment, moment + p.Sa, p.moment.begin());
  if (radial) std::copy(radial, radial + p.radial.size(), p.radial.begin());
  ++h->gen;
  return upload_coeffs(h);
}

int mtp_set_launch(mtp_handle* h, int threads, int bps, int apb) {
  if (!h) return MTP_E_INVALID;
  if (threads != 128 && threads != 256 && threads != 512)
    return fail(h, MTP_E_INVALID, "threads_per_block must be 128, 256 or 512");
  if (apb != 0 && apb != 1 && apb != 2 && apb != 4)
    return fail(h, MTP_E_INVALID, "atoms_per_block must be 0 (automatic), 1, 2 or 4");
  h->threads = threads;
  h->blocks_per_sm = std::max(0, bps);
  h->apb = apb;
  ++h->gen;
  return MTP_OK;
}

int mtp_get_launch(const mtp_handle* h, int* out5) {
  if (!h || !out5) return MTP_E_INVALID;
  out5[0] = h->last.lanes;
  out5[1] = h->last_blocks;
  out5[2] = static_cast<int>(h->last.fit.smem);
  out5[3] = h->last.fit.per_sm;
  out5[4] = h->last.A;
  return MTP_OK;
}

int mtp_sync_status(mtp_handle* h) {
  if (!h) return MTP_E_INVALID;
  return read_err_flags(h);
}

int mtp_compute_device(mtp_handle* h, int natoms, int stride, const int* d_itypes, const double* d_rijs,
                       const int* d_js, const int* d_jtypes, const int* d_counts, int flags, double* d_energy,
                       double* d_forces, double* d_virial, double* d_eatom, double* d_vatom) {
  if (!h) return MTP_E_INVALID;
  if (natoms < 0 || stride <= 0) return fail(h, MTP_E_INVALID, "natoms must be >= 0 and nbr_stride > 0");
  if (natoms > h->max_atoms) return fail(h, MTP_E_CAPACITY, "natoms exceeds max_atoms");
  if (stride > h->max_nbr) return fail(h, MTP_E_CAPACITY, "nbr_stride exceeds max_nbr");
  if (natoms > 0 && (!d_itypes || !d_rijs || !d_js || !d_jtypes || !d_forces))
    return fail(h, MTP_E_INVALID, "null input or forces pointer");
  if ((flags & MTP_EFLAG) && !d_energy) return fail(h, MTP_E_INVALID, "MTP_EFLAG without an energy pointer");
  if ((flags & MTP_VFLAG) && !d_virial) return fail(h, MTP_E_INVALID, "MTP_VFLAG without a virial pointer");
  if ((flags & MTP_EATOM) && !d_eatom) return fail(h, MTP_E_INVALID, "MTP_EATOM without an eatom pointer");
  if ((flags & MTP_VATOM) && !d_vatom) return fail(h, MTP_E_INVALID, "MTP_VATOM without a vatom pointer");
  const bool rebuild = !(flags & MTP_REUSE_NEIGHBORS);
  int st = run_device(h, natoms, stride, d_itypes, d_rijs, d_js, d_jtypes, d_counts, rebuild, false, d_forces,
                      (flags & MTP_VATOM) ? d_vatom : nullptr);
  if (st != MTP_OK) return st;
  if (flags & (MTP_EFLAG | MTP_VFLAG)) {
    st = write_totals(h, natoms, h->d_E, h->d_wown, h->d_partials, h->d_tot, (flags & MTP_EFLAG) ? d_energy : nullptr,
                      (flags & MTP_VFLAG) ? d_virial : nullptr);
    if (st != MTP_OK) return st;
  }
  if ((flags & MTP_EATOM) && natoms > 0)
    MTP_CUDA(h, cudaMemcpyAsync(d_eatom, h->d_E, natoms * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  h->calls++;
  return MTP_OK;
}

int mtp_compute_positions_device(mtp_handle* h, int nlocal, int nall, const double* d_x, const int* d_species,
                                 const int* d_owner, int list_stride, const int* d_neigh, const int* d_numneigh,
                                 int flags, double* d_energy, double* d_forces, double* d_virial, double* d_eatom,
                                 double* d_vatom) {
  if (!h) return MTP_E_INVALID;
  if (nlocal < 0 || nall < nlocal || list_stride < 0)
    return fail(h, MTP_E_INVALID, "need 0 <= nlocal <= nall and list_stride >= 0");
  if (nlocal > h->max_atoms) return fail(h, MTP_E_CAPACITY, "nlocal exceeds max_atoms");
  if (nlocal > 0 && (list_stride == 0 || !d_x || !d_species || !d_owner || !d_neigh || !d_numneigh || !d_forces))
    return fail(h, MTP_E_INVALID, "null input or forces pointer, or list_stride 0 with atoms");
  if ((flags & MTP_EFLAG) && !d_energy) return fail(h, MTP_E_INVALID, "MTP_EFLAG without an energy pointer");
  if ((flags & MTP_VFLAG) && !d_virial) return fail(h, MTP_E_INVALID, "MTP_VFLAG without a virial pointer");
  if ((flags & MTP_EATOM) && !d_eatom) return fail(h, MTP_E_INVALID, "MTP_EATOM without an eatom pointer");
  if ((flags & MTP_VATOM) && !d_vatom) return fail(h, MTP_E_INVALID, "MTP_VATOM without a vatom pointer");
  const int stride = h->max_nbr;
  if (nlocal > 0)
    MTP_CUDA(h, launch_rows_from_positions(nlocal, nall, d_x, d_species, d_owner, list_stride, d_neigh, d_numneigh,
                                           h->cutoff, stride, h->d_rijs, h->d_js, h->d_jtypes, h->d_counts,
                                           h->d_in_cnt, h->d_err, h->stream));
  int st = run_device(h, nlocal, stride, nlocal > 0 ? d_species : h->d_itypes, h->d_rijs, h->d_js, h->d_jtypes,
                      h->d_counts, true, true, d_forces, (flags & MTP_VATOM) ? d_vatom : nullptr);
  if (st != MTP_OK) return st;
  if (flags & (MTP_EFLAG | MTP_VFLAG)) {
    st = write_totals(h, nlocal, h->d_E, h->d_wown, h->d_partials, h->d_tot, (flags & MTP_EFLAG) ? d_energy : nullptr,
                      (flags & MTP_VFLAG) ? d_virial : nullptr);
    if (st != MTP_OK) return st;
  }
  if ((flags & MTP_EATOM) && nlocal > 0)
    MTP_CUDA(h, cudaMemcpyAsync(d_eatom, h->d_E, nlocal * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  h->calls++;
  return MTP_OK;
}

int mtp_compute(mtp_handle* h, int natoms, int stride, const int* itypes, const double* rijs, const int* js,
                const int* jtypes, const int* counts, int flags, double* energy, double* forces, double* virial,
                double* eatom, double* vatom) {
  if (!h) return MTP_E_INVALID;
  if (natoms < 0 || stride <= 0) return fail(h, MTP_E_INVALID, "natoms must be >= 0 and nbr_stride > 0");
  if (natoms > h->max_atoms)
    return fail(h, MTP_E_CAPACITY, "natoms " + std::to_string(natoms) + " exceeds max_atoms " +
                                        std::to_string(h->max_atoms));
  if (stride > h->max_nbr) return fail(h, MTP_E_CAPACITY, "nbr_stride exceeds max_nbr");
  if (natoms > 0 && (!itypes || !rijs || !js || !jtypes || !forces))
    return fail(h, MTP_E_INVALID, "null input or forces pointer");
  if ((flags & MTP_EFLAG) && !energy) return fail(h, MTP_E_INVALID, "MTP_EFLAG without an energy pointer");
  if ((flags & MTP_VFLAG) && !virial) return fail(h, MTP_E_INVALID, "MTP_VFLAG without a virial pointer");
  if ((flags & MTP_EATOM) && !eatom) return fail(h, MTP_E_INVALID, "MTP_EATOM without an eatom pointer");
  if ((flags & MTP_VATOM) && !vatom) return fail(h, MTP_E_INVALID, "MTP_VATOM without a vatom pointer");
  if (counts) {
    for (int i = 0; i < natoms; ++i)
      if (counts[i] < 0 || counts[i] > stride)
        return fail(h, MTP_E_CAPACITY, "atom " + std::to_string(i) + " has " + std::to_string(counts[i]) +
                                            " neighbours, more than the row length " + std::to_string(stride));
  }
  auto t0 = std::chrono::steady_clock::now();
  const size_t N = natoms;
  cudaStream_t s = h->stream;
  int st;
  if (natoms >= kPipelineMinAtoms) {
    st = run_host_pipelined(h, natoms, stride, itypes, rijs, js, jtypes, counts,
                            (flags & MTP_VATOM) ? h->d_vatom : nullptr);
    if (st != MTP_OK) {
      cudaStreamSynchronize(s);   // copies from the caller's buffers complete before the error returns
      return st;
    }
    MTP_CUDA(h, launch_totals(natoms, h->d_E, h->d_wown, h->d_partials, h->d_tot, h->d_err, nullptr, nullptr, s));
    MTP_CUDA(h, cudaMemcpyAsync(forces, h->d_F, 3 * N * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (flags & MTP_EATOM) MTP_CUDA(h, cudaMemcpyAsync(eatom, h->d_E, N * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (flags & MTP_VATOM)
      MTP_CUDA(h, cudaMemcpyAsync(vatom, h->d_vatom, 6 * N * sizeof(double), cudaMemcpyDeviceToHost, s));
    MTP_CUDA(h, cudaMemcpyAsync(h->h_tot, h->d_tot, 7 * sizeof(double), cudaMemcpyDeviceToHost, s));
    st = read_err_flags(h);   // synchronises the stream
  } else {
    st = run_small_call(h, natoms, stride, itypes, rijs, js, jtypes, counts, flags, forces, eatom, vatom);
  }
  if (st != MTP_OK) return st;
  if (flags & MTP_EFLAG) *energy = h->h_tot[0];
  if (flags & MTP_VFLAG)
    for (int c = 0; c < 6; ++c) virial[c] = h->h_tot[1 + c];
  h->calls++;
  double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  h->total_ms += ms;
  if (h->debug >= 2) std::fprintf(stderr, "[mtp_b200] call %lld: natoms=%d %.3f ms\n", h->calls, natoms, ms);
  return MTP_OK;
}

int mtp_compute_positions(mtp_handle* h, int nlocal, int nall, const double* x, const int* species, const int* owner,
                          int list_stride, const int* neigh, const int* numneigh, int flags, double* energy,
                          double* forces, double* virial, double* eatom, double* vatom) {
  if (!h) return MTP_E_INVALID;
  if (nlocal < 0 || nall < nlocal || list_stride < 0)
    return fail(h, MTP_E_INVALID, "need 0 <= nlocal <= nall and list_stride >= 0");
  if (nlocal > h->max_atoms)
    return fail(h, MTP_E_CAPACITY, "nlocal " + std::to_string(nlocal) + " exceeds max_atoms " +
                                        std::to_string(h->max_atoms));
  if (nlocal > 0 && (list_stride == 0 || !x || !species || !owner || !neigh || !numneigh || !forces))
    return fail(h, MTP_E_INVALID, "null input or forces pointer, or list_stride 0 with atoms");
  if ((flags & MTP_EFLAG) && !energy) return fail(h, MTP_E_INVALID, "MTP_EFLAG without an energy pointer");
  if ((flags & MTP_VFLAG) && !virial) return fail(h, MTP_E_INVALID, "MTP_VFLAG without a virial pointer");
  if ((flags & MTP_EATOM) && !eatom) return fail(h, MTP_E_INVALID, "MTP_EATOM without an eatom pointer");
  if ((flags & MTP_VATOM) && !vatom) return fail(h, MTP_E_INVALID, "MTP_VATOM without a vatom pointer");
  auto t0 = std::chrono::steady_clock::now();
  const cudaStream_t s = h->stream;
  const size_t N = nlocal, NA = nall, NN = N * list_stride;
  if (NA > h->all_cap) {
    MTP_CUDA(h, cudaStreamSynchronize(s));
    cudaFree(h->d_xall);
    cudaFree(h->d_spall);
    cudaFree(h->d_owner);
    h->d_xall = nullptr;
    h->d_spall = h->d_owner = nullptr;
    h->all_cap = 0;
    ++h->gen;
    MTP_CUDA(h, dalloc(&h->d_xall, 3 * NA));
    MTP_CUDA(h, dalloc(&h->d_spall, NA));
    MTP_CUDA(h, dalloc(&h->d_owner, NA));
    h->all_cap = NA;
  }
  if (NN > h->neigh_cap) {
    MTP_CUDA(h, cudaStreamSynchronize(s));
    cudaFree(h->d_neigh);
    h->d_neigh = nullptr;
    h->neigh_cap = 0;
    ++h->gen;
    MTP_CUDA(h, dalloc(&h->d_neigh, NN));
    h->neigh_cap = NN;
  }
  if (!h->d_numneigh) MTP_CUDA(h, dalloc(&h->d_numneigh, static_cast<size_t>(h->max_atoms)));
  const int stride = h->max_nbr;
  // copies, rows, evaluation, totals and read-backs; nothing here
  // synchronises or allocates, so run_graphable may capture it
  auto enqueue = [&]() -> int {
    if (nlocal > 0) {
      MTP_CUDA(h, cudaMemcpyAsync(h->d_xall, x, 3 * NA * sizeof(double), cudaMemcpyHostToDevice, s));
      MTP_CUDA(h, cudaMemcpyAsync(h->d_spall, species, NA * sizeof(int), cudaMemcpyHostToDevice, s));
      MTP_CUDA(h, cudaMemcpyAsync(h->d_owner, owner, NA * sizeof(int), cudaMemcpyHostToDevice, s));
      MTP_CUDA(h, cudaMemcpyAsync(h->d_neigh, neigh, NN * sizeof(int), cudaMemcpyHostToDevice, s));
      MTP_CUDA(h, cudaMemcpyAsync(h->d_numneigh, numneigh, N * sizeof(int), cudaMemcpyHostToDevice, s));
      MTP_CUDA(h, launch_rows_from_positions(nlocal, nall, h->d_xall, h->d_spall, h->d_owner, list_stride,
                                             h->d_neigh, h->d_numneigh, h->cutoff, stride, h->d_rijs, h->d_js,
                                             h->d_jtypes, h->d_counts, h->d_in_cnt, h->d_err, s));
    }
    int st = run_device(h, nlocal, stride, nlocal > 0 ? h->d_spall : h->d_itypes, h->d_rijs, h->d_js, h->d_jtypes,
                        h->d_counts, true, true, h->d_F, (flags & MTP_VATOM) ? h->d_vatom : nullptr);
    if (st != MTP_OK) return st;
    MTP_CUDA(h, launch_totals(nlocal, h->d_E, h->d_wown, h->d_partials, h->d_tot, h->d_err, nullptr, nullptr, s));
    if (nlocal > 0) {
      MTP_CUDA(h, cudaMemcpyAsync(forces, h->d_F, 3 * N * sizeof(double), cudaMemcpyDeviceToHost, s));
      if (flags & MTP_EATOM)
        MTP_CUDA(h, cudaMemcpyAsync(eatom, h->d_E, N * sizeof(double), cudaMemcpyDeviceToHost, s));
      if (flags & MTP_VATOM)
        MTP_CUDA(h, cudaMemcpyAsync(vatom, h->d_vatom, 6 * N * sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    MTP_CUDA(h, cudaMemcpyAsync(h->h_tot, h->d_tot, 8 * sizeof(double), cudaMemcpyDeviceToHost, s));   // flags in the last
    return MTP_OK;
  };
  HostCallKey key;
  key.kind = 1;
  key.natoms = nlocal;
  key.stride = list_stride;
  key.extra = nall;
  key.flags = flags & (MTP_EATOM | MTP_VATOM);
  key.gen = h->gen;
  const void* ptrs[8] = {x, species, owner, neigh, numneigh, forces,
                         (flags & MTP_EATOM) ? eatom : nullptr, (flags & MTP_VATOM) ? vatom : nullptr};
  for (int k = 0; k < 8; ++k) key.p[k] = ptrs[k];
  const bool pinned = nlocal > 0 && !h->profiling && host_pinned(x, 3 * NA * sizeof(double)) &&
                      host_pinned(species, NA * sizeof(int)) && host_pinned(owner, NA * sizeof(int)) &&
                      host_pinned(neigh, NN * sizeof(int)) && host_pinned(numneigh, N * sizeof(int)) &&
                      host_pinned(forces, 3 * N * sizeof(double)) &&
                      host_pinned(key.p[6], (flags & MTP_EATOM) ? N * sizeof(double) : 0) &&
                      host_pinned(key.p[7], (flags & MTP_VATOM) ? 6 * N * sizeof(double) : 0);
  const int st = run_graphable(h, key, pinned, enqueue);
  if (st != MTP_OK) return st;
  if (flags & MTP_EFLAG) *energy = h->h_tot[0];
  if (flags & MTP_VFLAG)
    for (int c = 0; c < 6; ++c) virial[c] = h->h_tot[1 + c];
  h->calls++;
  h->total_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  return MTP_OK;
}

int mtp_execute_potential(mtp_handle* h, int natoms, int nneigh_total, const double* const* atom_positions,
                          const int* atom_types, const int* const* neighbor_lists, const int* neighbor_counts,
                          const int* const* neighbor_types_lists, double volume, double* energy, double** forces,
                          double* stress) {
  (void)nneigh_total;
  if (!h) return MTP_E_INVALID;
  if (natoms < 0) return fail(h, MTP_E_INVALID, "natoms must be >= 0");
  if (natoms > h->max_atoms) return fail(h, MTP_E_CAPACITY, "natoms exceeds max_atoms");
  if (natoms > 0 && (!atom_positions || !atom_types || !neighbor_lists || !neighbor_counts || !neighbor_types_lists ||
                     !forces || !energy || !stress))
    return fail(h, MTP_E_INVALID, "null argument");
  const int stride = h->max_nbr;
  for (int i = 0; i < natoms; ++i) {
    const int c = neighbor_counts[i];
    if (c < 0 || c > stride)
      return fail(h, MTP_E_CAPACITY, "atom " + std::to_string(i) + " has " + std::to_string(c) +
                                          " neighbours, more than MAX_ATOMS_PER_NEIGHBOR");
  }
  // persistent page-locked staging (the reference bridge refilled persistent
  // NumPy buffers, zero_overhead.cpp:61-117): no allocation per step, and the
  // rows reach the GPU by DMA
  if (!h->hp_rij) {
    const size_t rows = static_cast<size_t>(h->max_atoms), slots = rows * stride;
    void *a = nullptr, *b = nullptr, *c = nullptr, *d = nullptr, *e = nullptr, *f = nullptr;
    const bool ok = cudaHostAlloc(&a, 3 * slots * sizeof(double), cudaHostAllocDefault) == cudaSuccess &&
                    cudaHostAlloc(&b, slots * sizeof(int), cudaHostAllocDefault) == cudaSuccess &&
                    cudaHostAlloc(&c, slots * sizeof(int), cudaHostAllocDefault) == cudaSuccess &&
                    cudaHostAlloc(&d, std::max<size_t>(rows, 1) * sizeof(int), cudaHostAllocDefault) == cudaSuccess &&
                    cudaHostAlloc(&e, std::max<size_t>(rows, 1) * sizeof(int), cudaHostAllocDefault) == cudaSuccess &&
                    cudaHostAlloc(&f, 3 * std::max<size_t>(rows, 1) * sizeof(double), cudaHostAllocDefault) ==
                        cudaSuccess;
    if (!ok) {
      for (void* q : {a, b, c, d, e, f})
        if (q) cudaFreeHost(q);
      cudaGetLastError();
      return fail(h, MTP_E_OOM, "mtp_execute_potential: page-locked staging allocation failed");
    }
    h->hp_rij = static_cast<double*>(a);
    h->hp_js = static_cast<int*>(b);
    h->hp_jt = static_cast<int*>(c);
    h->hp_cnt = static_cast<int*>(d);
    h->hp_types = static_cast<int*>(e);
    h->hp_F = static_cast<double*>(f);
  }
  // pack the counted slots of each row into the flat layout (what the
  // reference bridge copies into its NumPy buffers, zero_overhead.cpp:94-116);
  // slots past a row's count are never read
  for (int i = 0; i < natoms; ++i) {
    const int c = neighbor_counts[i];
    h->hp_cnt[i] = c;
    h->hp_types[i] = atom_types[i];
    if (c == 0) continue;
    std::memcpy(h->hp_rij + static_cast<size_t>(i) * stride * 3, atom_positions[i], 3 * c * sizeof(double));
    std::memcpy(h->hp_js + static_cast<size_t>(i) * stride, neighbor_lists[i], c * sizeof(int));
    std::memcpy(h->hp_jt + static_cast<size_t>(i) * stride, neighbor_types_lists[i], c * sizeof(int));
  }
  double vir[6] = {0, 0, 0, 0, 0, 0}, e = 0.0;
  int st = mtp_compute(h, natoms, stride, h->hp_types, h->hp_rij, h->hp_js, h->hp_jt, h->hp_cnt,
                       MTP_EFLAG | MTP_VFLAG, &e, h->hp_F, vir, nullptr, nullptr);
  if (st != MTP_OK) return st;
  *energy = e;
  for (int i = 0; i < natoms; ++i)
    for (int c = 0; c < 3; ++c) forces[i][c] = h->hp_F[3 * static_cast<size_t>(i) + c];
  // reference stress: +sym(sum r g)/V, order xx,yy,zz,yz,xz,xy (jax_backend.py:355-360)
  const double iv = 1.0 / volume;
  stress[0] = -vir[0] * iv;
  stress[1] = -vir[1] * iv;
  stress[2] = -vir[2] * iv;
  stress[3] = -vir[5] * iv;
  stress[4] = -vir[4] * iv;
  stress[5] = -vir[3] * iv;
  return MTP_OK;
}

int mtp_compute_batch_device(mtp_handle* h, int natoms, int stride, int nconfig, const int* d_itypes,
                             const double* d_rijs, const int* d_js, const int* d_jtypes, const int* d_counts,
                             const int* d_cfg, const double* d_volumes, double* d_energy, double* d_forces,
                             double* d_stress) {
  if (!h) return MTP_E_INVALID;
  if (natoms < 0 || stride <= 0 || nconfig < 0) return fail(h, MTP_E_INVALID, "bad sizes");
  if (natoms > h->max_atoms) return fail(h, MTP_E_CAPACITY, "natoms exceeds max_atoms");
  if (stride > h->max_nbr) return fail(h, MTP_E_CAPACITY, "nbr_stride exceeds max_nbr");
  if (natoms > 0 && (!d_itypes || !d_rijs || !d_js || !d_jtypes || !d_cfg || !d_volumes || !d_energy ||
                     !d_forces || !d_stress))
    return fail(h, MTP_E_INVALID, "null pointer");
  if (nconfig + 1 > h->cfg_cap) {
    if (h->d_cfg_ptr) cudaFree(h->d_cfg_ptr);
    h->d_cfg_ptr = nullptr;
    MTP_CUDA(h, dalloc(&h->d_cfg_ptr, nconfig + 1));
    h->cfg_cap = nconfig + 1;
  }
  MTP_CUDA(h, launch_config_ptr(natoms, nconfig, d_cfg, h->d_cfg_ptr, h->d_err, h->stream));
  int st = run_device(h, natoms, stride, d_itypes, d_rijs, d_js, d_jtypes, d_counts, true, false, d_forces, nullptr);
  if (st != MTP_OK) return st;
  MTP_CUDA(h, launch_config_totals(natoms, nconfig, h->d_cfg_ptr, h->d_E, h->d_wown, d_volumes, d_energy, d_stress,
                                   h->stream));
  h->calls++;
  return MTP_OK;
}

int mtp_adjoint_batch_device(mtp_handle* h, int natoms, int stride, int nconfig, const int* d_itypes,
                             const double* d_rijs, const int* d_js, const int* d_jtypes, const int* d_counts,
                             const int* d_cfg, const double* d_volumes, const double* d_gE, const double* d_gF,
                             const double* d_gS, double* d_gspecies, double* d_gmoment, double* d_gradial) {
  if (!h) return MTP_E_INVALID;
  if (natoms < 0 || stride <= 0 || nconfig < 0) return fail(h, MTP_E_INVALID, "bad sizes");
  if (natoms > h->max_atoms) return fail(h, MTP_E_CAPACITY, "natoms exceeds max_atoms");
  if (stride > h->max_nbr) return fail(h, MTP_E_CAPACITY, "nbr_stride exceeds max_nbr");
  if (!d_gspecies || !d_gmoment || !d_gradial) return fail(h, MTP_E_INVALID, "null gradient pointer");
  if (natoms > 0 && (!d_itypes || !d_rijs || !d_js || !d_jtypes || !d_cfg || !d_volumes || !d_gE || !d_gF || !d_gS))
    return fail(h, MTP_E_INVALID, "null pointer");
  // with the value space in global memory, 512 lanes give the SM twice the
  // warps for the same L2 footprint
  int lanes = h->threads > 0 ? h->threads : 256;
  const DeviceSchedule* ds = nullptr;
  int st = get_sizes(h, lanes, &ds);
  if (st != MTP_OK) return st;
  if (lanes < 512 && !adjoint_fits_shared(make_model(h, *ds), stride, lanes)) lanes = 512;
  // an operand is a value and its tangent, 16 bytes (also where the value space
  // is in global memory: L1 serves a gather by the same banks; entries ordered
  // for 8 bytes: level 28, 64 configurations 35.8 ms, for 16: 32.2 ms)
  st = get_schedule(h, lanes, 2 * access_width(true, 1), &ds);
  if (st != MTP_OK) return st;
  DevModel md = make_model(h, *ds);
  TrainIO tio{};
  tio.natoms = natoms;
  tio.nbr_stride = stride;
  tio.nconfig = nconfig;
  tio.itypes = d_itypes;
  tio.rijs = d_rijs;
  tio.js = d_js;
  tio.jtypes = d_jtypes;
  tio.counts = d_counts;
  tio.cfg = d_cfg;
  tio.volumes = d_volumes;
  tio.gE = d_gE;
  tio.gF = d_gF;
  tio.gS = d_gS;
  tio.err = h->d_err;
  std::string err;
  cudaError_t ce = launch_adjoint(md, tio, lanes, h->sm_count, h->train, d_gspecies, d_gmoment, d_gradial,
                                  h->stream, err);
  if (!err.empty()) return fail(h, MTP_E_CAPACITY, err);
  if (ce != cudaSuccess) return cuda_fail(h, ce, "adjoint");
  h->calls++;
  return MTP_OK;
}

namespace {
int ensure_cells(mtp_handle* h, int n, int ncell) {
  CellScratch& c = h->cells;
  if (n > c.n_cap) {
    if (c.cell) cudaFree(c.cell);
    if (c.img) cudaFree(c.img);
    if (c.atoms) cudaFree(c.atoms);
    c.cell = c.img = c.atoms = nullptr;
    c.n_cap = 0;
    MTP_CUDA(h, dalloc(&c.cell, n));
    MTP_CUDA(h, dalloc(&c.img, 3 * static_cast<size_t>(n)));
    MTP_CUDA(h, dalloc(&c.atoms, n));
    c.n_cap = n;
  }
  if (ncell > c.cell_cap) {
    if (c.cnt) cudaFree(c.cnt);
    if (c.ptr) cudaFree(c.ptr);
    if (c.cursor) cudaFree(c.cursor);
    if (c.blk) cudaFree(c.blk);
    c.cnt = c.ptr = c.cursor = c.blk = nullptr;
    c.cell_cap = 0;
    MTP_CUDA(h, dalloc(&c.cnt, ncell));
    MTP_CUDA(h, dalloc(&c.ptr, ncell + 1));
    MTP_CUDA(h, dalloc(&c.cursor, ncell));
    MTP_CUDA(h, dalloc(&c.blk, ncell / 1024 + 2));
    c.cell_cap = ncell;
  }
  return MTP_OK;
}
}  // namespace

int mtp_neighbors_device(mtp_handle* h, int natoms, const double* d_pos, const double* cell9, const int* d_types,
                         double cutoff, int stride, int* d_js, int* d_image, int* d_jtypes, int* d_counts) {
  if (!h) return MTP_E_INVALID;
  if (natoms < 0 || stride <= 0 || !(cutoff > 0.0) || !cell9) return fail(h, MTP_E_INVALID, "bad arguments");
  if (natoms > 0 && (!d_pos || !d_types || !d_js || !d_image || !d_jtypes || !d_counts))
    return fail(h, MTP_E_INVALID, "null pointer");
  Box b;
  if (!make_box(cell9, cutoff, b)) return fail(h, MTP_E_INVALID, "singular cell");
  if (b.nc[0] < 1 || b.nc[1] < 1 || b.nc[2] < 1)
    return fail(h, MTP_E_INVALID, "cell thinner than the cutoff: build these rows on the host");
  const long long ncell = static_cast<long long>(b.nc[0]) * b.nc[1] * b.nc[2];
  if (ncell > (1LL << 28)) return fail(h, MTP_E_CAPACITY, "too many cells");
  int st = ensure_cells(h, natoms, static_cast<int>(ncell));
  if (st != MTP_OK) return st;
  MTP_CUDA(h, launch_neighbors(natoms, d_pos, b, d_types, cutoff, stride, d_js, d_image, d_jtypes, d_counts,
                               h->cells, h->d_err, h->stream));
  return MTP_OK;
}

int mtp_pack_rij_device(mtp_handle* h, int natoms, int stride, const double* d_pos, const double* cell9,
                        const int* d_js, const int* d_image, const int* d_counts, double* d_rijs) {
  if (!h) return MTP_E_INVALID;
  if (natoms < 0 || stride <= 0 || !cell9) return fail(h, MTP_E_INVALID, "bad arguments");
  if (natoms > 0 && (!d_pos || !d_js || !d_image || !d_counts || !d_rijs)) return fail(h, MTP_E_INVALID, "null pointer");
  Box b;
  if (!make_box(cell9, 1.0, b)) return fail(h, MTP_E_INVALID, "singular cell");
  MTP_CUDA(h, launch_pack_rij(natoms, stride, d_pos, b, d_js, d_image, d_counts, d_rijs, h->stream));
  return MTP_OK;
}

int mtp_verlet_device(mtp_handle* h, int natoms, double* d_x, double* d_v, const double* d_f, const int* d_types,
                      const double* masses, int nmasses, double dt, int stage) {
  if (!h) return MTP_E_INVALID;
  if (natoms < 0 || !masses || nmasses <= 0 || nmasses > kMaxMdSpecies || (stage != 1 && stage != 2))
    return fail(h, MTP_E_INVALID, "bad arguments");
  VerletParams p{};
  p.dt = dt;
  p.ftm2v = 1.0 / 1.0364269e-4;   // LAMMPS 'metal' force->ftm2v
  for (int t = 0; t < kMaxMdSpecies; ++t) p.inv_mass[t] = 1.0 / masses[std::min(t, nmasses - 1)];
  MTP_CUDA(h, launch_verlet(natoms, d_x, d_v, d_f, d_types, p, stage, h->stream));
  return MTP_OK;
}

int mtp_profile(mtp_handle* h, int enable) {
  if (!h) return MTP_E_INVALID;
  h->profiling = enable != 0;
  h->prof_used = 0;
  return MTP_OK;
}

int mtp_profile_read(mtp_handle* h, double* ms, int* launches) {
  if (!h || !ms || !launches) return MTP_E_INVALID;
  MTP_CUDA(h, cudaStreamSynchronize(h->stream));
  double tot = 0.0;
  for (int i = 0; i < h->prof_used; ++i) {
    float x = 0.f;
    MTP_CUDA(h, cudaEventElapsedTime(&x, h->prof_events[i].first, h->prof_events[i].second));
    tot += x;
  }
  *ms = tot;
  *launches = h->prof_used;
  return MTP_OK;
}

int mtp_measure_fma_peak(double* fp64, double* fp32) {
  if (!fp64 || !fp32) return MTP_E_INVALID;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return MTP_E_NODEVICE;
  }
  return measure_fma_peak(fp64, fp32) == cudaSuccess ? MTP_OK : MTP_E_CUDA;
}

int mtp_host_alloc(size_t bytes, void** out) {
  if (!out) return fail(nullptr, MTP_E_INVALID, "mtp_host_alloc: null output pointer");
  *out = nullptr;
  if (bytes == 0) return MTP_OK;
  const cudaError_t e = cudaHostAlloc(out, bytes, cudaHostAllocDefault);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *out = nullptr;
    return fail(nullptr, e == cudaErrorMemoryAllocation ? MTP_E_OOM : MTP_E_CUDA,
                std::string("mtp_host_alloc: ") + cudaGetErrorString(e));
  }
  return MTP_OK;
}

int mtp_host_free(void* p) {
  if (!p) return MTP_OK;
  const cudaError_t e = cudaFreeHost(p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(nullptr, MTP_E_CUDA, std::string("mtp_host_free: ") + cudaGetErrorString(e));
  }
  return MTP_OK;
}

}  // extern "C"

// ===========================================================================
// Allocation-free evaluation (mtp_compute_device_noalloc)
// ===========================================================================
// Some callers cannot let a library call cudaMalloc: code that runs while a
// CUDA stream is being captured into a graph (allocation is illegal there),
// code that must not synchronise the device (cudaMalloc/cudaFree may), and
// hosts whose memory pool owns the whole device.  This variant of
// mtp_compute_device keeps every piece of its scratch memory in one
// file-scope device array of fixed size instead of handle buffers, and uses
// only the contraction schedules the handle already uploaded.
namespace {

constexpr size_t al256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

struct NoAllocLayout {
  size_t grad, energy, wown, in_cnt, in_ptr, in_slot, blk, partials, tot, total;
};

constexpr NoAllocLayout noalloc_layout() {
  NoAllocLayout L{};
  const size_t atoms = MTP_NOALLOC_MAX_ATOMS, slots = MTP_NOALLOC_MAX_SLOTS;
  size_t o = 0;
  L.grad = o;      o = al256(o + slots * 3 * sizeof(double));
  L.energy = o;    o = al256(o + atoms * sizeof(double));
  L.wown = o;      o = al256(o + atoms * 6 * sizeof(double));
  L.in_cnt = o;    o = al256(o + atoms * sizeof(int));
  L.in_ptr = o;    o = al256(o + (atoms + 1) * sizeof(int));
  L.in_slot = o;   o = al256(o + slots * sizeof(int));
  L.blk = o;       o = al256(o + (atoms / 1024 + 2) * sizeof(int));
  L.partials = o;  o = al256(o + 7 * kReduceBlocks * sizeof(double));
  L.tot = o;       o = al256(o + kTotals * sizeof(double));
  L.total = o;
  return L;
}

constexpr NoAllocLayout kNoAlloc = noalloc_layout();

// The scratch (about 8.5 MB).  Every GPU that loads this library holds it
// until the process exits; all calls on a device share it.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAlloc.total];

// Device address of g_noalloc_scratch on the current device.  In host code
// the symbol is only a host-side stand-in, so the address is asked for once
// per device (with that device current) and cached for the life of the
// process; a reset of the device's primary context (cudaDeviceReset) makes the
// cached address stale, which the header states as a limit of this path.
int noalloc_base(mtp_handle* h, unsigned char** out) {
  static std::mutex mu;
  static unsigned char* base[64] = {};
  int dev = -1;
  MTP_CUDA(h, cudaGetDevice(&dev));
  if (dev != h->device) return fail(h, MTP_E_INVALID, "the current CUDA device is not the handle's device");
  if (dev < 0 || dev >= 64) return fail(h, MTP_E_INVALID, "device ordinal above 63");
  std::lock_guard<std::mutex> lock(mu);
  if (!base[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) return cuda_fail(h, e, "cudaGetSymbolAddress(g_noalloc_scratch)");
    base[dev] = static_cast<unsigned char*>(p);
  }
  *out = base[dev];
  return MTP_OK;
}

}  // namespace

extern "C" {

int mtp_compute_device_noalloc(mtp_handle* h, int natoms, int stride, const int* d_itypes, const double* d_rijs,
                               const int* d_js, const int* d_jtypes, const int* d_counts, double* d_energy,
                               double* d_forces, double* d_virial) {
  if (!h) return MTP_E_INVALID;
  if (natoms < 0 || stride <= 0) return fail(h, MTP_E_INVALID, "natoms must be >= 0 and nbr_stride > 0");
  if (natoms > MTP_NOALLOC_MAX_ATOMS)
    return fail(h, MTP_E_CAPACITY, "natoms " + std::to_string(natoms) + " exceeds the allocation-free limit of " +
                                        std::to_string(MTP_NOALLOC_MAX_ATOMS) + " atoms");
  if (static_cast<long long>(natoms) * stride > MTP_NOALLOC_MAX_SLOTS)
    return fail(h, MTP_E_CAPACITY, "natoms * nbr_stride exceeds the allocation-free limit of " +
                                        std::to_string(MTP_NOALLOC_MAX_SLOTS) + " neighbour slots");
  if (stride > h->max_nbr) return fail(h, MTP_E_CAPACITY, "nbr_stride exceeds max_nbr");
  if (natoms > 0 && (!d_itypes || !d_rijs || !d_js || !d_jtypes || !d_forces || !d_energy || !d_virial))
    return fail(h, MTP_E_INVALID, "null pointer");
  unsigned char* base = nullptr;
  int st = noalloc_base(h, &base);
  if (st != MTP_OK) return st;
  const bool fp64 = h->precision == MTP_PRECISION_FP64;

  // launch shape within the handle's request whose programs are on the device;
  // the value space must fit in shared memory (its global-memory form would need
  // an allocation)
  std::vector<Shape> shapes;
  st = shared_shapes(h, natoms, stride, fp64, &shapes);
  if (st != MTP_OK) return st;
  const DeviceSchedule* ds = nullptr;
  const Shape shape = best_uploaded_shape(h, shapes, fp64, &ds);
  if (!ds)
    return fail(h, MTP_E_CAPACITY,
                "no uploaded schedule gives a shared-memory launch within the handle's launch limits (either the "
                "value space of this basis does not fit in shared memory, which the allocation-free path cannot "
                "replace by global memory, or no allocating call has uploaded a schedule for these limits yet)");

  double* grad = reinterpret_cast<double*>(base + kNoAlloc.grad);
  double* energy = reinterpret_cast<double*>(base + kNoAlloc.energy);
  double* wown = reinterpret_cast<double*>(base + kNoAlloc.wown);
  int* in_cnt = reinterpret_cast<int*>(base + kNoAlloc.in_cnt);
  int* in_ptr = reinterpret_cast<int*>(base + kNoAlloc.in_ptr);
  int* in_slot = reinterpret_cast<int*>(base + kNoAlloc.in_slot);
  int* blk = reinterpret_cast<int*>(base + kNoAlloc.blk);
  double* partials = reinterpret_cast<double*>(base + kNoAlloc.partials);
  double* tot = reinterpret_cast<double*>(base + kNoAlloc.tot);

  // The array keeps the previous call's contents.  The incoming-slot counters
  // must start at zero (launch_incoming clears them first) and the totals' counter
  // does (it ends every launch at zero);
  // every other piece is fully rewritten before it is read: each slot's
  // gradient (zero for skipped slots), each site energy and per-atom virial,
  // the scan blocks, the partials and the totals.
  DevModel md = make_model(h, *ds);
  DevIO io{};
  io.natoms = natoms;
  io.nbr_stride = stride;
  io.n_pad = stride;
  io.itypes = d_itypes;
  io.rijs = d_rijs;
  io.jtypes = d_jtypes;
  io.counts = d_counts;
  io.site_energy = energy;
  io.pair_grad = grad;
  io.err = h->d_err;
  io.vscratch = nullptr;
  MTP_CUDA(h, launch_incoming(natoms, stride, d_js, d_jtypes, d_counts, in_cnt, in_ptr, in_slot, blk, false, h->stream));
  MTP_CUDA(h, launch_eval(md, io, shape.fit, shape.lanes, launch_blocks(h, shape, natoms), fp64, false, shape.A,
                          h->stream));
  MTP_CUDA(h, launch_force_gather(natoms, stride, d_rijs, d_counts, grad, in_ptr, in_slot, true, d_forces, wown, nullptr,
                                  h->stream));
  st = write_totals(h, natoms, energy, wown, partials, tot, d_energy, d_virial);
  if (st != MTP_OK) return st;
  h->calls++;
  return MTP_OK;
}

}  // extern "C"
