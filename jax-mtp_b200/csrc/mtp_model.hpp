// mtp_model.hpp - host-side potential tables and the contraction schedule.
//
// The potential is the MLIP .mtp file the reference reads with read_mtp
// (motep_original_files/mtp.py:31-70).  The schedule turns its
// alpha_index_times list (m[i3] += mult * m[i1] * m[i2], conversion.py:95-102)
// into lane programs a CUDA block executes without atomics:
//
//   * forward: one pass per tree depth; each lane owns whole target moments
//     and accumulates their products in a register;
//   * reverse (dE/dm): the adjoint of every product is gathered per source
//     moment (dm[s] += mult * dm[t] * m[other]); long source lists are split
//     into chunks that write partial slots, summed in a fixed order by a
//     following combine pass.
//
// Every pass is a dense [steps][lanes] array of 8-byte entries so a warp
// reads its entries with one coalesced 256-byte load per step:
//
//   x = a | b << 16                     operand slots of the product
//   y = mult | op << 14 | dst << 16     integer multiplicity (< 2^14), flush
//                                       op (none/store/add), flush slot
//
// Steps are padded to a multiple of kStepAlign with no-op entries (operands
// the constant-zero slot, y = 0), and kStepAlign no-op rows follow the last
// pass, so a lane may request the kStepAlign rows after any step without a
// bounds test.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

namespace mtp {

constexpr int kMaxR = 8;       // radial functions supported by the kernels
constexpr int kMaxK = 16;      // Chebyshev terms supported by the kernels
constexpr int kMaxDegree = 12; // monomial degree supported by the kernels
constexpr int kMaxPasses = 16;
constexpr int kStepAlign = 4;  // pass steps are a multiple of this; as many no-op rows end the program
constexpr int kMaxGroupWarps = 16;  // warps of the largest block, which the force phase may group on one neighbour chunk
constexpr int kMaxChains = (kMaxDegree + 1) * (kMaxDegree + 2) / 2;
constexpr int kMaxRunOffsets = 36;  // 2 + 3 + 5 + 9 + 17: offsets of the cuts into 1, 2, 4, 8 and 16 runs

struct Potential {
  std::string version, potential_name, potential_tag, radial_basis_type;
  double scaling = 1.0, min_dist = 0.0, max_dist = 0.0;
  int S = 0, R = 0, K = 0, M = 0, B = 0, T = 0, Sa = 0;
  std::vector<double> radial;   // [S][S][R][K]
  std::vector<int> basic;       // [B][4] (mu, a, b, c)
  std::vector<int> times;       // [T][4] (i1, i2, mult, i3)
  std::vector<int> mapping;     // [Sa]
  std::vector<double> species;  // [S]
  std::vector<double> moment;   // [Sa]
};

// Parse .mtp text; returns false and sets err on malformed input.
bool parse_mtp_text(const std::string& text, Potential& out, std::string& err);
bool parse_mtp_file(const std::string& path, Potential& out, std::string& err);

// Program entry ops.
enum : uint32_t { kOpNone = 0, kOpStore = 1, kOpAdd = 2 };
// Fields of the second entry word.
constexpr uint32_t kMultMask = 0x3FFFu;
constexpr int kOpShift = 14;
constexpr int kDstShift = 16;

struct Pass {
  int offset = 0;   // first entry (index into Schedule::entries)
  int steps = 0;    // entries per lane (a multiple of kStepAlign)
  // steps each warp of the block runs: its longest lane's program rounded up
  // to kStepAlign (the rows after that are no-ops for all of its lanes)
  std::vector<int> wsteps;
};

struct Schedule {
  int lanes = 0;          // threads per block the programs were built for
  int width = 4;          // bytes per operand access the entry order was tuned for
  // Value-space layout (indices into the per-atom value array V):
  int v_m = 0;            // moments m[0..M)
  int v_dm = 0;           // adjoints dE/dm (dm_pos)
  int v_part = 0;         // partial sums of split lists
  int n_part = 0;
  int v_zero = 0;         // constant 0
  int v_one = 0;          // constant 1
  int v_size = 0;
  // monomials of the basic moments
  int D = 0;              // max degree
  int P = 0;              // distinct monomials
  std::vector<int> mono_abc;    // [P][4] (a, b, c, degree), degree descending
  std::vector<int> mono_k;      // [P][kMaxR] basic-moment index for each mu or -1
  // the same for the evaluation kernel: a | b << 4 | c << 8 | n << 12 |
  // (first of n entries in mono_list) << 16 with n = 1 + the monomial's
  // largest mu; mono_list holds basic-moment indices, 0xFFFF for none
  std::vector<int> mono_word, mono_list;
  // Force phase: the monomials are taken as Horner chains in u_z, one per pair
  // (a, b) with a + b <= D, b ascending and a descending; step k = 0 .. top =
  // D - a - b of a chain holds the monomial u_x^a u_y^b u_z^(top - k).
  // chain_mode >= 0: a level-structured basis (adjoint_layout) whose step k has
  // the radial functions mu < min(R, (k + chain_mode) / 2 + 1); -1: every step
  // has all R (adjoint 0 where the basis has no moment).  Chain slots are
  // steps in order, radial functions within a step, each chain padded to an
  // even length (16 bytes of its copy); n3_src[slot] is the adjoint position it copies, or -1.
  int chain_mode = -1;
  int n3_len = 0;
  std::vector<int> n3_src;      // [n3_len]
  // dE/dm of moment k lives at v_dm + dm_pos[k]; the adjoint region ends at v_part
  std::vector<int> dm_pos;
  // One word per chain, top | a << 4 | b << 8 | (first slot / 2) << 16, and the
  // list cut into W = 1, 2, 4, 8 and 16 runs of about equal cost (one per warp
  // of a group): run w of W is n3_words[n3_off[o + w] .. n3_off[o + w + 1])
  // with o = W - 1 + log2 W.
  std::vector<int> n3_words, n3_off;
  std::vector<int> dm_zero;     // adjoint positions that no pass stores and no seed sets (must read as 0)
  std::vector<int> zero_list;   // non-basic moments never written (must read as 0)
  std::vector<Pass> fwd, rev;   // passes in execution order
  std::vector<uint32_t> entries;  // pairs (x, y) per entry: 2 words; kStepAlign no-op rows at the end
  int max_depth = 0;
};

// Build the schedule for `lanes` threads per block whose operand accesses are
// `width` bytes (sizeof(real) x atoms per block; it sets the bank model the
// entry order is tuned for).  Fails (false, err) if the table does not have a
// write-before-read order, or exceeds index limits.
// With `programs` false everything but the programs is made (value-space size,
// tables, all checks of the table): enough to size a launch.
bool build_schedule(const Potential& pot, int lanes, Schedule& out, std::string& err, int width = 4,
                    bool programs = true);

// Local search over a built schedule against shared-memory bank conflicts:
// an entry whose bank key sets a gather's wavefront count trades steps with
// another entry of the same job (the flush stays at the job's last step), or
// in a forward pass its two operands trade places, whenever that lowers the
// wavefronts of both steps (bank model of build_schedule's `width`).  The
// sums are unchanged up to their order; candidates come from a fixed-seed
// generator, so the result is a pure function of the schedule.
void refine_schedule(Schedule& s);

// Execute the schedule for one atom on the host (bit-for-bit the device
// arithmetic order, in double): V must have v_size entries with basic moments
// in V[v_m .. v_m + B) set.  Fills moments, adjoints (seeded with moment
// coefficients), and returns sum_alpha theta_alpha m[map_alpha].
double emulate_schedule(const Potential& pot, const Schedule& s, std::vector<double>& V);

// Position of every moment's adjoint within the adjoint region (dm_pos,
// distinct); returns Schedule::chain_mode: o >= 0 if the basis is
// level-structured with that offset, that is, its basic moments (mu, a, b, c)
// are those with a + b + c <= D and mu < min(R, (D - a - b - c + o) / 2 + 1)
// (the MLIP templates up to level 24: o = 0; 26 and 28: o = 1 and 2, with six
// radial functions), else -1.  On such a basis the basic moments' adjoints
// take their force-phase chain slots as positions (each chain padded to an even
// length) and the others follow, so the copy into chain slots is a
// copy in a row; otherwise dm_pos[k] = k.
int adjoint_layout(const Potential& pot, std::vector<int>& dm_pos);

// Seeds of the reverse pass: unique moments of the mapping with summed theta.
void seed_list(const Potential& pot, std::vector<int>& idx, std::vector<double>& val);

}  // namespace mtp
