// Row form of the x / z pass (d = 2, 3, 5, 7): the launcher's view.
//
// The one-at-a-time passes carry the whole tableau through the program and
// rewrite it at every random measurement: n measurements of 2n x 2n residues
// each, one behind the other.  But a generator's column goes through the
// gates independently of every other column, and only the rows that a later
// measurement (or RESET, or N1) reads are ever needed.  So:
//   raw pass   : the gates of the whole program first, each CTA a few column
//                words of all qudits, layer by layer (layers of gates on
//                disjoint qudits, built by the host).  A measurement dumps its
//                row x_q over the 2n initial generators (S: the stabilizer
//                half, T: the destabilizer half) and puts the generator Z_q
//                that it leaves in the tableau into a column of its own (K
//                columns), whose entries later rows need;
//   chain pass : the measurements in order on those rows alone.  A random one
//                (S_j != 0, pivot p its first generator, e = S_j[p]^-1) adds
//                a F to every later row, F = -e S_j | -e T_j without p and
//                a = S_i[p], then sets T_i[p] = e a and S_i[p] = the raw entry
//                of row i in measurement j's K column: the rank-1 update of
//                the tableau, on the rows that are still needed;
//   extra pass : RESET's z_q rows and the N1 rows (stabilizer half only, which
//                is all the phase pass reads) through the same updates, in
//                parallel over rows.
// Phases.  Odd d: with X^x Z^z = omega^(-xz/2) W(x, z) products of commuting
// W add their phases, H and CNOT change none, and P and the Paulis add a
// linear form of the column: one more raw column (the constant, K lane 0) and
// a vector V of the stabilizers' phases, updated like a row.  d = 2: the rows
// are signed Pauli strings i^k prod X^S Z^T over the initial generators; k
// follows the gates word by word and the updates row by row, and V holds the
// stabilizers' signs.  The trace written is that of trace_bits.cuh (d = 2, the
// destabilizer half of factor rows zero) or of trace_u8.cuh (odd d, rows
// packed) over the stabilizer half, with the same pivots, factors and phases:
// no record depends on the destabilizers' deltas.  The row form's phase pass
// replays it, for d = 2 the programs without N1 before their last measurement
// (the others keep the passes that read the coin pass's masks).
#pragma once
#include <cstddef>
#include <cuda_runtime.h>

#include "common.cuh"

namespace sdim {

// A row's element holds 32 generators' residues in bit planes: one word (d =
// 2), two (d = 3, planes3.cuh), three padded to four (d = 5, 7).
constexpr int kRowLanes = 32;
__host__ __device__ constexpr int row_elem_bytes(int d) { return d == 2 ? 4 : d == 3 ? 8 : 16; }
__host__ __device__ constexpr bool row_dim(int d) { return d == 2 || d == 3 || d == 5 || d == 7; }
__host__ __device__ inline int row_elems(int n) { return (n + kRowLanes - 1) / kRowLanes; }

// Measurements of one panel of the chain pass: a lane each, and one for the
// stabilizers' phases.
constexpr int kRowPanel = 31;
// Flags of a row program's op (above its qudit and target, 11 bits each).
constexpr uint32_t kRopH = 1u << 22, kRopHInv = 1u << 23, kRopP = 1u << 24, kRopPInv = 1u << 25, kRopC = 1u << 26,
                   kRopCInv = 1u << 27;
constexpr uint32_t kRopM = 1u << 28;      // M or RESET
constexpr uint32_t kRopReset = 1u << 29;  // RESET
constexpr uint32_t kRopN = 1u << 30;      // N1 rows follow
constexpr uint32_t kRopK = 1u << 31;      // changes the constants
// Most warps of a chain-pass CTA, and those of an extra-pass CTA.
constexpr int kRowWarps = 16;

// Row program, built by the host encoder (abi.cu: append_rows), in the blob:
//   ops[i] = {qudit | target << 11 | flags (kRop...), y, z, w}, layer by layer.
//     y = a measurement's ordinal, else what a P or Pauli adds to the constants
//     (sign exponents for d = 2) of x_q and, << 3, of z_q; z = 1 + extra row of
//     a RESET's z_q, else z (w of a measurement) = 1 + the first of the two
//     extra rows of an N1 on the qudit that follows with no op on it between,
//     w of a CNOT the same for its target.  An N1 of its own has flag kRopN
//     alone;
//   lay[l] .. lay[l + 1]: the ops of layer l (pairwise disjoint qudits);
//   minfo[m] = N1 ordinals before measurement m | RESET << 31;
//   xinfo[r] = {measurements whose updates extra row r takes, kind << 30 |
//     index}: kind 0 the z_q row of RESET `index`, 1 (2) the x_q (z_q) row of
//     N1 ordinal `index`.
struct RowProgram {
  int64_t ops_off = -1, lay_off = -1, minfo_off = -1, xinfo_off = -1, nhdr_off = -1;  // uint2 words of the blob
  int nops = 0, nlayers = 0, nx = 0;
  int nk = 0;  // measurements with a K column
  int nn1 = 0;           // N1 ordinals before the last measurement
  double fires = 0.0;    // expected number of them that any of 32 shots fires
};

struct RowDesc {
  const uint4* ops;
  const uint32_t* lay;
  const uint32_t* minfo;
  const uint2* xinfo;
  uint8_t* raw;    // nm rows: S[E] T[E] K[EK]
  uint8_t* xraw;   // nx rows: S[E] K[EK]
  uint8_t* kpart;  // d = 2: sign exponents per measurement and word, [nm][E]
  uint8_t* ksign;  // d = 2: sign exponents gathered from the updates, [nm]
  uint8_t* nz;     // set by the updates: the row has an S entry, [nm]
  uint8_t* vg;     // V for the other CTAs of a cluster, [2][E]
  uint8_t* opf;    // factor rows F of the random measurements, [..][2 E]
  int4* opm;       // their {pivot, exponent | commute parity << 8, ordinal, 1 + last op of the panel
                   // before it with its pivot (0: none) | no later one has it << 6}
  int* pop;        // first op of each panel, [panels + 1]
  uint32_t* opw;   // odd d: each panel's matrix W, [panels][32][8] words (rows_kernels.cuh: PanelOps::Wt)
  uint4* mhdr;     // the trace
  uint8_t* mrow;   // rows of rowb bytes, two per measurement
  uint8_t* nrow;   // rows of rowb bytes, two per N1 ordinal
  int n, d, nops, nlayers, nm, nx, nk;
  int E, EK;
  int rowb;         // bytes of a trace row
  int tile_begin;   // first raw-pass CTA of this program
  int x_begin;      // first extra-pass CTA of this program
};

struct RowBytes {
  size_t raw, xraw, kpart, ksign, nz, vg, opf, opm, pop, opw, total;  // offsets, and the total
};

inline RowBytes row_bytes(int n, int d, int nm, int nx, int nk) {
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t E = row_elems(n), EK = (nk + (d == 2 ? 0 : 1) + kRowLanes - 1) / kRowLanes;
  const size_t eb = row_elem_bytes(d);
  RowBytes b;
  b.raw = 0;
  b.xraw = b.raw + up((size_t)nm * (2 * E + EK) * eb);
  b.kpart = b.xraw + up((size_t)nx * (E + EK) * eb);
  b.ksign = b.kpart + up(d == 2 ? (size_t)nm * E : 0);
  b.nz = b.ksign + up(d == 2 ? (size_t)nm : 0);
  b.vg = b.nz + up((size_t)nm);
  b.opf = b.vg + up(2 * E * eb);
  b.opm = b.opf + up((size_t)nm * 2 * E * eb);
  b.pop = b.opm + up((size_t)nm * sizeof(int4));
  b.opw = b.pop + up(((size_t)nm / kRowPanel + 2) * sizeof(int));
  b.total = b.opw + up(d == 2 ? 0 : ((size_t)nm / kRowPanel + 1) * 1024);
  return b;
}

// Column words (units) of a program's raw pass: d = 2 pairs the S and T words
// of a position, for the signs.
inline int row_units(int n, int d, int nk) {
  const int E = row_elems(n), EK = (nk + (d == 2 ? 0 : 1) + kRowLanes - 1) / kRowLanes;
  return (d == 2 ? E : 2 * E) + EK;
}

// How the chain pass spreads a row of E elements: its S (and T) elements per
// lane, 16 added when several warps share a row.  One warp with whole rows
// needs no barrier a step, but walks all its elements in each: up to four for
// d = 2 (128 qubits: 122 us, with a warp per element 135), two for odd d (128
// qudits of d = 5: 197 us with four a lane, 184 with a warp per element; 100
// qutrits 145 and 135).  Then two a lane (256 qudits of d = 5: 359 us, one 368;
// 500: 706, one 744) and four past 24 (1,000 of d = 7: 1677 us, two 1767).
// Programs of one slice are one launch: kRowSliceSmall, a warp per element of up
// to four, and kRowSliceMid, two a lane of up to eight, are apart from wider
// rows, since a larger group gets smaller clusters.
constexpr int kRowSliceSmall = 16 + 32 + 1, kRowSliceMid = 16 + 32 + 2;
inline int row_slice(int E, int d) {
  return E <= 1 ? 1 : E <= 2 ? 2 : E <= 4 ? (d == 2 ? 4 : kRowSliceSmall) : E <= 8 ? kRowSliceMid : E <= 24 ? 18 : 20;
}

// A program in the row form's phase pass.
struct RowPhaseDesc {
  CircuitDesc c;
  const uint4* mhdr;
  const uint8_t* mrow;  // rowb bytes each: factor row, z_q row of a RESET
  const uint8_t* nrow;  // odd d: rowb bytes each: x_q, z_q at an N1
  const uint2* nhdr;    // odd d: N1 (coin threshold, opcode)
  int nm, nn1, E, rowb;
  int pitch;        // bytes of a measurement's rows that a window stages: both, or the factor row alone
  int lg;           // a shot is 2^lg lanes
  int block_begin;  // first CTA (4 warps) of this program
};
// Elements a lane of the phase pass holds: one while the launch's warps stay
// below a few per scheduler (the chain of a measurement bounds it), up to four
// for many shots (the issue of the per-lane overhead bounds it).
inline int row_phase_lg(int E, int wpl) {
  int lg = 0;
  while ((wpl << lg) < E && lg < 5) ++lg;
  return lg;
}
inline size_t row_phase_smem(int pitch) { return (size_t)2 * 32 * (16 + pitch) + 4 * 2 * 32 * 36; }
// Bytes of a packed trace row over E elements (a multiple of 16).
inline int row_trace_bytes(int E, int d) { return (E * row_elem_bytes(d) + 15) / 16 * 16; }

// The frame pass of one program (k_frame.cu has the frame rules).
struct RowFrameDesc {
  const uint4* ops;      // its row program
  const uint32_t* lay;
  const uint2* xinfo;
  const uint2* nhdr;     // odd d: N1 (coin threshold, opcode)
  const uint8_t* ref;    // records of the reference shot
  uint8_t* out;          // nshots x nm records
  uint8_t* words;        // frame words of the records: nm elements per 32 shots
  const uint2* masks;    // d = 2: the coin pass's fire masks, mshots shots a chunk, from shot mrel on
  unsigned long long seed;
  long long shot0;       // stream index of the first shot, below 2^32
  long long mshots, mrel;
  int nlayers, n, nm, nshots;
  int nused;   // N1 ordinals before the last measurement
  int nchunk;  // d = 2: chunks of 32 of them
  int cap;     // d = 2: entries of a warp for fired ordinals
};

// The launchers of one d (k_rows_<d>.cu).
struct RowOps {
  cudaError_t (*set_smem)(int optin);
  size_t (*raw_smem)(int n, int lg);
  size_t (*chain_smem)(int n, int block);
  size_t (*extra_smem)(int n);
  int (*extra_per_cta)(int n);
  // raw pass: `tiles` CTAs of `block` threads, each 2^lg units of one program
  void (*raw)(int tiles, int block, int lg, size_t smem, cudaStream_t s, const RowDesc* descs, int nd);
  // chain pass: programs of one row_slice, a cluster of `ctas` CTAs (1, 2, 4 or
  // 8) of `block` threads per program; rawt > 0: with the raw pass in front,
  // 2^lg units a CTA on rawt threads (smem at least raw_smem)
  cudaError_t (*chain)(int slice, int ctas, int block, int rawt, int lg, size_t smem, cudaStream_t s, const RowDesc* descs, int nd);
  // extra pass: `ctas` CTAs, extra_per_cta rows each (close: follow.cuh)
  void (*extra)(bool close, int ctas, size_t smem, cudaStream_t s, const RowDesc* descs, int nd);
  // phase pass: `blocks` CTAs of 128 threads, wpl (1, 2 or 4) elements a lane
  void (*phase)(bool close, int wpl, int blocks, size_t smem, cudaStream_t s, const RowPhaseDesc* descs, int nd);
  // frame pass: `blocks` CTAs of `warps` (1 to 4) warps, 32 shots each
  size_t (*frame_smem)(const RowFrameDesc& f, int warps);
  void (*frame)(int blocks, int warps, size_t smem, cudaStream_t s, const RowFrameDesc& f);
  // the records from the frame pass's words and the reference shot's records
  void (*frame_out)(cudaStream_t s, const RowFrameDesc& f);
};
const RowOps& row_ops_2();
const RowOps& row_ops_3();
const RowOps& row_ops_5();
const RowOps& row_ops_7();
inline const RowOps& row_ops(int d) { return d == 2 ? row_ops_2() : d == 3 ? row_ops_3() : d == 5 ? row_ops_5() : row_ops_7(); }

}  // namespace sdim
