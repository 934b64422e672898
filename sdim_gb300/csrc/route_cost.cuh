// Estimated times of a program's routes, from which a run chooses which of its
// programs take the row form (rows.cuh).
//
// The row form's chain finishes a lone program sooner than the shot-group
// engines and the tableau passes, but it is a launch of several kernels with a
// CTA (or a cluster) per program, and it carries every row through every panel
// before it: work that grows with the square of the measurements.  Which route
// is the faster one therefore turns on how many programs share the device, on
// the shots, and on measurements against qudits.  Measured on GB300, row form
// and the other route (us):
//     1 x   49 qubits (a memory), 145 measurements, 1 shot 102    505
//     1 x    3 qudits of d = 7, 2,000 measurements       3969   5193
//     1 x    3 qudits of d = 7, 20,000 measurements    170496  51700
//   300 x   31 qudits of d = 7, 200 measurements, 1 shot  587    848
//   300 x    3 qudits of d = 7, 2,000 measurements      49678   5104
//  4000 x   31 qubits, 8 measurements, 1 shot             846     37
//  4000 x   31 qubits, 31 measurements, 200 shots         979   1685
// The constants below are fitted to 6,210 such pairs: d = 2, 3, 7, 3 to 400
// qudits, 3 to 4,000 measurements, with noise and without, 1 to 2,000 shots, 1 to
// 4,000 programs a run.  Four fifths of the estimates are within 30% of the
// measured time, and the choice (choose_row_form) costs at most 2% over the faster
// of the two in 95% of the pairs, 1.23 times in 99% and 1.8 times at worst.  (The row
// form for all of them: slower in 20% of the pairs, up to 29 times; for none: slower
// in 77%, up to 52 times.)
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>

#include "rows.cuh"

namespace sdim {

struct RouteShape {
  int n, d, nmeas, nn1, gates;  // gates: the other device instructions
  int layers, nx;               // of the row program
  long long shots;
  bool trace;  // without the row form: the trace engine's tableau pass, else the shot groups
};

// Microseconds of a program alone (latency), of one SM's time that it takes among
// many (work), and of its descriptors (host).
struct RouteCost {
  double latency, work, host;
};

// Replay of one shot, d = 2: much the same on both routes.
inline double replay_us_d2(const RouteShape& p) { return 0.00016 * (p.nmeas * (1 + p.n / 64.0) + p.nn1); }

// Row form, programs of its launch sharing the device.
inline RouteCost row_cost(const RouteShape& p, long long programs, int num_sms) {
  const double nm = p.nmeas, full = std::floor(nm / kRowPanel);
  const bool odd = p.d != 2;
  const int E = row_elems(p.n);
  int group = 1;  // lanes of a row (d = 2), as row_group
  while (group < E && group < 32) group <<= 1;
  // the launch shape (plan_row_group), and the warps that a program's row updates have
  int ctas = 1;
  if (p.nmeas > 2 * kRowPanel)
    for (int k = 8; k > 1 && ctas == 1; k >>= 1)
      if (k * programs <= num_sms) ctas = k;
  const bool batch = ctas * programs > num_sms;
  const int block = !batch || E > 8 ? 32 * kRowWarps : E > 4 ? 256 : 128;
  const double warps = ctas > 1 ? (ctas - 1) * kRowWarps : block / 32;
  // a row through a panel's updates: a warp each for odd d, a lane group for d = 2
  const double updates = full * nm - 0.5 * kRowPanel * full * (full + 1);
  const double task = odd ? 1.8 * updates : (group == 1 ? 3.5 : 2.5) * updates * group / 32;
  RouteCost c;
  c.latency = 20 + (p.nx ? 6 : 0) + 0.27 * p.layers + (odd ? 0.71 : 0.50) * nm + task / warps;
  c.work = (0.48 * p.layers + 0.71 * nm) * block / (32.0 * kRowWarps) + 0.09 * task + (odd ? 0.11 : 0.003) * p.nx;
  if (!batch) c.work = std::min(c.work, c.latency);  // an SM to itself
  c.work += (double)p.shots * (odd ? 0.003 + (p.d == 3 ? 0.00125 : 0.0017) * std::max(1.0, 0.35 * E) * nm + 0.0004 * p.nn1
                                   : replay_us_d2(p));
  c.host = 0.17;
  return c;
}

// The program's route without the row form.
inline RouteCost other_cost(const RouteShape& p) {
  const double n = p.n, nm = p.nmeas, shots = (double)p.shots;
  const bool odd = p.d != 2;
  RouteCost c{0.0, 0.0, 0.0};
  if (!p.trace) {  // one warp per 32 shots, each with a tableau of its own
    c.latency = 13 + p.gates * (odd ? 0.012 * n : 0.26) + p.nn1 * (odd ? 0.74 : 0.25) +
                nm * (odd ? 2.4 + 0.0008 * n * n : 0.66 + 0.011 * n);
    c.work = std::ceil(shots / 32) * c.latency * (odd ? 0.074 : 0.041) * (1 + 2e-4 * n * n);
  } else {  // one CTA, pair or cluster for the x / z pass, then a replay
    const double chain = p.gates * 0.17 + nm * (odd ? 3.2 + 0.016 * n : 2.3 + 0.0047 * n) + p.nn1 * (odd ? 2.0 : 0.0);
    const double part = odd ? (p.d == 3 ? 0.12 : 0.23) * (1 + 3.2e-5 * n * n) : 0.53 * (1 + 0.0012 * n);
    c.latency = 26 + chain;
    c.host = 0.09;
    c.work = chain * std::min(1.0, part) +
             shots * (odd ? 0.001 + std::max(0.0016, 3.2e-5 * n) * nm + 0.0018 * p.nn1 : replay_us_d2(p));
  }
  return c;
}

// Which programs of a run take the row form (programs[i]: how many share p[i]'s
// launch).  A run's time is estimated as the longest latency and the work over
// all SMs, added as squares, the descriptors, and kGroupLaunch where shot groups
// run (their work queue's reset, descriptors and launches).  The row form is for
// all or for none (none where that is 5% shorter), unless a split -- for a bound
// on the latency, for every program the route of less work and descriptors within
// the bound -- is half as long as either: engines beside one another take each
// other's SMs, which the estimate leaves out.  Of 60 mixed batches (12 to 2,500
// programs, 4 to 1,024 qudits, 1 to 600 shots) splits that were estimated up to a
// third shorter than the row form for all took up to 2.2 times as long, and the
// row form for all up to 29 times less than none.
constexpr double kGroupLaunch = 4.0;

struct RunCost {  // of the programs' chosen routes
  double longest = 0.0, work = 0.0, host = 0.0;
  bool groups = false;
  void add(const RouteCost& c) {
    longest = std::max(longest, c.latency);
    work += c.work;
    host += c.host;
  }
  double time(int num_sms) const {
    const double w = work / num_sms;
    return std::sqrt(longest * longest + w * w) + host + (groups ? kGroupLaunch : 0.0);
  }
};

// A run of one program.
inline bool row_form_alone(const RouteShape& p, int num_sms) {
  RunCost row, other;
  row.add(row_cost(p, 1, num_sms));
  other.add(other_cost(p));
  other.groups = !p.trace;
  return other.time(num_sms) >= 0.95 * row.time(num_sms);
}

inline std::vector<char> choose_row_form(const std::vector<RouteShape>& p, const std::vector<long long>& programs,
                                         int num_sms) {
  const size_t k = p.size();
  std::vector<RouteCost> row(k), other(k);
  RunCost all, none, least;  // the row form for all, for none; the least of either
  double most = 0.0;
  for (size_t i = 0; i < k; ++i) {
    const RouteCost &r = row[i] = row_cost(p[i], programs[i], num_sms), &o = other[i] = other_cost(p[i]);
    all.add(r);
    none.add(o);
    none.groups |= !p[i].trace;
    least.add(RouteCost{std::min(r.latency, o.latency), std::min(r.work, o.work), std::min(r.host, o.host)});
    most = std::max(most, std::max(r.latency, o.latency));
  }
  const bool rows = none.time(num_sms) >= 0.95 * all.time(num_sms);
  std::vector<char> best(k, rows), take(k);
  double best_time = 0.5 * (rows ? all : none).time(num_sms);
  // (no split is shorter than `least`, none with a latency past `bound` than the bound)
  for (double bound = least.longest; least.time(num_sms) < best_time && bound < best_time; bound *= 1.3) {
    RunCost s;
    for (size_t i = 0; i < k; ++i) {
      const RouteCost &r = row[i], &o = other[i];
      const double more = (r.work - o.work) / num_sms + r.host - o.host;  // of the row form, in the run's time
      take[i] = o.latency > bound || (r.latency <= bound && more <= 0.0);
      s.add(take[i] ? r : o);
      s.groups |= !take[i] && !p[i].trace;
    }
    if (s.time(num_sms) < best_time) {
      best_time = s.time(num_sms);
      best = take;
    }
    if (bound >= most) break;
  }
  return best;
}

// The frame route: whether shots 1 .. nshots - 1 run on bit planes (k_rows_frame)
// or a byte per qudit and shot (k_frame_pass).  The planes' warps walk the layers
// two to twenty times sooner, but each holds all its N1 samples in shared memory:
// with thousands of ordinals a few warps an SM are left, and many shots take turn
// after turn.  Measured on GB300, planes and bytes (ms):
//   7 qudits of d = 7, 2,500 ordinals, 20,000 shots      1.54   2.25
//                                     100,000 shots      5.57   2.56
//   7 qubits, 60,000 ordinals of probability 0.001, 20,000 shots   16.5   41.2
//                                                  300,000 shots  144.9   95.4
//   7 qubits, 10,000 ordinals, 300,000 shots             7.95  15.73
//   100 qubits, 60,000 ordinals, 300,000 shots          39.3   95.3
// On 112 such pairs (d = 2, 3, 7, 7 and 100 qudits, 1,000 to 400,000 ordinals,
// 2,000 to 300,000 shots) the estimates below take the faster kernel every time.
struct FrameShape {
  int n, d, nmeas, used, layers;  // used: N1 ordinals before the last measurement
  long long ops;
  double fires;  // expected number of them that any of 32 shots fires
  long long shots;
};

inline double frame_turns(long long shots, int warps_per_sm, int num_sms) {
  return (double)shots / (32.0 * num_sms * warps_per_sm);
}

// Microseconds with that many warps resident on an SM.
inline double frame_planes_us(const FrameShape& f, int warps_per_sm, int num_sms) {
  const int held = std::min(warps_per_sm, 40);
  const double turns = frame_turns(f.shots, held, num_sms);
  const double a_turn = 20 + f.layers * (f.d == 2 ? 0.235 : f.d == 3 ? 0.28 : 0.37) + f.used * (f.d == 2 ? 0.02 : 0.027) +
                        (f.d == 2 ? 0.3 * f.fires : 0.0);
  return a_turn * std::max(1.0, turns) * (1 + 0.05 * held * std::min(1.0, turns));
}
inline double frame_bytes_us(const FrameShape& f, int warps_per_sm, int num_sms) {
  const int held = std::min(warps_per_sm, 32);
  const double turns = frame_turns(f.shots, held, num_sms);
  const double a_turn = f.ops * (f.d == 2 ? 0.28 : 0.46) + (f.d == 2 ? 1.5 : 3.4) * (f.n + f.nmeas);
  return a_turn * std::max(1.0, turns) * (1 + 0.004 * held * std::min(1.0, turns));
}

}  // namespace sdim
