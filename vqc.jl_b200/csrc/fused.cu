// The fused tile engine: apply!(::QCircuit, state) (generic.jl:26-31) and the
// reverse sweep of the circuit pullback (circuitdiff.jl:61-75) with many gates
// per HBM round trip.
//
// The reference runs one full pass over the state per gate.  Here a host
// planner groups the gates into *passes*.  A pass picks a set Q of M "tile"
// qubits (always including the lowest qubits, so every tile is made of
// contiguous runs of amplitudes); every CTA loads whole tiles (the 2^M
// amplitudes that share all non-tile bits) into shared memory, applies every
// gate of the pass to them, and writes them back: one HBM read + write per
// pass instead of per gate.
//   * a gate whose matrix acts on one or two target qubits (after stripping
//     control qubits, read off the matrix) works on 4 tile bits ("register
//     bits"): each thread owns the 16 amplitudes spanning them, in registers
//     (compiled passes) or at its own places of the tile (interpreted ones),
//     and the pass is cut into *stages*, each with one register-bit set;
//     between stages the amplitudes change owners through shared memory
//     (XOR-swizzled, so the 16-byte / 8-byte accesses are free of bank
//     conflicts);
//   * controls on thread bits are tested once per op, on register bits they
//     select addresses, on non-tile qubits they are tested once per tile;
//   * diagonal gates (CZ, CPHASE, ...) act on any qubits, tile or not;
//   * consecutive one-qubit gates on the same qubit are merged into one 2x2.
// In the reverse sweep (ADJ) each op applies U^dagger to both the cotangent
// and the state and accumulates the reduced matrix
//   A[a][b] = sum conj(lambda_a) psi_b   over the op's target pairs
// (per thread over its 8 pairs in the state's precision, then in FP64 across
// the warp, the CTA and the grid, in a fixed order); the host contracts A
// with D_j = B^dagger dB/dtheta_j of each parameter j of the (merged) block.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <optional>
#include <mutex>
#include <set>
#include <thread>
#include <tuple>
#include <type_traits>

#include "engine.h"
#include "subspace.cuh"
#include "tile_f32.cuh"
#include "tile_kernels.cuh"
#include "tile_plan.cuh"

namespace vqc {

// The tile kernels themselves live in tile_kernels_impl.cuh (tile_inst_*.cu).

// Sums the per-CTA partials of many passes over their grids in a fixed order:
// one item per pass (blockIdx.y), block x = slot (defined with the serving
// support below).
__global__ void __launch_bounds__(256) k_reduce_slots_batch(const RedItem* __restrict__ items);

// ----------------------------------------------------------------------------- host planner
// A gate in planner form: one op, or "standalone" (kept as a GateSpec).
struct PItem {
  bool standalone = false;
  int gate = -1;  // index in the caller's gate list
  FOp op;
};

static inline int popc64(uint64_t x) { return __builtin_popcountll(x); }

// Reads a gate's structure off its (sorted, possibly daggered) matrix.
// Returns false when the gate cannot be fused (3+ target qubits).
static bool to_fop(const GateSpec& g, FOp& f) {
  const int k = g.k, d = 1 << k;
  f = FOp();
  for (int b = 0; b < k; ++b) f.qubits |= 1ull << g.sp[b];
  if (g.ns == 0) {  // identity
    f.kind = kOpDiag;
    f.nd = 0;
    f.mat = {cd(1)};
    return true;
  }
  if (k == 1) {  // one-qubit gates (diagonal ones too) run in registers and merge
    f.kind = kOpU1;
    f.tq[0] = g.sp[0];
    f.mat = g.U;
    return true;
  }
  if (g.mode == kDiag) {
    f.kind = kOpDiag;
    f.nd = k;
    for (int b = 0; b < k; ++b) f.dq[b] = g.sp[b];
    f.mat.assign(d, cd(0));
    for (int j = 0; j < d; ++j) f.mat[j] = g.U[(size_t)j * d + j];
    return true;
  }
  // controls: bits constant over the active set
  int ctrl_bits = 0, cval_bits = 0;
  for (int b = 0; b < k; ++b) {
    bool all1 = true, all0 = true;
    for (int s = 0; s < g.ns; ++s) {
      if (g.S[s] >> b & 1)
        all0 = false;
      else
        all1 = false;
    }
    if (all1 || all0) {
      ctrl_bits |= 1 << b;
      if (all1) cval_bits |= 1 << b;
    }
  }
  int tb[5], nt = 0;
  for (int b = 0; b < k; ++b)
    if (!(ctrl_bits >> b & 1)) tb[nt++] = b;
  if (nt == 0 || nt > 2) return false;
  for (int b = 0; b < k; ++b)
    if (ctrl_bits >> b & 1) {
      f.cmask |= 1ull << g.sp[b];
      if (cval_bits >> b & 1) f.cval |= 1ull << g.sp[b];
    }
  f.kind = nt == 1 ? kOpU1 : kOpU2;
  for (int i = 0; i < nt; ++i) f.tq[i] = g.sp[tb[i]];
  const int dn = 1 << nt;
  f.mat.assign((size_t)dn * dn, cd(0));
  auto full = [&](int a) {  // target-subspace index -> gate index
    int j = cval_bits;
    for (int i = 0; i < nt; ++i)
      if (a >> i & 1) j |= 1 << tb[i];
    return j;
  };
  for (int a = 0; a < dn; ++a)
    for (int c = 0; c < dn; ++c) f.mat[(size_t)a * dn + c] = g.U[(size_t)full(a) * d + full(c)];
  return true;
}

// Restriction of a full sorted-order k-qubit matrix to the op's target subspace.
static Mat2 restrict_to(const GateSpec& g, const FOp& f, const Mat& D) {
  const int k = g.k, d = 1 << k;
  int cval_bits = 0, tb[2], nt = 0;
  for (int b = 0; b < k; ++b) {
    const uint64_t q = 1ull << g.sp[b];
    if (f.cmask & q) {
      if (f.cval & q) cval_bits |= 1 << b;
    } else {
      tb[nt++] = b;
    }
  }
  const int dn = 1 << nt;
  Mat2 R((size_t)dn * dn);
  auto full = [&](int a) {
    int j = cval_bits;
    for (int i = 0; i < nt; ++i)
      if (a >> i & 1) j |= 1 << tb[i];
    return j;
  };
  for (int a = 0; a < dn; ++a)
    for (int c = 0; c < dn; ++c) R[(size_t)a * dn + c] = D[(size_t)full(a) * d + full(c)];
  return R;
}

template <class A, class B>
static Mat2 mat2_mul(const A& a, const B& b) {
  Mat2 c(4);
  for (int r = 0; r < 2; ++r)
    for (int k = 0; k < 2; ++k) c[r * 2 + k] = a[r * 2] * b[k] + a[r * 2 + 1] * b[2 + k];
  return c;
}
template <class A>
static Mat2 mat2_dag(const A& a) {
  return {std::conj(a[0]), std::conj(a[2]), std::conj(a[1]), std::conj(a[3])};
}

struct PlanStage {
  std::vector<int> rs;   // tile-bit indices (ascending)
  std::vector<int> ops;  // indices into PlanPass::ops
};
struct PlanPass {
  bool standalone = false;
  int gate = -1;                 // standalone: the caller's gate
  std::vector<int> tile_q;       // M global qubits, ascending
  std::vector<FOp> ops;
  std::vector<PlanStage> stages;
  int nslots = 0;
};

static void tile_bits(const PlanPass& p, int (&tbit)[64]) {
  for (int& b : tbit) b = -1;
  for (int b = 0; b < (int)p.tile_q.size(); ++b) tbit[p.tile_q[b]] = b;
}

struct TileConfig {
  int M;      // tile bits
  int clow;   // always-resident low qubits
};

static TileConfig tile_config(int dtype, int n) {
  // 2^12 FP32 or 2^11 FP64 amplitudes per tile (32 KiB per state), smaller
  // tiles for smaller states; the lowest 4 (FP32) / 3 (FP64) qubits are always
  // tile qubits so that a tile is made of 128-byte runs (11-qubit FP32 tiles
  // for the reverse sweep measured slower: more passes at the same pass cost;
  // 3 always-resident FP32 qubits give 10 % fewer passes at 1.4x the reverse
  // pass time, 11.6 vs 12.6 gradients/s at n = 26; 2^12 FP64
  // amplitudes, a tenth fewer passes: 9.67 against 9.72 ms for a 27-qubit
  // circuit, 3.66 against 3.65 ms for a 23-qubit gradient, and 128 KB of tiles)
  const int M = std::min(dtype == VQC_C64 ? 12 : 11, n);
  return {M, std::min(dtype == VQC_C64 ? 4 : 3, M)};
}
constexpr int kMinTileBits = 9;  // 32 threads x 16 amplitudes

// Greedy pass formation (see the file comment).  items are in execution order.
static void plan_passes(int n, const TileConfig& tc, bool adj, std::vector<PItem>& items, std::vector<PlanPass>& out) {
  const int M = tc.M;
  std::vector<char> done(items.size(), 0);
  size_t first = 0;
  while (true) {
    while (first < items.size() && done[first]) ++first;
    if (first >= items.size()) break;
    if (items[first].standalone) {
      PlanPass p;
      p.standalone = true;
      p.gate = items[first].gate;
      out.push_back(std::move(p));
      done[first] = 1;
      continue;
    }
    PlanPass p;
    uint64_t Q = 0;
    for (int q = 0; q < std::min(tc.clow, n); ++q) Q |= 1ull << q;
    uint64_t blocked = 0;
    std::vector<int> last_on(n, -1);  // last op index in p.ops touching qubit q
    for (size_t i = first; i < items.size(); ++i) {
      if (done[i]) continue;
      PItem& it = items[i];
      const uint64_t qs = it.op.qubits;
      if (it.standalone) {  // runs after this pass: its qubits stay blocked
        blocked |= qs;
        continue;
      }
      if (qs & blocked) {
        blocked |= qs;
        continue;
      }
      FOp& f = it.op;
      uint64_t need = 0;
      if (f.kind == kOpU1) need = 1ull << f.tq[0];
      if (f.kind == kOpU2) need = (1ull << f.tq[0]) | (1ull << f.tq[1]);
      const bool fits = popc64(Q | need) <= M;
      const bool slot_ok = (!(adj && f.acc) || p.nslots < kMaxSlots) && (int)p.ops.size() < kMaxOpsPerPass;
      if (!fits || !slot_ok) {
        blocked |= qs;
        continue;
      }
      Q |= need;
      done[i] = 1;
      // merge consecutive uncontrolled one-qubit ops on the same qubit
      if (f.kind == kOpU1 && f.cmask == 0) {
        const int prev = last_on[f.tq[0]];
        if (prev >= 0) {
          FOp& g = p.ops[prev];
          if (g.kind == kOpU1 && g.cmask == 0 && g.tq[0] == f.tq[0]) {
            // g applied first, then f: merged = f.mat * g.mat
            const Mat2 merged = mat2_mul(f.mat, g.mat);
            if (adj) {
              // g's gradients were taken at g's output side = f's input: move them
              // to the block input (f is applied after g, so D -> F^dag D F); in
              // the reverse sweep the op matrices are U^dagger: f.mat = U_f^dagger,
              // the block input lies after f, and D_g moves by conjugation with
              // f.mat^dagger
              const Mat2 Fd = mat2_dag(f.mat);
              for (PGrad& pg : g.grads) pg.D = mat2_mul(f.mat, mat2_mul(pg.D, Fd));
              for (PGrad& pg : f.grads) g.grads.push_back(std::move(pg));
              if (f.acc && !g.acc) {
                g.acc = true;
                ++p.nslots;
              }
            }
            g.mat = merged;
            continue;
          }
        }
      }
      if (adj && f.acc) ++p.nslots;
      p.ops.push_back(std::move(f));
      for (uint64_t m = qs; m; m &= m - 1) last_on[__builtin_ctzll(m)] = (int)p.ops.size() - 1;
    }
    // fill the tile with the lowest remaining qubits
    for (int q = 0; q < n && popc64(Q) < M; ++q) Q |= 1ull << q;
    for (int q = 0; q < n; ++q)
      if (Q >> q & 1) p.tile_q.push_back(q);
    out.push_back(std::move(p));
  }
}

// Phases deferred.  A 2x2 M = c U, U unitary with |m00| = |m11|, is a diag(1, p) T,
// a = m00, |p| = 1, T = [[1, x], [-conj(x), 1]], and T takes half the products of a
// general 2x2 (8 instead of 16 FMAs per pair of amplitudes); the tile passes are
// bound by their arithmetic.  The phase p stays behind as a pending diag(1, p) on
// the qubit and a as a factor g of the whole state.  A pending phase passes a
// control and a diagonal gate unchanged, turns another gate on its qubit into one
// with rotated off-diagonal entries, and is absorbed by the next uncontrolled
// one-qubit gate there; the last such gate (before the end of the circuit, or a
// gate outside the tile passes) takes its whole matrix and g, so no pass is added.
//
// The amplitudes in flight are the true ones times 1 / |g|, so |g| is bounded: the
// first deferred gate of a pass and every 8th after it (forward 16th, FP64 32nd) take
// the norm of g (real diagonal, 12 FMAs), and so does one that would take |g| out of
// a window, [1e-12, 1e12] (forward 1e-18, FP64 1e-60).  The gates are walked in the order they run, stage by
// stage: a stage runs every layer of its few register qubits, so in any other order
// (the planner's, 192 ops to a pass) the factors of one qubit pair's forty layers
// would meet before the gates meant to take them.  A deferred gate's factor is
// |cos| of a half angle, one half in the geometric mean: 2^-8 between two norms in
// the FP32 reverse sweep, which sums products of two such amplitudes, 2^-16 in the
// forward one (every 8th there: 64.0 against 63.2 ms for the 30-qubit circuit); the
// window is reached by chance less than twice in 10^5 such runs of random gates, by
// gates near X (RX(pi)) at once.
//
// Which form a gate takes depends on its place alone, not on its angle (but for
// the window, |m00| < kMinPivot and exact zeros), so that new angles reuse compiled
// passes.  T is a multiple of a unitary whatever |x|: a large x is as accurate as a
// small one.
//
// Only where the passes are compiled (states of 2^18 FP32, 2^23 FP64 amplitudes
// and more): the interpreted ones are bound by latency, and a CNOT that was a
// swap of two loads becomes a product (serving's reverse launches 66 -> 81 us).
// Measured: reverse pass 1,060 -> 957 us and forward 350 -> 325 us at 2^26 FP32,
// U3 + CZ + Toffoli pass 7.9 -> 5.6 ms at 2^30 FP32 and 2.3 -> 1.75 ms at 2^27 FP64.
// Accuracy: T is taken from the unitary nearest to M; g, p and the products with them
// are kept in long double and every entry is rounded once; x is rounded before
// -conj(x) is formed and g takes up the change of modulus, so T is a multiple of a
// unitary exactly.  Against 80-bit arithmetic (13 qubits, 12 circuits each of RX RY RZ +
// CRX, RY RZ + CNOT, U3 + CZ + Toffoli and U3 + CNOT; whole matrices in brackets):
// FP32 state 4.0 to 4.5e-7 (4.1 to 4.6e-7), gradient 3.8 to 5.8e-7 (4.8 to 6.6e-7);
// FP64 state 1.1 to 2.2e-15 (1.0 to 2.2e-15), gradient 2.2e-15 (2.0 to 2.7e-15).  The FP32 gradient's
// own forward sweep keeps whole matrices (its passes gain 2 % of the gradient's
// time), so that sweep's energy is unchanged.
//
// The reverse sweep applies the same ops to both states, so its reduced
// matrices come out in the pending frame: A[a][b] = |g|^2 conj(p_a) p_b A'[a][b]
// over the op's target.  The phases are folded into the D matrices here; |g| when
// the op has run is FOp::norm (AccRef::scale is its square).
constexpr double kMinPivot = 1e-9;
using cl = std::complex<long double>;
class Deferred {
 public:
  // Marks the ops of the sweep that a later uncontrolled one-qubit op on their qubit follows.
  Deferred(int n, bool adj, bool f32, std::vector<PlanPass>& passes)
      : adj_(adj), f32_(f32), every_(!f32 ? 32 : (adj ? 8 : 16)), min_(!f32 ? 1e-60 : (adj ? 1e-12 : 1e-18)),
        tol_(f32 ? 1e-13 : 1e-14),
        least_(f32 ? 1e-30 : 1e-280), ph_(n, cl(1)) {
    std::vector<char> open(n, 0);
    for (size_t pi = passes.size(); pi-- > 0;) {
      PlanPass& p = passes[pi];
      if (p.standalone) {
        std::fill(open.begin(), open.end(), 0);
        continue;
      }
      for (size_t i = p.ops.size(); i-- > 0;) {
        FOp& f = p.ops[i];
        if (f.kind != kOpU1 || f.cmask) continue;
        f.later = open[f.tq[0]];
        open[f.tq[0]] = 1;
      }
    }
  }
  // A reverse sweep with gates outside the tile passes defers nothing: their
  // reduced matrices are taken in the plain frame.
  static bool applies(bool adj, const std::vector<PlanPass>& passes) {
    for (const PlanPass& p : passes)
      if (adj && p.standalone) return false;
    return true;
  }
  // The sweep's next pass, its stages formed.
  void pass(PlanPass& p) {
    since_ = every_;  // (the pass's first deferred gate takes the norm)
    for (const PlanStage& st : p.stages)
      for (int oi : st.ops) op(p.ops[oi]);
  }

 private:
  // (plain products and norms: the library's test for infinities and take hypot,
  // a microsecond per gate; a long double holds the square of any matrix entry)
  static cl mul(const cl& a, const cl& b) {
    return cl(a.real() * b.real() - a.imag() * b.imag(), a.real() * b.imag() + a.imag() * b.real());
  }
  static cl mulc(const cl& a, const cl& b) {  // a conj(b)
    return cl(a.real() * b.real() + a.imag() * b.imag(), a.imag() * b.real() - a.real() * b.imag());
  }
  static long double mod(const cl& a) { return std::sqrt(a.real() * a.real() + a.imag() * a.imag()); }

  void op(FOp& f) {
    Mat& m = f.mat;
    const cl one(1);
    if (f.kind == kOpU2) {
      const cl a = ph_[f.tq[0]], b = ph_[f.tq[1]];
      if (a != one || b != one) {
        const cl c[4] = {one, a, b, mul(a, b)};
        for (int r = 0; r < 4; ++r)
          for (int q = 0; q < 4; ++q)
            if (m[4 * r + q] != cd(0)) m[4 * r + q] = cd(mulc(mul(cl(m[4 * r + q]), c[q]), c[r]));
      }
    } else if (f.kind == kOpU1 && f.cmask) {
      const cl p = ph_[f.tq[0]];
      if (p != one) {
        if (m[1] != cd(0)) m[1] = cd(mul(cl(m[1]), p));
        if (m[2] != cd(0)) m[2] = cd(mulc(cl(m[2]), p));
      }
    } else if (f.kind == kOpU1) {
      one_qubit(f);
    }
    f.norm = (double)ng_;
    if (adj_ && f.acc && f.kind == kOpU1) {  // the reduced matrix's frame
      const cl p = ph_[f.tq[0]];
      if (p != one)
        for (PGrad& pg : f.grads) pg.D[1] = cd(mul(cl(pg.D[1]), p)), pg.D[2] = cd(mulc(cl(pg.D[2]), p));
    }
  }
  void one_qubit(FOp& f) {
    cl& p = ph_[f.tq[0]];
    const cl m0(f.mat[0]), m1 = mul(cl(f.mat[1]), p), m2(f.mat[2]), m3 = mul(cl(f.mat[3]), p);
    const long double n0 = mod(m0), n1 = mod(m1), n2 = mod(m2), n3 = mod(m3);
    const long double top = std::max(std::max(n0, n3), std::max(n1, n2));
    const long double c = (n0 + n3) / 2, s = (n1 + n2) / 2, ng = ng_ * c;
    if (f.later && std::min(n0, n3) > kMinPivot * top && std::abs(n0 - n3) <= tol_ * top &&
        std::abs(n1 - n2) <= tol_ * top && ng > least_ && ng < 1 / least_) {
      // The unitary nearest to M / |.|: the entries' phases, of moduli c, s, s, c,
      // satisfy arg m1 + arg m2 = arg m0 + arg m3 + pi but for the rounding r of the
      // matrix, which is shared out (taking any three entries as they are would put
      // all of it into the fourth); r is below 1e-4 where the gate qualifies, so the
      // angle is its sine and the turn by d is 1 - d^2 / 2 + i d
      cl e0 = m0 / n0, e3 = m3 / n3, x(0);
      long double r = 0;
      bool unitary = true;
      if (n1 > 0 && n2 > 0) {
        cl e1 = m1 / n1;
        const cl z = mulc(mul(e1, m2 / n2), mul(e0, e3));
        r = -z.imag();
        // (what r changes of M's entries; a small c has a loose phase)
        unitary = z.real() < 0 && std::abs(r) < 1e-4L && std::abs(r) * c * s <= tol_ * top * top;
        const long double cc = c * c / (c * c + s * s), d0 = r * (1 - cc) / 2, d1 = -r * cc / 2;
        const cl t0(1 - d0 * d0 / 2, d0);
        e0 = mul(e0, t0), e3 = mul(e3, t0), e1 = mul(e1, cl(1 - d1 * d1 / 2, d1));
        x = mulc(e1, e0) * (s / c);
      }
      if (unitary) {
        p = whole_turns(mulc(e3, e0));
        const bool whole = since_ >= every_ || ng < min_ || ng > 1 / min_;
        const long double d = whole ? rounded(ng) : 1.0L;
        const cl w(rounded(d * x.real()), rounded(d * x.imag()));
        const long double turn = c * std::sqrt((1 + std::norm(x)) / (1 + std::norm(w / d))) / d;
        g_ = mul(g_, e0) * turn;
        ng_ *= turn;
        since_ = whole ? 0 : since_ + 1;
        f.form = whole ? kFormRC : (w == cl(0) ? kFormId : kFormUD);
        f.mat = {cd(d), cd(w), -std::conj(cd(w)), cd(d)};
        return;
      }
    }
    f.mat = {cd(mul(m0, g_)), cd(mul(m1, g_)), cd(mul(m2, g_)), cd(mul(m3, g_))};
    g_ = cl(1);
    ng_ = 1;
    p = cl(1);
  }
  long double rounded(long double v) const { return f32_ ? (long double)(float)v : (long double)(double)v; }
  // A phase within rounding of 1, i, -1 or -i is that one (a rounding error must
  // not decide which form the next gates take).
  cl whole_turns(const cl& p) const {
    if (std::abs(p.imag()) < tol_ / 10) return cl(p.real() > 0 ? 1 : -1);
    if (std::abs(p.real()) < tol_ / 10) return cl(0, p.imag() > 0 ? 1 : -1);
    return p;
  }
  bool adj_, f32_;
  int every_, since_ = 0;
  long double min_, tol_, least_;  // (least_: a norm a matrix entry can hold)
  std::vector<cl> ph_;
  cl g_ = cl(1);          // the deferred factor,
  long double ng_ = 1;    // its norm
};

// Conflict check of a register-bit set for the shared-memory swizzle.
// FP64: 16-byte amplitudes, quarter-warps over the tile swizzle Swz<double>;
// FP32: 8-byte amplitudes, half-warps over Swz<float>.  Packed FP32: 16-byte
// pairs, the lowest three thread bits (tile bits outside rs, ascending) must
// fall in distinct classes of the pair swizzle, class = (tile bit - 1) mod 3.
static bool rs_conflict_free(uint32_t rs, int M, int dtype, bool packed) {
  const int want = packed || dtype != VQC_C64 ? 3 : 4;
  int seen = 0, k = 0;
  for (int b = packed ? 1 : 0; b < M && k < want; ++b) {
    if (rs >> b & 1) continue;
    int res;
    if (packed)
      res = (b - 1) % 3;
    else if (dtype == VQC_C64)
      res = b < 4 ? b : (b < 8 ? b - 4 : -1);
    else
      res = b < 3 ? b : (b < 9 ? (b - 3) % 3 : -1);
    if (res < 0 || (seen >> res & 1)) return false;
    seen |= 1 << res;
    ++k;
  }
  return true;
}

// Cuts a pass into stages: runs of ops whose target bits fit the register
// set (4 tile bits; for FP32 tile bit 0 is always one of them, the lane bit
// of the packed layout).  The free bits left over are filled preferring the
// stage's control bits (register controls are compile-time cases in the FP32
// body), then a bank-conflict-free layout.
static void plan_stages(PlanPass& p, int M, int dtype, bool packed, int rb = kRegBits) {
  p.stages.clear();
  int tbit[64];  // global qubit -> tile bit, -1 outside the tile
  tile_bits(p, tbit);
  auto tile_mask_of = [&](uint64_t qubits) {
    uint32_t t = 0;
    for (uint64_t m = qubits; m; m &= m - 1) {
      const int b = tbit[__builtin_ctzll(m)];
      if (b >= 0) t |= 1u << b;
    }
    return t;
  };
  std::vector<int> pending(p.ops.size()), rest;
  for (size_t i = 0; i < pending.size(); ++i) pending[i] = (int)i;
  while (!pending.empty()) {
    PlanStage st;
    uint64_t blocked = 0;
    uint32_t rs = packed ? 1u : 0u;
    rest.clear();
    for (int oi : pending) {
      const FOp& f = p.ops[oi];
      if (f.qubits & blocked) {
        blocked |= f.qubits;
        rest.push_back(oi);
        continue;
      }
      uint32_t u = rs;
      if (f.kind == kOpU1 || f.kind == kOpU2) u |= 1u << tbit[f.tq[0]];
      if (f.kind == kOpU2) u |= 1u << tbit[f.tq[1]];
      if (__builtin_popcount(u) <= rb) {
        rs = u;
        st.ops.push_back(oi);
      } else {
        blocked |= f.qubits;
        rest.push_back(oi);
      }
    }
    // fill the register set to rb bits: control bits of the stage's ops first
    int cand[64], nc = 0;
    uint32_t listed = rs;
    for (int oi : st.ops)
      for (uint32_t m = tile_mask_of(p.ops[oi].cmask); m; m &= m - 1) {
        const int b = __builtin_ctz(m);
        if (!(listed >> b & 1)) cand[nc++] = b;
        listed |= 1u << b;
      }
    for (int b = 0; b < M; ++b)
      if (!(listed >> b & 1)) cand[nc++] = b;
    const int need_more = rb - __builtin_popcount(rs);
    nc = std::min(nc, 10);
    uint32_t best = 0;
    bool found = false;
    for (int mask = 0; mask < (1 << nc) && !found; ++mask) {
      if (__builtin_popcount(mask) != need_more) continue;
      uint32_t t = rs;
      for (int m = mask; m; m &= m - 1) t |= 1u << cand[__builtin_ctz(m)];
      if (!best) best = t;
      if (rs_conflict_free(t, M, dtype, packed)) {
        best = t;
        found = true;
      }
    }
    if (!found) prof_note("plan_stages_bank_conflicted", 1);
    for (uint32_t m = best; m; m &= m - 1) st.rs.push_back(__builtin_ctz(m));
    p.stages.push_back(std::move(st));
    pending.swap(rest);
  }
}

// Tile bits of the warp index (thread bits 5 and up) in a stage's layout.
static uint32_t warp_bits(const PlanStage& st, int M, int rb = kRegBits) {
  uint32_t rest = (1u << M) - 1;
  for (int b : st.rs) rest &= ~(1u << b);
  for (int i = 0; i < std::min(5, M - rb); ++i) rest &= rest - 1;
  return rest;
}

// A stage with no ops whose loads (or stores) of HBM are whole 128-byte runs:
// the same tile bits on the warp index as `st` (so a warp barrier separates the
// two), its lowest five other bits on the lanes, the rest in registers.
static PlanStage coalesced_stage(const PlanStage& st, int M, bool packed, int rb) {
  const uint32_t wb = warp_bits(st, M, rb);
  PlanStage c;
  if (packed) c.rs.push_back(0);
  for (int b = M - 1, left = rb - (int)c.rs.size(); left > 0; --b)
    if (!(wb >> b & 1)) {
      c.rs.push_back(b);
      --left;
    }
  std::sort(c.rs.begin(), c.rs.end());
  return c;
}
// The first and last stage of a pass read and write HBM in their own layout:
// with register bits among the lowest qubits a warp's 16-byte accesses lie 128
// bytes or more apart, a sector for every access.  A coalesced stage before
// (after) such a one costs one more exchange through shared memory, inside the
// warp.  Measured per pass, without and with: 326 -> 281 us forward and 955 -> 921
// us reverse at 2^26 FP32, 1.75 -> 1.34 ms (U3 + CZ + Toffoli) at 2^27 FP64, 616 ->
// 545 us on a 13-qubit FP64 density matrix, 21 -> 20 us forward at 2^21 FP32.
// States below 2^18 amplitudes wait for latency, not for sectors.
constexpr int kCoalesceQubits = 18;
static void coalesce_ends(PlanPass& p, int M, int dtype, bool packed, int rb) {
  const uint32_t run = packed ? 0xeu : (dtype == VQC_C64 ? 0xfu : 0x7u);  // the bits of a 128-byte run
  auto scattered = [&](const PlanStage& st) {
    uint32_t m = 0;
    for (int b : st.rs) m |= 1u << b;
    return (m & run) != 0;
  };
  if (scattered(p.stages.back())) p.stages.push_back(coalesced_stage(p.stages.back(), M, packed, rb));
  if (scattered(p.stages.front())) p.stages.insert(p.stages.begin(), coalesced_stage(p.stages.front(), M, packed, rb));
}

// ----------------------------------------------------------------------------- execution
struct Device {
  std::vector<unsigned char> buf;
  template <class T>
  size_t put(const T* p, size_t n) {
    size_t off = (buf.size() + 15) & ~size_t(15);
    buf.resize(off + sizeof(T) * n);
    std::memcpy(buf.data() + off, p, sizeof(T) * n);
    return off;
  }
};

// Dynamic shared memory of one pass: the tile(s), the accumulation slots (one
// row of 8 doubles per warp and slot) and the pass's descriptors.
static size_t pass_smem(size_t amp, int M, bool adj, const PassShape& ps, int rb = kRegBits) {
  const size_t nw = (size_t(1) << (M - rb)) / 32, npool = (size_t)ps.npool * amp;
  return (adj ? 2 : 1) * (amp << M) + (adj ? (size_t)ps.nslots * nw * 8 * sizeof(double) : 0) +
         (ps.packed ? sizeof(DevStageF) : sizeof(DevStage)) * ps.nstages + sizeof(DevOp) * ps.nops +
         ((npool + 15) & ~size_t(15));
}

// The library's kernel for a pass of that shape (not compiled at run time).
template <bool ADJ>
static const void* packed_kernel(int M) {
  switch (M) {
    case 12: return (const void*)k_tile_packed<12, ADJ>;
    case 11: return (const void*)k_tile_packed<11, ADJ>;
    case 10: return (const void*)k_tile_packed<10, ADJ>;
    default: return (const void*)k_tile_packed<9, ADJ>;
  }
}
template <class R, bool ADJ>
static const void* tile_kernel(int M, const PassShape& ps) {
  return ps.packed ? packed_kernel<ADJ>(M) : (const void*)k_tile<R, ADJ>;
}

// Lets kernel k use all the shared memory a block may have, once per device
// and kernel: a limit set per launch could be lowered by another thread between
// its setting and its launch (the serving loop's planners size the same kernels).
static int allow_smem(int device, const void* k) {
  static std::mutex mu;
  static std::set<std::pair<int, const void*>> done;
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({device, k})) return VQC_OK;
  cudaFuncAttributes fa;
  VQC_CK(cudaFuncGetAttributes(&fa, k));
  VQC_CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              device_info(device).max_smem_optin - (int)fa.sharedSizeBytes));
  done.insert({device, k});
  return VQC_OK;
}

// Resident CTAs of a tile kernel over the whole device (the occupancy query
// costs a microsecond or two, for every pass of every call: kept per kernel and
// shared-memory size).
static int kernel_grid(int device, const void* k, int nt, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, int, size_t>, int> known;
  const auto key = std::make_tuple(device, k, nt, smem);
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = known.find(key);
    if (it != known.end()) return it->second;
  }
  int per_sm = 0;
  if (allow_smem(device, k) ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, nt, smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    per_sm = 1;
  }
  std::lock_guard<std::mutex> lk(mu);
  return known[key] = device_info(device).sms * per_sm;
}

template <class R, int M, bool ADJ>
static int launch_tile(vqc_state h, const TileItem& item, const PassShape& ps, double flops) {
  const size_t smem = pass_smem(sizeof(cplx<R>), M, ADJ, ps);
  const void* k = tile_kernel<R, ADJ>(M, ps);
  if (int rc = allow_smem(h->device, k)) return rc;
  ProfScope prof(h->stream, ADJ ? "tile_adjoint" : "tile_forward",
                 (double)(ADJ ? 4 : 2) * h->size() * sizeof(cplx<R>), flops);
  void* args[] = {const_cast<TileItem*>(&item)};
  VQC_CK(cudaLaunchKernel(k, dim3(item.ncta), dim3(1 << (M - kRegBits)), args, smem, h->stream));
  return VQC_OK;
}

// A compiled FP64 pass; its matrices (host copy) are the kernel's second parameter.
template <int M, bool ADJ>
static int launch_tile64(vqc_state h, const void* k, const TileItem& item, const PassShape& ps, const void* host_pool,
                         double flops) {
  const size_t smem = pass_smem(sizeof(double2), M, ADJ, ps);
  if (int rc = allow_smem(h->device, k)) return rc;
  ProfScope prof(h->stream, ADJ ? "tile_adjoint" : "tile_forward",
                 (double)(ADJ ? 4 : 2) * h->size() * sizeof(double2), flops);
  void* args[] = {const_cast<TileItem*>(&item), const_cast<void*>(host_pool)};
  VQC_CK(cudaLaunchKernel(k, dim3(item.ncta), dim3(1 << (M - kRegBits)), args, smem, h->stream));
  return VQC_OK;
}

int standalone_adjoint(vqc_state h, void* lam, void* y, const GateSpec& gs, bool acc, double* out);

// The structure class of a one-qubit matrix (exact zeros: the matrices are
// built from closed forms, so structural zeros are exact).
static int u1_form(const Mat& m) {
  const cd u00 = m[0], u01 = m[1], u10 = m[2], u11 = m[3], one(1), zero(0);
  const bool diag = u01 == zero && u10 == zero, off = u00 == zero && u11 == zero;
  if (diag) return u00 == one && u11 == one ? kFormId : kFormDiag;
  if (off) return u01 == one && u10 == one ? kFormSwap : kFormOff;
  if (u00.imag() == 0 && u01.imag() == 0 && u10.imag() == 0 && u11.imag() == 0) return kFormReal;
  if (u00.imag() == 0 && u11.imag() == 0 && u01.real() == 0 && u10.real() == 0) return kFormRI;
  if (u00.imag() == 0 && u11.imag() == 0) return kFormRC;
  return kFormGen;
}
static int u1_form(const FOp& f) { return f.form >= 0 ? f.form : u1_form(f.mat); }

// Which entries of the reduced matrix the op's parameters need.
static int acc_kind(const FOp& f) {
  bool diag = false, off = false;
  for (const PGrad& pg : f.grads) {
    if (pg.D.size() < 4) return kAccFull;
    if (pg.D[0] != cd(0) || pg.D[3] != cd(0)) diag = true;
    if (pg.D[1] != cd(0) || pg.D[2] != cd(0)) off = true;
  }
  if (diag && !off) return kAccDiag;
  if (off && !diag) return kAccOff;
  return kAccFull;
}
// Every D of the op anti-Hermitian (as U^dagger dU/dtheta of a unitary family
// is): four values are then accumulated instead of eight (kAccAH).  rounding: what
// of D, relative to it, counts as the rounding of U^dagger dU and of the merges.
constexpr double kRounding32 = 1e-12, kRounding64 = 1e-14;
static bool acc_anti_hermitian(const FOp& f, double rounding) {
  for (const PGrad& pg : f.grads) {
    if (pg.D.size() != 4) return false;
    double scale = 0;
    for (const cd& d : pg.D) scale = std::max(scale, std::abs(d));
    const double eps = rounding * scale;
    if (std::abs(pg.D[0].real()) > eps || std::abs(pg.D[3].real()) > eps ||
        std::abs(pg.D[1] + std::conj(pg.D[2])) > eps)
      return false;
  }
  return !f.grads.empty();
}

// A diagonal gate with one entry that is not 1: that entry, else -1.
static int single_entry(const FOp& f) {
  int k0 = -1;
  for (int k = 0; k < (int)f.mat.size(); ++k)
    if (f.mat[k] != cd(1)) {
      if (k0 >= 0) return -1;
      k0 = k;
    }
  return k0;
}

// FMA-pipe lane operations (fused multiply-adds, multiplies, adds) of one pass
// over the whole state of n qubits, as the tile bodies implement its ops: a
// one-qubit op costs per amplitude pair and state 16 (general form), 12 (real
// diagonal), 8 (the other structured forms) or 0 (swap, identity), and in the reverse sweep its
// reduced-matrix accumulation 16 / 8 per pair (12 / 8 / 4 for the
// anti-Hermitian projection); a two-qubit op 64 per amplitude quad and state;
// a diagonal op 4 per state and amplitude that an entry other than 1 touches
// (a flip of sign none), 4 more for its accumulation.  Controls scale by the
// fraction of amplitudes they enable.  The numerator of the compute roofline
// (vqc_fma_peak is the denominator).
static double pass_fma_ops(const PlanPass& p, int n, bool adj) {
  const double pairs = std::ldexp(1.0, n - 1), amps = std::ldexp(1.0, n);
  const int nst = adj ? 2 : 1;
  static const int per_pair[kForms] = {16, 8, 8, 8, 0, 8, 12, 8, 0};  // by kForm*
  double ops = 0;
  for (const FOp& f : p.ops) {
    const double act = std::ldexp(1.0, -popc64(f.cmask));
    if (f.kind == kOpU1) {
      double o = (double)per_pair[u1_form(f)] * nst;
      if (adj && f.acc) {
        const int k = acc_kind(f);
        if (acc_anti_hermitian(f, kRounding32))
          o += k == kAccFull ? 12 : (k == kAccOff ? 8 : 4);
        else
          o += k == kAccFull ? 16 : 8;
      }
      ops += o * pairs * act;
    } else if (f.kind == kOpU2) {
      ops += 64.0 * nst * (amps / 4) * act;
    } else if (f.kind == kOpDiag) {
      const int k0 = single_entry(f);
      const double touched = k0 < 0 ? 1.0 : (f.mat[k0] == cd(-1) ? 0.0 : std::ldexp(1.0, -f.nd));
      ops += 4.0 * nst * amps * touched + (adj && f.acc ? 4.0 * amps : 0.0);
    }
  }
  return ops;
}

// The controls of an op by place: qubits outside the tile (one test per tile),
// thread bits (one test per op), register bits (rc, and the amplitudes they
// enable in rmask).
struct RegCtl {  // register controls: (j-bit, value)
  int n = 0;
  std::pair<int, int> c[8];
  const std::pair<int, int>* begin() const { return c; }
  const std::pair<int, int>* end() const { return c + n; }
};
static void place_controls(DevOp& o, uint64_t cmask, uint64_t cval, uint64_t tile_mask, const int (&tbit)[64],
                           const std::vector<int>& rs, RegCtl& rc) {
  for (uint64_t m = cmask; m; m &= m - 1) {
    const int q = __builtin_ctzll(m), v = (int)(cval >> q & 1);
    if (!(tile_mask >> q & 1)) {
      o.gmask |= 1ull << q;
      if (v) o.gval |= 1ull << q;
      continue;
    }
    const int b = tbit[q], j = (int)(std::find(rs.begin(), rs.end(), b) - rs.begin());
    if (j < (int)rs.size()) {
      rc.c[rc.n++] = {j, v};
    } else {
      o.cmask |= 1u << b;
      if (v) o.cval |= 1u << b;
    }
  }
  uint32_t need = 0, val = 0, rmask = 0;
  for (auto& c : rc) need |= 1u << c.first, val |= (uint32_t)c.second << c.first;
  for (uint32_t j = 0; j < (1u << rs.size()); ++j)
    if ((j & need) == val) rmask |= 1u << j;
  o.rmask = (int32_t)rmask;
  if (o.cmask) o.code |= kCodeCtl;
  if (o.gmask) o.code |= kCodeGCtl;
}

// A stage's index tables: global offsets of tile indices by bit, and the
// thread's nibble tables by doubling (thr: its tile bits, ascending).
struct StageTables {
  int64_t g[16];
  int thr[16], nthr = 0;
  StageTables(const PlanPass& p, int M, uint32_t rsmask) {
    for (int b = 0; b < M; ++b) {
      g[b] = int64_t(1) << p.tile_q[b];
      if (!(rsmask >> b & 1)) thr[nthr++] = b;
    }
  }
  int64_t global(uint32_t t) const {
    int64_t r = 0;
    for (; t; t &= t - 1) r |= g[__builtin_ctz(t)];
    return r;
  }
  template <class Put>
  void nibbles(Put put) const {
    for (int k = 0; k < 2; ++k) {
      uint32_t t[16] = {0};
      int64_t gt[16] = {0};
      put(k, 0, 0u, int64_t(0));
      for (int i = 0; i < 4; ++i)
        for (int nib = 1 << i; nib < 2 << i; ++nib) {
          const int low = nib ^ (1 << i);
          const bool on = 4 * k + i < nthr;
          t[nib] = t[low] | (on ? 1u << thr[4 * k + i] : 0u);
          gt[nib] = gt[low] | (on ? g[thr[4 * k + i]] : 0);
          put(k, nib, t[nib], gt[nib]);
        }
    }
  }
};

// One stage of the FP32 (packed) tile body: its DevStageF tables, its ops
// (j-bit targets, register controls as compile-time cases or a mask, the
// coefficient layouts of tile_f32.cuh) and their pool blocks.
static void stage_f32(const PlanPass& p, const PlanStage& st, int M, uint64_t tile_mask, const int (&tbit)[64], bool adj,
                      int& slot, int row, std::vector<DevStageF>& ds, std::vector<DevOp>& dops, std::vector<float2>& pool, size_t pool_begin,
                      std::vector<AccRef>* accs, int rb) {
  DevStageF s{};
  const std::vector<int>& rs = st.rs;  // ascending, rs[0] = tile bit 0
  const int na = 1 << rb, np = na / 2;  // register amplitudes, pairs
  uint32_t rsmask = 0;
  for (int b : rs) rsmask |= 1u << b;
  uint32_t dep[32];
  for (int j = 0; j < na; ++j) {
    uint32_t t = 0;
    for (int i = 0; i < rb; ++i)
      if (j >> i & 1) t |= 1u << rs[i];
    dep[j] = t;
    s.dep[j] = t;
  }
  const StageTables tabs(p, M, rsmask);
  tabs.nibbles([&](int k, int nib, uint32_t t, int64_t g) {
    s.thr[k][nib] = t;
    s.swt[k][nib] = f32t::swz_pair(t >> 1);
    s.gthr[k][nib] = g;
  });
  for (int m = 0; m < np; ++m) {
    s.swm[m] = f32t::swz_pair(dep[2 * m] >> 1);
    s.gdep[m] = tabs.global(dep[2 * m]);
  }
  auto jbit = [&](int b) { return (int)(std::find(rs.begin(), rs.end(), b) - rs.begin()); };
  auto put = [&](double a, double b) { pool.push_back(make_float2((float)a, (float)b)); };
  auto dup = [&](double a) { put(a, a); };
  auto dup3 = [&](cd a) { dup(a.real()), dup(a.imag()), dup(-a.imag()); };
  auto lane3 = [&](cd a, cd b) {
    put(a.real(), b.real()), put(a.imag(), b.imag()), put(-a.imag(), -b.imag());
  };
  s.op_begin = (int)dops.size();
  for (int oi : st.ops) {
    const FOp& f = p.ops[oi];
    DevOp o{};
    o.code = f.kind;
    o.slot = -1;
    RegCtl rc;
    place_controls(o, f.cmask, f.cval, tile_mask, tbit, rs, rc);
    int rctl = 0;
    if (rc.n) rctl = (rc.n == 1 && rc.c[0].second == 1) ? rc.c[0].first + 1 : 7;
    while (pool.size() % 2) put(0, 0);  // each op's block starts on 16 bytes
    o.mat = (int)(pool.size() - pool_begin);
    if (f.kind == kOpU1) {
      const int tb = jbit(tbit[f.tq[0]]), form = u1_form(f);
      o.code |= op_r_bits(tb, 0) | form_bits(form) | (rctl << 16);
      if (adj && f.acc) o.code |= (acc_kind(f) << 14) | (acc_anti_hermitian(f, kRounding32) ? kCodeAH : 0);
      const cd u00 = f.mat[0], u01 = f.mat[1], u10 = f.mat[2], u11 = f.mat[3];
      if (tb != 0) {
        switch (form) {
          case kFormGen:
            for (const cd& u : {u00, u01, u10, u11}) {
              dup(u.real());
              dup(u.imag());
              dup(-u.imag());
            }
            break;
          case kFormRI:
            dup(u00.real()), dup(u01.imag()), dup(-u01.imag()), dup(u11.real()), dup(u10.imag()), dup(-u10.imag());
            break;
          case kFormReal: dup(u00.real()), dup(u01.real()), dup(u10.real()), dup(u11.real()); break;
          case kFormDiag:
            dup(u00.real()), dup(u00.imag()), dup(-u00.imag()), dup(u11.real()), dup(u11.imag()), dup(-u11.imag());
            break;
          case kFormUD:
          case kFormOff:
            dup3(u01), dup3(u10);
            break;
          case kFormRC:
            dup(u00.real()), dup3(u01), dup(u11.real()), dup3(u10);
            break;
          default: break;
        }
      } else {
        switch (form) {
          case kFormGen:
            put(u00.real(), u11.real()), put(u01.real(), u10.real()), put(u00.imag(), u11.imag());
            put(-u00.imag(), -u11.imag()), put(u01.imag(), u10.imag()), put(-u01.imag(), -u10.imag());
            break;
          case kFormRI: put(u00.real(), u11.real()), put(-u01.imag(), -u10.imag()), put(u01.imag(), u10.imag()); break;
          case kFormReal: put(u00.real(), u11.real()), put(u01.real(), u10.real()); break;
          case kFormDiag:
            put(u00.real(), u11.real()), put(u00.imag(), u11.imag()), put(-u00.imag(), -u11.imag());
            break;
          case kFormUD:
          case kFormOff: lane3(u01, u10); break;
          case kFormRC:
            put(u00.real(), u11.real()), lane3(u01, u10);
            break;
          default: break;
        }
      }
    } else {
      if (f.kind == kOpU2) o.code |= op_r_bits(jbit(tbit[f.tq[0]]), jbit(tbit[f.tq[1]]));
      if (f.kind == kOpDiag) {
        const int k0 = single_entry(f);
        if (k0 >= 0) {
          o.code |= (f.mat[k0] == cd(-1) ? kDiagFlip : kDiagOne) << kDiagShift;
          o.rmask = k0;
        }
      }
      for (const cd& c : f.mat) put(c.real(), c.imag());
    }
    o.nd = f.nd;
    for (int i = 0; i < 5; ++i) {
      o.dbit[i] = -1;
      o.dglob[i] = 0;
      if (i < f.nd) {
        if (tile_mask >> f.dq[i] & 1)
          o.dbit[i] = tbit[f.dq[i]];
        else
          o.dglob[i] = f.dq[i];
      }
    }
    if (adj && f.acc) {
      o.slot = slot++;
      if (f.kind == kOpDiag) {
        // the accumulation runs as its own op right after the diagonal
        dops.push_back(o);
        DevOp a = o;
        a.code = (a.code & ~15) | kOpAccD;
        dops.push_back(a);
        if (accs) accs->push_back(AccRef{row + o.slot, f.grads, f.norm * f.norm});
        continue;
      }
      if (accs) accs->push_back(AccRef{row + o.slot, f.grads, f.norm * f.norm, (o.code & kCodeAH) != 0});
      o.code |= kCodeAcc;
    }
    dops.push_back(o);
  }
  s.op_end = (int)dops.size();
  ds.push_back(s);
}

template <class R, int M, bool ADJ>
static void serialize_plan(int n, int dtype, std::vector<PlanPass>& passes, SerialPlan& sp, std::vector<AccRef>* accs,
                           Deferred* defer, bool packed = false, int rb = kRegBits) {
  Device d;
  std::vector<cplx<R>> pool;
  std::vector<PassLoc>& locs = sp.locs;
  locs.assign(passes.size(), PassLoc());
  int row = 0;
  for (size_t pi = 0; pi < passes.size(); ++pi) {
    PlanPass& p = passes[pi];
    if (p.standalone) {
      locs[pi].standalone = true;
      locs[pi].gate = p.gate;
      continue;
    }
    plan_stages(p, M, dtype, packed, rb);
    if (defer) defer->pass(p);
    for (const FOp& f : p.ops) sp.norm_lo = std::min(sp.norm_lo, f.norm), sp.norm_hi = std::max(sp.norm_hi, f.norm);
    if (n >= kCoalesceQubits) coalesce_ends(p, M, dtype, packed, rb);
    std::vector<DevStage> ds;
    std::vector<DevOp> dops;
    int tbit[64];
    tile_bits(p, tbit);
    uint64_t tile_mask = 0;
    for (int q : p.tile_q) tile_mask |= 1ull << q;
    int slot = 0;
    while ((pool.size() * sizeof(cplx<R>)) % 16) pool.push_back(mkc<R>(R(0), R(0)));
    const size_t pool_begin = pool.size();
    std::vector<DevStageF> dsf;
    for (const PlanStage& st : p.stages) {
      if constexpr (std::is_same<R, float>::value) {
        if (packed) {
          stage_f32(p, st, M, tile_mask, tbit, ADJ, slot, row, dsf, dops, pool, pool_begin, accs, rb);
          continue;
        }
      }
      DevStage s{};
      uint32_t rsmask = 0;
      for (int b : st.rs) rsmask |= 1u << b;
      const StageTables tabs(p, M, rsmask);
      for (int j = 0; j < 16; ++j) {
        uint32_t t = 0;
        for (int i = 0; i < kRegBits; ++i)
          if (j >> i & 1) t |= 1u << st.rs[i];
        s.dep[j] = t;
        s.swm[j] = Swz<R>::f(t);
        s.gdep[j] = tabs.global(t);
      }
      tabs.nibbles([&](int k, int nib, uint32_t t, int64_t g) {
        s.thr[k][nib] = t;
        s.swt[k][nib] = Swz<R>::f(t);
        s.gthr[k][nib] = g;
      });
      s.cta = warp_bits(st, M) != warp_bits(p.stages[(&st - p.stages.data() + 1) % p.stages.size()], M);
      s.op_begin = (int)dops.size();
      for (int oi : st.ops) {
        const FOp& f = p.ops[oi];
        DevOp o{};
        o.code = f.kind;
        o.slot = -1;
        auto slot_of = [&](int b) { return (int)(std::find(st.rs.begin(), st.rs.end(), b) - st.rs.begin()); };
        // a phase on one entry of a diagonal gate is an op behind controls
        const int k0 = f.kind == kOpDiag ? single_entry(f) : -1;
        uint64_t cm = f.cmask, cv = f.cval;
        for (int i = 0; k0 >= 0 && i < f.nd; ++i) {
          cm |= 1ull << f.dq[i];
          if (k0 >> i & 1) cv |= 1ull << f.dq[i];
        }
        RegCtl rc;
        place_controls(o, cm, cv, tile_mask, tbit, st.rs, rc);
        int sel = k0 < 0 ? kSelDiag : (f.mat[k0] == cd(-1) ? kSelFlip : kSelPhase);
        if (f.kind == kOpU1) {
          const int r = slot_of(tbit[f.tq[0]]), form = interpreted_form<R>(u1_form(f));
          sel = kSelU1 + (r | (rc.n ? 4 : 0) | form << 3);
          const double rounding = sizeof(R) == 4 ? kRounding32 : kRounding64;
          if (ADJ && f.acc) o.code |= (acc_kind(f) << 14) | (acc_anti_hermitian(f, rounding) ? kCodeAH : 0);
        }
        if (f.kind == kOpU2) sel = kSelU2 + slot_of(tbit[f.tq[0]]) * 4 + slot_of(tbit[f.tq[1]]);
        if (k0 >= 0) o.code = (o.code & ~15) | kOpPhase;
        // the thread's amplitudes it acts on, for the interpreted body
        uint32_t held = 0;
        int nfree = 0;
        if (f.kind == kOpU1 || f.kind == kOpU2)
          for (int i = 0; i < (f.kind == kOpU1 ? 1 : 2); ++i) {
            const int r = slot_of(tbit[f.tq[i]]);
            held |= 1u << r;
            o.target[i] = (uint16_t)(s.swm[1 << r] * sizeof(cplx<R>));
          }
        for (auto& c : rc) {
          held |= 1u << c.first;
          if (c.second) o.first ^= (uint16_t)(s.swm[1 << c.first] * sizeof(cplx<R>));
        }
        for (int r = 0; r < kRegBits; ++r)
          if (!(held >> r & 1)) {
            if (nfree < 3) o.step[nfree] = (uint16_t)(s.swm[1 << r] * sizeof(cplx<R>));
            ++nfree;
          }
        o.code |= sel << kSelShift | nfree << 16;
        o.mat = (int)(pool.size() - pool_begin);
        if (k0 >= 0)
          pool.push_back(mkc<R>((R)f.mat[k0].real(), (R)f.mat[k0].imag()));
        else
          for (const cd& c : f.mat) pool.push_back(mkc<R>((R)c.real(), (R)c.imag()));
        o.nd = f.nd;
        for (int i = 0; i < 5; ++i) {
          o.dbit[i] = -1;
          o.dglob[i] = 0;
          if (i < f.nd) {
            if (tile_mask >> f.dq[i] & 1)
              o.dbit[i] = tbit[f.dq[i]];
            else
              o.dglob[i] = f.dq[i];
          }
        }
        if (ADJ && f.acc) {
          o.slot = slot++;
          if (f.kind == kOpDiag) {
            // the accumulation runs as its own op right after the diagonal, over
            // every bin (no controls)
            dops.push_back(o);
            DevOp a = o;
            a.code = kOpAccD | kCodeAcc | (kSelAccD << kSelShift);
            a.cmask = a.cval = 0;
            a.gmask = a.gval = 0;
            dops.push_back(a);
            if (accs) accs->push_back(AccRef{row + o.slot, f.grads, f.norm * f.norm});
            continue;
          }
          if (accs) accs->push_back(AccRef{row + o.slot, f.grads, f.norm * f.norm, (o.code & kCodeAH) != 0});
          o.code |= kCodeAcc;
        }
        dops.push_back(o);
      }
      s.op_end = (int)dops.size();
      ds.push_back(s);
    }
    p.nslots = slot;
    DevPass P{};
    P.nontile_mask = ((n >= 64) ? ~0ull : ((1ull << n) - 1)) & ~tile_mask;
    P.ntiles = int64_t(1) << (n - M);
    locs[pi].ntiles = P.ntiles;
    P.nslots = slot;
    P.nops = (int)dops.size();
    P.npool = (int)(pool.size() - pool_begin);
    locs[pi].pool_begin = pool_begin;
    locs[pi].shape.nslots = ADJ ? slot : 0;
    locs[pi].shape.nstages = (int)p.stages.size();
    locs[pi].shape.nops = P.nops;
    locs[pi].shape.npool = P.npool;
    locs[pi].row0 = row;
    row += slot;
    locs[pi].nslots = slot;
    locs[pi].fma_ops = pass_fma_ops(p, n, ADJ);
    // stage indices are local to this pass's stage array
    P.stage_begin = 0;
    P.stage_end = (int)p.stages.size();
    locs[pi].pass = d.put(&P, 1);
    if (packed)
      locs[pi].stages = d.put(dsf.data(), dsf.size());
    else
      locs[pi].stages = d.put(ds.data(), ds.size());
    locs[pi].shape.packed = packed;
    // op indices in stages are local to this pass's op array
    locs[pi].ops = d.put(dops.data(), std::max<size_t>(dops.size(), 1));
  }
  for (int i = 0; i < 4; ++i) pool.push_back(mkc<R>(R(0), R(0)));  // the staging copy reads whole 16-byte words
  sp.pool_off = d.put(pool.data(), pool.size());
  sp.rows = row;
  sp.buf.swap(d.buf);
}

static void note_plan(bool adj, const std::vector<PlanPass>& passes) {
  long long np = 0, ns = 0, no = 0, nsa = 0, nd = 0;
  for (auto& p : passes) {
    if (p.standalone) {
      ++nsa;
      continue;
    }
    ++np;
    ns += (long long)p.stages.size();
    no += (long long)p.ops.size();
    for (const FOp& f : p.ops) nd += f.form >= 0;
  }
  prof_note(adj ? "plan_adjoint_passes" : "plan_forward_passes", np);
  prof_note(adj ? "plan_adjoint_stages" : "plan_forward_stages", ns);
  prof_note(adj ? "plan_adjoint_ops" : "plan_forward_ops", no);
  prof_note("plan_standalone_gates", nsa);
  prof_note(adj ? "plan_adjoint_deferred" : "plan_forward_deferred", nd);
}

template <int M, bool ADJ>
static int launch_tile_jit(vqc_state h, const void* k, void* psi, void* lam, const DevPass* dp, const void* ds,
                           const DevOp* dops, const void* pool, double* partials, int grid, const PassShape& ps,
                           const void* host_pool, double flops, int rb = kRegBits) {
  const int NT = 1 << (M - rb);
  const size_t smem = pass_smem(sizeof(float2), M, ADJ, ps) + jit_extra_smem(ADJ, M, rb);
  if (int rc = allow_smem(h->device, k)) return rc;
  ProfScope prof(h->stream, ADJ ? "tile_adjoint" : "tile_forward", (double)(ADJ ? 4 : 2) * h->size() * sizeof(float2),
                 flops);
  // the last parameter is the pass's matrix pool by value (host copy)
  void* args[] = {&psi, &lam, (void*)&dp, (void*)&ds, (void*)&dops, (void*)&pool, &partials, const_cast<void*>(host_pool)};
  VQC_CK(cudaLaunchKernel(k, dim3(grid), dim3(NT), args, smem, h->stream));
  return VQC_OK;
}

// JIT tile passes for FP32 states of at least 2^18 amplitudes (VQC_JIT=auto),
// all FP32 tile passes (on), none (off).
static bool use_jit(const vqc_state h) {
  const int mode = jit_mode();
  return h->dtype == VQC_C64 && (mode == 1 || (mode == 2 && h->nq >= 18)) && jit_available();
}
// The packed FP32 plan layout: for the compiled passes, or forced with
// VQC_JIT=interp (the packed interpreter, the compiled kernels' fallback).
static bool use_packed(const vqc_state h) { return h->dtype == VQC_C64 && (use_jit(h) || jit_mode() == 3); }
// FP64 passes planned for compiled kernels (deferred phases) and compiled: states of
// at least 2^kCompileQubits64 amplitudes (auto), all (on).  Compiling a call's passes
// takes the host some seconds and saves 2 ms a call at 23 qubits but 0.2 ms at 20,
// and a stream of different circuits of 20-22 qubits met a compile in most calls (5
// against 400 requests a second).  Smaller states run whole matrices interpreted;
// deferred phases cost them 5 to 10 % (U3 + CNOT 705 against 655 us at 20 qubits and
// 1,952 against 1,759 us at 22, an 11-qubit density matrix 1,983 against 1,823 us).
constexpr int kCompileQubits64 = 23;
static bool use_jit64(const vqc_state h) {
  const int mode = jit_mode();
  return h->dtype == VQC_C128 && (mode == 1 || (mode == 2 && h->nq >= kCompileQubits64)) && jit_available();
}
static uint64_t new_call() {
  static std::atomic<uint64_t> n{0};
  return ++n;
}
// VQC_JIT_WIDE=1: compiled forward passes with 32 amplitudes per thread (four
// free register bits per stage: 3.0 instead of 3.8 stages per pass on the
// headline circuit).  Off by default: measured slower at 2^26 amplitudes
// (0.40 against 0.355 ms per pass: five 128-thread CTAs per SM at 96
// registers, with spills), and NVRTC takes 15-140 s per such pass (1-2 s at
// 16 amplitudes), in its optimizer, not in ptxas.
static bool wide_forward() {
  const char* v = std::getenv("VQC_JIT_WIDE");
  return v && *v && std::atoi(v) != 0;
}

// An upper bound of one pass's serialised bytes (serialize_plan): at most one
// stage per op, two op records per op, 32 matrix entries (+ alignment) per op.
template <class R>
static size_t op_bytes_bound(const PlanPass& p) {
  const size_t nops = p.ops.size() + 3;  // (a stage per op, and coalesced ones at both ends)
  return 3 * 16 + sizeof(DevPass) + nops * std::max(sizeof(DevStageF), sizeof(DevStage)) + 2 * nops * sizeof(DevOp) +
         (34 * nops + 8) * sizeof(cplx<R>);
}

// op_used != nullptr: the pass descriptors go to the op buffer at op_off
// (reserved by the caller) and *op_used receives their size, so that later
// chunks of one sweep can be uploaded while these passes run.
template <class R, int M, bool ADJ>
static int run_plan(vqc_state h, void* psi, void* lam, std::vector<PlanPass>& passes, const std::vector<GateSpec>& specs,
                    std::vector<AccRef>* accs, double* rows_dev, uint64_t call, Deferred* defer, size_t op_off = 0,
                    size_t* op_used = nullptr) {
  const int n = h->nq;
  SerialPlan sp;
  const bool packed = use_packed(h);
  // wide compiled forward passes (VQC_JIT_WIDE=1): 32 amplitudes per thread,
  // four free register bits per stage; the generic kernels take 16
  int rb = (!ADJ && packed && use_jit(h) && wide_forward()) ? kWideRegBits : kRegBits;
  const size_t accs0 = accs ? accs->size() : 0;
  std::vector<PlanPass> plain;  // (to plan again at 16 amplitudes)
  std::optional<Deferred> before;
  if (rb != kRegBits) {
    plain = passes;
    if (defer) before = *defer;
  }
  serialize_plan<R, M, ADJ>(n, h->dtype, passes, sp, accs, defer, packed, rb);
  note_plan(ADJ, passes);
  // run-time specialised kernels (FP32), one per pass structure
  std::vector<const void*> jk(passes.size(), nullptr);
  if constexpr (std::is_same<R, float>::value) {
    if (packed && use_jit(h)) {
      auto compile = [&]() {
        std::vector<JitPassRef> refs(passes.size());
        for (size_t pi = 0; pi < passes.size(); ++pi)
          if (!sp.locs[pi].standalone)
            refs[pi] = JitPassRef{(const DevStageF*)(sp.buf.data() + sp.locs[pi].stages), sp.locs[pi].shape.nstages,
                                  (const DevOp*)(sp.buf.data() + sp.locs[pi].ops), sp.locs[pi].shape.npool};
        jit_pass_kernels(M, ADJ, refs, jk, false, true, rb);
      };
      compile();
      if (rb != kRegBits) {
        // a wide pass without a kernel (beyond the parameter space, or a failed
        // compile) has no generic kernel: plan the whole sweep at 16 amplitudes
        bool missing = false;
        for (size_t pi = 0; pi < passes.size(); ++pi) missing = missing || (!sp.locs[pi].standalone && !jk[pi]);
        if (missing) {
          rb = kRegBits;
          sp = SerialPlan();
          if (accs) accs->resize(accs0);
          passes = std::move(plain);
          if (defer) *defer = *before;
          serialize_plan<R, M, ADJ>(n, h->dtype, passes, sp, accs, defer, packed, rb);
          jk.assign(passes.size(), nullptr);
          compile();
        }
      }
    }
  }
  if constexpr (std::is_same<R, double>::value) {
    if (use_jit64(h)) {
      std::vector<JitPassRef64> refs(passes.size());
      for (size_t pi = 0; pi < passes.size(); ++pi)
        if (!sp.locs[pi].standalone)
          refs[pi] = JitPassRef64{(const DevStage*)(sp.buf.data() + sp.locs[pi].stages), sp.locs[pi].shape.nstages,
                                  (const DevOp*)(sp.buf.data() + sp.locs[pi].ops), sp.locs[pi].shape.npool};
      jit_pass_kernels64(M, ADJ, refs, jk, call, jit_mode() == 1);
    }
  }
  const std::vector<PassLoc>& locs = sp.locs;
  const size_t pool_off = sp.pool_off;
  std::vector<int> grids(passes.size(), 0);
  for (size_t pi = 0; pi < passes.size(); ++pi) {
    if (locs[pi].standalone) continue;
    const size_t smem = pass_smem(sizeof(cplx<R>), M, ADJ, locs[pi].shape);
    int g = jk[pi] ? kernel_grid(h->device, jk[pi], 1 << (M - rb), smem + jit_extra_smem(ADJ, M, rb))
                         : kernel_grid(h->device, tile_kernel<R, ADJ>(M, locs[pi].shape), 1 << (M - kRegBits), smem);
    // the CTAs' partial sums group alike in both kernels of an FP64 pass
    if constexpr (ADJ && std::is_same<R, double>::value)
      if (use_jit64(h)) g = device_info(h->device).sms * jit_min_blocks64(true);
    grids[pi] = (int)std::min<int64_t>(g, locs[pi].ntiles);
  }
  // partial sums scratch: one row of 8 doubles per (CTA, slot) of every pass,
  // summed over the CTAs by one launch after the sweep (the same fixed order
  // per slot as a reduction after each pass)
  std::vector<size_t> poff(passes.size(), 0);
  size_t need = 0;
  int max_slots = 0;
  for (size_t pi = 0; pi < passes.size(); ++pi)
    if (!locs[pi].standalone && locs[pi].nslots > 0) {
      poff[pi] = need / sizeof(double);
      need += (size_t)grids[pi] * locs[pi].nslots * 8 * sizeof(double);
      max_slots = std::max(max_slots, locs[pi].nslots);
    }
  double* partials = nullptr;
  if (ADJ && need > 0) {
    if (int rc = reserve_buffer(h, &h->fused_scratch, &h->fused_scratch_bytes, need)) return rc;
    partials = (double*)h->fused_scratch;
  }
  // the reduction items travel with the pass descriptors
  size_t red_off = 0, nred = 0;
  if (ADJ && need > 0) {
    std::vector<RedItem> red;
    for (size_t pi = 0; pi < passes.size(); ++pi)
      if (!locs[pi].standalone && locs[pi].nslots > 0)
        red.push_back(RedItem{partials + poff[pi], grids[pi], locs[pi].nslots, rows_dev + (size_t)locs[pi].row0 * 8});
    red_off = (sp.buf.size() + 15) & ~size_t(15);
    nred = red.size();
    sp.buf.resize(red_off + sizeof(RedItem) * nred);
    std::memcpy(sp.buf.data() + red_off, red.data(), sizeof(RedItem) * nred);
  }
  int rc = op_used ? upload_ops_at(h, op_off, sp.buf.data(), sp.buf.size()) : upload_ops(h, sp.buf.data(), sp.buf.size());
  if (rc) return rc;
  if (op_used) *op_used = sp.buf.size();
  const unsigned char* base = (const unsigned char*)h->opbuf + op_off;
  for (size_t pi = 0; pi < passes.size(); ++pi) {
    if (locs[pi].standalone) {
      const GateSpec& gs = specs[locs[pi].gate];
      if (ADJ) {
        if ((rc = standalone_adjoint(h, lam, psi, gs, false, nullptr))) return rc;
      } else {
        if ((rc = launch_gate(gs, psi, n, h->dtype, h->device, h->stream))) return rc;
      }
      continue;
    }
    const int grid = grids[pi];
    double* pp = partials ? partials + poff[pi] : nullptr;
    const DevPass* dp = (const DevPass*)(base + locs[pi].pass);
    const void* ds = (const void*)(base + locs[pi].stages);
    const DevOp* dops = (const DevOp*)(base + locs[pi].ops);
    const void* dpool = base + pool_off + locs[pi].pool_begin * sizeof(cplx<R>);
    TileItem it{psi, lam, dp, ds, dops, dpool, pp, locs[pi].ntiles, grid, M, DevPass()};
    std::memcpy(&it.p, sp.buf.data() + locs[pi].pass, sizeof(DevPass));
    if (jk[pi]) {
      if constexpr (std::is_same<R, double>::value)
        if ((rc = launch_tile64<M, ADJ>(h, jk[pi], it, locs[pi].shape,
                                        sp.buf.data() + pool_off + locs[pi].pool_begin * sizeof(double2),
                                        2.0 * locs[pi].fma_ops)))
          return rc;
      if constexpr (std::is_same<R, float>::value)
        if ((rc = launch_tile_jit<M, ADJ>(h, jk[pi], psi, lam, dp, ds, dops, dpool, pp, grid,
                                          locs[pi].shape,
                                          sp.buf.data() + pool_off + locs[pi].pool_begin * sizeof(float2),
                                          2.0 * locs[pi].fma_ops, rb)))
          return rc;
    } else if ((rc = launch_tile<R, M, ADJ>(h, it, locs[pi].shape, 2.0 * locs[pi].fma_ops))) {
      return rc;
    }
  }
  if (nred > 0) {
    k_reduce_slots_batch<<<dim3(max_slots, (unsigned)nred), 256, 0, h->stream>>>((const RedItem*)(base + red_off));
    VQC_CK(cudaGetLastError());
  }
  return VQC_OK;
}

// Bytes of the reverse sweep's partial sums, an upper bound for its largest chunk
// (chunks of 1, 2, 4, ... consecutive tile passes, see reverse_impl): a handle's
// scratch is sized once, before the first chunk.  Grown chunk by chunk it drained
// the stream and allocated up to six times in the first gradient of a handle.
template <class R>
static size_t partials_bound(vqc_state h, int M, const std::vector<PlanPass>& passes) {
  // resident CTAs: two tiles each
  const int64_t per_sm = std::max<int64_t>(device_info(h->device).max_smem_optin / (2 * (sizeof(cplx<R>) << M)), 1);
  const size_t grid = (size_t)std::min<int64_t>(int64_t(1) << (h->nq - M), device_info(h->device).sms * per_sm);
  size_t most = 0, take = 1;
  for (size_t i = 0; i < passes.size();) {
    size_t slots = 0, k = 0;
    for (; i < passes.size() && !passes[i].standalone && k < take; ++i, ++k)
      for (const FOp& f : passes[i].ops) slots += f.acc;
    if (k == 0)
      ++i;
    else
      take = std::min(2 * take, passes.size());
    most = std::max(most, slots);
  }
  return grid * most * 8 * sizeof(double);
}

int fused_supported(vqc_state h) { return h->nq >= kMinTileBits && h->nq <= 40; }

template <class R, int M>
static int forward_impl(vqc_state h, const vqc_gate* gates, int ngates, const double* mats, bool defer) {
  std::vector<GateSpec> specs(ngates);
  std::vector<PItem> items(ngates);
  // gate analysis, on up to four host threads for long circuits (it precedes
  // the first launch: the device waits for it)
  auto analyze = [&](int i0, int i1) {
    for (int i = i0; i < i1; ++i) {
      if (analyze_gate(h->nq, gates[i].nq, gates[i].pos, mats + gates[i].mat, false, specs[i])) return i;
      items[i].gate = i;
      items[i].standalone = !to_fop(specs[i], items[i].op);
    }
    return -1;
  };
  const int nth = ngates >= 1024 ? (int)std::min(4u, std::max(1u, std::thread::hardware_concurrency())) : 1;
  std::vector<int> bad(nth, -1);
  std::vector<std::thread> pool;
  for (int t = 1; t < nth; ++t)
    pool.emplace_back([&, t] { bad[t] = analyze((int)((int64_t)ngates * t / nth), (int)((int64_t)ngates * (t + 1) / nth)); });
  bad[0] = analyze(0, (int)((int64_t)ngates / nth));
  for (auto& th : pool) th.join();
  for (int t = 0; t < nth; ++t)
    if (bad[t] >= 0)  // again on this thread, for its error message
      return analyze_gate(h->nq, gates[bad[t]].nq, gates[bad[t]].pos, mats + gates[bad[t]].mat, false, specs[bad[t]]);
  std::vector<PlanPass> passes;
  plan_passes(h->nq, tile_config(h->dtype, h->nq), false, items, passes);
  std::optional<Deferred> deferred;
  if (defer && (use_packed(h) || use_jit64(h))) deferred.emplace(h->nq, false, h->dtype == VQC_C64, passes);
  Deferred* df = deferred ? &*deferred : nullptr;
  const uint64_t call = new_call();
  const char* pc = std::getenv("VQC_PLAN_CHUNKS");  // 0: one serialisation for the whole sweep
  if (passes.size() < 4 || (pc && *pc && std::atoi(pc) == 0))
    return run_plan<R, M, false>(h, h->d, nullptr, passes, specs, nullptr, nullptr, call, df);
  // Serialised and launched in chunks of 1, 2, 4, ... passes: the host plans
  // the next chunk while the device runs the previous ones, instead of the
  // device waiting for the whole sweep's descriptors (about 1.5 ms for 2,000
  // gates).  Each chunk's descriptors get their own region of the op buffer.
  size_t bound = 256;
  for (const PlanPass& p : passes) bound += op_bytes_bound<R>(p);
  int rc = reserve_ops(h, bound);
  if (rc) return rc;
  size_t off = 0, take = 1;
  const uint64_t compiles = jit_compiles();
  for (size_t first = 0, last; first < passes.size(); first = last, take *= 2) {
    last = jit_compiles() != compiles ? passes.size() : std::min(passes.size(), first + take);
    std::vector<PlanPass> chunk(std::make_move_iterator(passes.begin() + first),
                                std::make_move_iterator(passes.begin() + last));
    size_t used = 0;
    if ((rc = run_plan<R, M, false>(h, h->d, nullptr, chunk, specs, nullptr, nullptr, call, df, off, &used))) return rc;
    off = (off + used + 255) & ~size_t(255);
  }
  return VQC_OK;
}

int apply_circuit_fused(vqc_state h, const vqc_gate* gates, int ngates, const double* mats, bool defer) {
  if (!fused_supported(h)) {
    for (int i = 0; i < ngates; ++i) {
      int rc = apply_gate_raw(h, gates[i].nq, gates[i].pos, mats + gates[i].mat);
      if (rc) return rc;
    }
    return VQC_OK;
  }
  switch (tile_config(h->dtype, h->nq).M + (h->dtype == VQC_C64 ? 0 : 100)) {
    case 12: return forward_impl<float, 12>(h, gates, ngates, mats, defer);
    case 11: return forward_impl<float, 11>(h, gates, ngates, mats, defer);
    case 10: return forward_impl<float, 10>(h, gates, ngates, mats, defer);
    case 9: return forward_impl<float, 9>(h, gates, ngates, mats, defer);
    case 111: return forward_impl<double, 11>(h, gates, ngates, mats, defer);
    case 110: return forward_impl<double, 10>(h, gates, ngates, mats, defer);
    default: return forward_impl<double, 9>(h, gates, ngates, mats, defer);
  }
}

// Reverse sweep on the tile engine.  grads[j] receive the partials.  Gates
// the tile engine cannot take (3+ targets, or 2 targets with parameters) run
// through the per-gate adjoint path.
int per_gate_params_grad(vqc_state h, void* lam, void* y, const GateSpec& gs, const std::vector<ParamInfo>& ps,
                         double* grads);

// The reverse sweep's op list: gates last to first (specs hold U^dagger),
// with the reduced-matrix accumulation on every op that carries parameters.
static std::vector<PItem> reverse_items(const std::vector<GateSpec>& specs,
                                        const std::vector<std::vector<ParamInfo>>& params) {
  const int ng = (int)specs.size();
  std::vector<PItem> items;
  items.reserve(ng);
  for (int i = ng - 1; i >= 0; --i) {
    PItem it;
    it.gate = i;
    const GateSpec& gs = specs[i];
    bool ok = to_fop(gs, it.op);
    if (ok && !params[i].empty()) {
      FOp& f = it.op;
      if (f.kind == kOpU1) {
        f.acc = true;
        for (const ParamInfo& pi : params[i]) f.grads.push_back(PGrad{pi.index, restrict_to(gs, f, pi.D)});
      } else if (f.kind == kOpDiag && f.nd <= 2 && f.nd >= 1) {
        f.acc = true;
        const int d = 1 << gs.k;
        for (const ParamInfo& pi : params[i]) {
          PGrad pg{pi.index, {}};
          pg.D.assign(d, cd(0));
          for (int j = 0; j < d; ++j) pg.D[j] = pi.D[(size_t)j * d + j];
          f.grads.push_back(std::move(pg));
        }
      } else {
        ok = false;
      }
    }
    it.standalone = !ok;
    items.push_back(std::move(it));
  }
  return items;
}

template <class R, int M>
static int reverse_impl(vqc_state h, void* lam, void* y, const std::vector<GateSpec>& specs,
                        const std::vector<std::vector<ParamInfo>>& params, double* grads) {
  std::vector<PItem> items = reverse_items(specs, params);
  std::vector<PlanPass> passes;
  plan_passes(h->nq, tile_config(h->dtype, h->nq), true, items, passes);
  std::optional<Deferred> deferred;
  if ((use_packed(h) || use_jit64(h)) && Deferred::applies(true, passes))
    deferred.emplace(h->nq, true, h->dtype == VQC_C64, passes);
  // standalone gates with parameters: split their passes out so the per-gate
  // path can evaluate the partials right after the uncompute
  std::vector<AccRef> accs;
  int total_rows = 0;
  for (auto& p : passes)
    if (!p.standalone) {
      int s = 0;
      for (auto& f : p.ops) s += f.acc ? 1 : 0;
      total_rows += s;
    }
  if (int rc = reserve_buffer(h, &h->accbuf, &h->accbuf_bytes, sizeof(double) * 8 * total_rows)) return rc;
  const uint64_t call = new_call();
  int row_base = 0;
  const uint64_t compiles = jit_compiles();
  size_t bound = 256, off = 0, take = 1;
  for (const PlanPass& p : passes) bound += op_bytes_bound<R>(p) + sizeof(RedItem) + 256;
  if (int rc = reserve_ops(h, bound)) return rc;
  if (int rc = reserve_buffer(h, &h->fused_scratch, &h->fused_scratch_bytes, partials_bound<R>(h, M, passes))) return rc;
  for (size_t pi = 0; pi < passes.size(); ++pi) {
    if (passes[pi].standalone) {
      const int gi = passes[pi].gate;
      const GateSpec& gs = specs[gi];
      if (params[gi].empty()) {
        int rc = standalone_adjoint(h, lam, y, gs, false, nullptr);
        if (rc) return rc;
      } else {
        int rc = per_gate_params_grad(h, lam, y, gs, params[gi], grads);
        if (rc) return rc;
      }
      continue;
    }
    // consecutive tile passes in chunks of 1, 2, 4, ... passes, each in its own
    // region of the op buffer (as the forward sweep): the device starts on the
    // first while the host serialises the rest
    size_t pj = pi;
    std::vector<PlanPass> group;
    if (jit_compiles() != compiles) take = passes.size();
    while (pj < passes.size() && !passes[pj].standalone && group.size() < take) group.push_back(std::move(passes[pj++]));
    take = std::min(2 * take, passes.size());  // (a sweep has a chunk per gate outside the passes: doubling is bounded)
    std::vector<AccRef> gaccs;
    size_t used = 0;
    int rc = run_plan<R, M, true>(h, y, lam, group, specs, &gaccs, (double*)h->accbuf + (size_t)row_base * 8, call,
                                   deferred ? &*deferred : nullptr, off, &used);
    if (rc) return rc;
    off = (off + used + 255) & ~size_t(255);
    for (auto& a : gaccs) {
      a.row += row_base;
      accs.push_back(std::move(a));
    }
    for (auto& g : group) row_base += g.nslots;
    pi = pj - 1;
  }
  // contract A with the D matrices
  std::vector<double> A((size_t)std::max(row_base, 1) * 8);
  if (row_base > 0)
    VQC_CK(cudaMemcpyAsync(A.data(), h->accbuf, sizeof(double) * 8 * row_base, cudaMemcpyDeviceToHost, h->stream));
  VQC_CK(cudaStreamSynchronize(h->stream));
  contract_grads(accs, A.data(), grads);
  return VQC_OK;
}

int reverse_sweep_fused(vqc_state h, void* lam, void* y, const std::vector<GateSpec>& specs,
                        const std::vector<std::vector<ParamInfo>>& params, double* grads) {
  switch (tile_config(h->dtype, h->nq).M + (h->dtype == VQC_C64 ? 0 : 100)) {
    case 12: return reverse_impl<float, 12>(h, lam, y, specs, params, grads);
    case 11: return reverse_impl<float, 11>(h, lam, y, specs, params, grads);
    case 10: return reverse_impl<float, 10>(h, lam, y, specs, params, grads);
    case 9: return reverse_impl<float, 9>(h, lam, y, specs, params, grads);
    case 111: return reverse_impl<double, 11>(h, lam, y, specs, params, grads);
    case 110: return reverse_impl<double, 10>(h, lam, y, specs, params, grads);
    default: return reverse_impl<double, 9>(h, lam, y, specs, params, grads);
  }
}

}  // namespace vqc

namespace vqc {

// g_j = Re sum_ab D_j[a][b] A[a][b] for every parameter of every accumulating op
// (U1: D is 2x2 row-major and A[a][b] sits at 2a+b; AccD: diagonal bins in order).
void contract_grads(const std::vector<AccRef>& accs, const double* A, double* grads) {
  for (const AccRef& a : accs) {
    const double* r = &A[(size_t)a.row * 8];
    if (a.ah) {
      // r = (Im A00, Im A11, Re A01 - Re A10, Im A01 + Im A10), D anti-Hermitian
      for (const PGrad& pg : a.grads)
        grads[pg.param] = a.scale * (-pg.D[0].imag() * r[0] - pg.D[3].imag() * r[1] + pg.D[1].real() * r[2] -
                                     pg.D[1].imag() * r[3]);
      continue;
    }
    const cd Av[4] = {cd(r[0], r[1]), cd(r[2], r[3]), cd(r[4], r[5]), cd(r[6], r[7])};
    for (const PGrad& pg : a.grads) {
      double g = 0;
      for (size_t i = 0; i < pg.D.size() && i < 4; ++i) g += (pg.D[i] * Av[i]).real();
      grads[pg.param] = a.scale * g;
    }
  }
}

// ----------------------------------------------------------------------------- serving support
__global__ void __launch_bounds__(256) k_reduce_slots_batch(const RedItem* __restrict__ items) {
  __shared__ double sm[8][8];
  const RedItem it = items[blockIdx.y];
  const int slot = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (slot >= it.nslots) return;
  for (int val = 0; val < 8; ++val) {
    double s = 0;
    for (int b = threadIdx.x; b < it.nblocks; b += blockDim.x)
      s += it.partials[((size_t)b * it.nslots + slot) * 8 + val];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) sm[warp][val] = s;
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    double s = 0;
    for (int wp = 0; wp < (int)(blockDim.x >> 5); ++wp) s += sm[wp][threadIdx.x];
    it.out[(size_t)slot * 8 + threadIdx.x] = s;
  }
}

template <class R, int M>
static int build_plan_tm(int n, int dtype, const std::vector<GateSpec>& fspecs, const std::vector<GateSpec>& rspecs,
                         const std::vector<std::vector<ParamInfo>>& params, bool want_grad, bool packed,
                         ReqPlan& rp) {
  const TileConfig tc = tile_config(dtype, n);
  auto shape_max = [packed](const SerialPlan& sp) {
    PassShape m;
    m.packed = packed;
    for (const PassLoc& l : sp.locs) {
      m.nslots = std::max(m.nslots, l.shape.nslots);
      m.nstages = std::max(m.nstages, l.shape.nstages);
      m.nops = std::max(m.nops, l.shape.nops);
      m.npool = std::max(m.npool, l.shape.npool);
    }
    return m;
  };
  std::vector<PItem> items(fspecs.size());
  for (size_t i = 0; i < fspecs.size(); ++i) {
    items[i].gate = (int)i;
    items[i].standalone = !to_fop(fspecs[i], items[i].op);
  }
  std::vector<PlanPass> passes;
  plan_passes(n, tc, false, items, passes);
  for (const PlanPass& p : passes)
    if (p.standalone) return fail(VQC_ERR_UNSUPPORTED, "serving takes gates with at most two target qubits");
  std::optional<Deferred> deferred;
  if (packed) deferred.emplace(n, false, dtype == VQC_C64, passes);
  serialize_plan<R, M, false>(n, dtype, passes, rp.fwd, nullptr, deferred ? &*deferred : nullptr, packed);
  rp.fwd_max = shape_max(rp.fwd);
  if (want_grad) {
    std::vector<PItem> ritems = reverse_items(rspecs, params);
    std::vector<PlanPass> rpasses;
    plan_passes(n, tc, true, ritems, rpasses);
    for (const PlanPass& p : rpasses)
      if (p.standalone)
        return fail(VQC_ERR_UNSUPPORTED, "serving takes parameterised gates with one target qubit (or diagonal)");
    if (packed) deferred.emplace(n, true, dtype == VQC_C64, rpasses);
    serialize_plan<R, M, true>(n, dtype, rpasses, rp.adj, &rp.accs, deferred ? &*deferred : nullptr, packed);
    rp.adj_max = shape_max(rp.adj);
  }
  rp.M = M;
  rp.ntiles = int64_t(1) << (n - M);
  return VQC_OK;
}

static int build_plan_any(int n, int dtype, const std::vector<GateSpec>& fspecs, const std::vector<GateSpec>& rspecs,
                          const std::vector<std::vector<ParamInfo>>& params, bool want_grad, bool packed,
                          ReqPlan& rp) {
  switch (tile_config(dtype, n).M + (dtype == VQC_C64 ? 0 : 100)) {
    case 12: return build_plan_tm<float, 12>(n, dtype, fspecs, rspecs, params, want_grad, packed, rp);
    case 11: return build_plan_tm<float, 11>(n, dtype, fspecs, rspecs, params, want_grad, packed, rp);
    case 10: return build_plan_tm<float, 10>(n, dtype, fspecs, rspecs, params, want_grad, packed, rp);
    case 9: return build_plan_tm<float, 9>(n, dtype, fspecs, rspecs, params, want_grad, packed, rp);
    case 111: return build_plan_tm<double, 11>(n, dtype, fspecs, rspecs, params, want_grad, false, rp);
    case 110: return build_plan_tm<double, 10>(n, dtype, fspecs, rspecs, params, want_grad, false, rp);
    default: return build_plan_tm<double, 9>(n, dtype, fspecs, rspecs, params, want_grad, false, rp);
  }
}

// The compiled batch kernels of a packed plan's passes (false when one has
// none); compile = false only looks them up.
static bool plan_kernels(int M, bool adj, const SerialPlan& sp, std::vector<const void*>& ks, bool compile) {
  std::vector<JitPassRef> refs(sp.locs.size());
  for (size_t i = 0; i < sp.locs.size(); ++i)
    refs[i] = JitPassRef{(const DevStageF*)(sp.buf.data() + sp.locs[i].stages), sp.locs[i].shape.nstages,
                         (const DevOp*)(sp.buf.data() + sp.locs[i].ops), sp.locs[i].shape.npool};
  if (jit_pass_kernels(M, adj, refs, ks, true, compile)) return false;
  for (const void* k : ks)
    if (!k) return false;
  return true;
}

// Serving compiles the passes of requests of at least 2^18 amplitudes (where
// the device time of a mix concentrates); smaller requests share the generic
// kernel's single launch per step kind.
constexpr int kServeJitMinQubits = 18;

int serve_build_plan(int n, int dtype, const std::vector<GateSpec>& fspecs, const std::vector<GateSpec>& rspecs,
                     const std::vector<std::vector<ParamInfo>>& params, bool want_grad, bool compiled, ReqPlan& rp,
                     ReqPlan* to_compile) {
  if (n < kMinTileBits || n > 40) return fail(VQC_ERR_UNSUPPORTED, "serving takes 9 to 40 qubits");
  if (compiled && dtype == VQC_C64 && n >= kServeJitMinQubits && jit_available()) {
    int rc = build_plan_any(n, dtype, fspecs, rspecs, params, want_grad, true, rp);
    if (rc) return rc;
    if (plan_kernels(rp.M, false, rp.fwd, rp.fwd_k, false) &&
        (!want_grad || plan_kernels(rp.M, true, rp.adj, rp.adj_k, false)))
      return VQC_OK;
    // not compiled yet: this request runs the classic plan on the generic kernel
    if (to_compile) *to_compile = std::move(rp);
    rp = ReqPlan();
  }
  return build_plan_any(n, dtype, fspecs, rspecs, params, want_grad, false, rp);
}

void serve_compile_plan(const ReqPlan& packed, bool want_grad) {
  std::vector<const void*> ks;
  plan_kernels(packed.M, false, packed.fwd, ks, true);
  if (want_grad) plan_kernels(packed.M, true, packed.adj, ks, true);
}

int serve_jit_gridx(int M, bool adj, const std::vector<const void*>& ks, const SerialPlan& sp, int64_t ntiles,
                    int device) {
  int grid = ks.empty() ? device_info(device).sms : 1 << 30;
  for (size_t i = 0; i < ks.size(); ++i)
    grid = std::min(grid, kernel_grid(device, ks[i], 1 << (M - kRegBits),
                                      pass_smem(sizeof(float2), M, adj, sp.locs[i].shape)));
  return (int)std::max<int64_t>(1, std::min<int64_t>(ntiles, grid));
}

size_t serve_pass_smem(int dtype, int M, bool adj, const PassShape& shape) {
  return pass_smem(dtype == VQC_C64 ? sizeof(float2) : sizeof(double2), M, adj, shape);
}

int serve_launch_jit(int M, bool adj, const void* kernel, const TileItem* d_items, int nitems, int gridx,
                     size_t smem, cudaStream_t stream) {
  int device = 0;
  VQC_CK(cudaGetDevice(&device));
  if (int rc = allow_smem(device, kernel)) return rc;
  ProfScope prof(stream, adj ? "serve_tile_adjoint" : "serve_tile_forward", 0);
  void* args[] = {(void*)&d_items};
  VQC_CK(cudaLaunchKernel(kernel, dim3(gridx, nitems), dim3(1 << (M - kRegBits)), args, smem, stream));
  return VQC_OK;
}

static const void* batch_kernel(int dtype, bool adj) {
  if (dtype == VQC_C64) return adj ? (const void*)k_tile_batch<float, true> : (const void*)k_tile_batch<float, false>;
  return adj ? (const void*)k_tile_batch<double, true> : (const void*)k_tile_batch<double, false>;
}

int serve_tile_gridx(int dtype, int M, bool adj, const PassShape& maxs, int64_t max_ntiles, int device) {
  const size_t smem = serve_pass_smem(dtype, M, adj, maxs);
  const int g = kernel_grid(device, batch_kernel(dtype, adj), 1 << (M - kRegBits), smem);
  return (int)std::max<int64_t>(1, std::min<int64_t>(max_ntiles, g));
}

int serve_launch_tiles(int dtype, int M, bool adj, const TileItem* d_items, int nitems, int gridx,
                       size_t smem, cudaStream_t stream) {
  const void* k = batch_kernel(dtype, adj);
  int device = 0;
  VQC_CK(cudaGetDevice(&device));
  if (int rc = allow_smem(device, k)) return rc;
  ProfScope prof(stream, adj ? "serve_tile_adjoint" : "serve_tile_forward", 0);
  void* args[] = {(void*)&d_items};
  VQC_CK(cudaLaunchKernel(k, dim3(gridx, nitems), dim3(1 << (M - kRegBits)), args, smem, stream));
  return VQC_OK;
}

int serve_launch_reduce(const RedItem* d_items, int nitems, int maxslots, cudaStream_t stream) {
  if (nitems == 0 || maxslots == 0) return VQC_OK;
  k_reduce_slots_batch<<<dim3(maxslots, nitems), 256, 0, stream>>>(d_items);
  VQC_CK(cudaGetLastError());
  return VQC_OK;
}

}  // namespace vqc
