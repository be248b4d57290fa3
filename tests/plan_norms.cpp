// Plans circuits on the host and prints the range of the deferred norm over the
// passes of the forward and of the reverse sweep, in the order the ops run, the
// rows of the reverse sweep and a hash of the passes' structure
// (test_plan_norms.py).
//   plan_norms <family> <qubits> <layers> <seed>
// families: blocks2, blocks3 (RZ RY RZ on every qubit, CZ inside blocks, RY a
// parameter in every tenth layer), pi (RX(pi) rounded to float, CZ brickwork,
// RX a parameter in every fourth layer), u3 (U3 and CZ brickwork; in every third
// layer the U3 of one qubit lies next to theta = pi, 1e-8 to 1e-2 off).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>

#include "tile_plan.cuh"

using namespace vqc;

int main(int argc, char** argv) {
  if (argc != 5) return 2;
  const std::string fam = argv[1];
  const int n = std::atoi(argv[2]), layers = std::atoi(argv[3]);
  std::mt19937 rng(std::atoi(argv[4]));
  std::vector<vqc_gate> gates;
  std::vector<double> mats;
  std::vector<vqc_param> params;
  auto put = [&](const std::vector<cd>& U) {
    const int at = (int)mats.size();
    for (cd u : U) mats.push_back(u.real()), mats.push_back(u.imag());
    return at;
  };
  auto add = [&](std::vector<int> pos, const std::vector<cd>& U) {
    vqc_gate g{};
    g.nq = (int)pos.size();
    for (size_t i = 0; i < pos.size(); ++i) g.pos[i] = pos[i];
    g.mat = put(U);
    gates.push_back(g);
  };
  auto param = [&](const std::vector<cd>& dU) {
    vqc_param p{};
    p.gate = (int)gates.size() - 1;
    p.kind = VQC_PARAM_DERIVATIVE;
    p.dmat = put(dU);
    params.push_back(p);
  };
  auto angle = [&]() { return std::uniform_real_distribution<double>(0, 2 * M_PI)(rng); };
  const cd i(0, 1);
  auto rz = [&](int q) {
    const double t = angle() / 2;
    add({q}, {std::polar(1.0, -t), 0, 0, std::polar(1.0, t)});
  };
  for (int l = 0; l < layers; ++l) {
    for (int q = 0; q < n; ++q) {
      if (fam == "pi") {
        const double t = (double)(float)M_PI / 2, c = std::cos(t), s = std::sin(t);
        add({q}, {c, -i * s, -i * s, c});
        if (l % 4 == 1) param({-s / 2, -i * c / 2.0, -i * c / 2.0, -s / 2});
      } else {
        double t = angle() / 2;
        if (fam == "u3") {
          if (l % 3 == 0 && q == (5 * l + 3) % n) t = M_PI / 2 - std::pow(10.0, -2 - 6 * t / M_PI);
          const double c = std::cos(t), s = std::sin(t), p = angle(), m = angle();
          add({q}, {c, -std::polar(s, m), std::polar(s, p), std::polar(c, p + m)});
          continue;
        }
        const double c = std::cos(t), s = std::sin(t);
        rz(q);
        add({q}, {c, -s, s, c});
        if (l % 10 == 5) param({-s / 2, -c / 2, c / 2, -s / 2});
        rz(q);
      }
    }
    const int block = fam == "blocks2" ? 2 : (fam == "blocks3" ? 3 : 0);
    for (int q = block ? 0 : l % 2; q + 1 < n; q += block ? 1 : 2)
      if (!block || q / block == (q + 1) / block) add({q, q + 1}, {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0, 0, 0, -1});
  }
  std::vector<GateSpec> fwd(gates.size()), rev;
  std::vector<std::vector<ParamInfo>> per_gate;
  for (size_t g = 0; g < gates.size(); ++g)
    if (analyze_gate(n, gates[g].nq, gates[g].pos, mats.data() + gates[g].mat, false, fwd[g])) return 1;
  if (prepare_reverse(n, gates.data(), (int)gates.size(), mats.data(), params.data(), (int)params.size(), rev, per_gate))
    return 1;
  ReqPlan classic, packed;
  if (serve_build_plan(n, VQC_C64, fwd, rev, per_gate, true, true, classic, &packed)) return 1;
  if (packed.fwd.locs.empty()) return 3;  // (no run-time compiler here: nothing is deferred)
  double lo = 1, hi = 1;
  for (const AccRef& a : packed.accs) lo = std::min(lo, std::sqrt(a.scale)), hi = std::max(hi, std::sqrt(a.scale));
  lo = std::min(lo, packed.adj.norm_lo), hi = std::max(hi, packed.adj.norm_hi);
  uint64_t hash = 1469598103934665603ull;
  for (const SerialPlan* sp : {&packed.fwd, &packed.adj})
    for (const PassLoc& l : sp->locs) {
      const DevOp* ops = (const DevOp*)(sp->buf.data() + l.ops);
      for (int o = 0; o < l.shape.nops; ++o)
        for (int v : {ops[o].code, ops[o].mat, ops[o].rmask}) hash = (hash ^ (uint32_t)v) * 1099511628211ull;
    }
  std::printf("%.6e %.6e %.6e %.6e %zu %016llx\n", packed.fwd.norm_lo, packed.fwd.norm_hi, lo, hi, packed.accs.size(),
              (unsigned long long)hash);
  return 0;
}
