// What the re-planner and the table builder make of a program, as JSON: no device needed.
//   plan_probe BLOB LANES
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <iterator>

#include "loader.h"
#include "plan_format.h"
#include "replan.h"

int main(int argc, char **argv) {
  if (argc != 3) return 2;
  std::ifstream f(argv[1], std::ios::binary);
  const std::vector<uint8_t> blob((std::istreambuf_iterator<char>(f)), {});
  b2::VmProgram p, q;
  b2::DeviceTables wire, t;
  b2::ReplanStats st;
  std::string err;
  bool unimpl = false;
  if (!b2::VmProgram::Parse(blob.data(), blob.size(), &p, &err) || !b2::BuildDeviceTables(p, 0, &wire, &err, &unimpl)) {
    std::fprintf(stderr, "%s\n", err.c_str());
    return 1;
  }
  const bool planned = b2::Replan(p, static_cast<uint32_t>(std::atoi(argv[2])), &q, &st);
  if (!planned) { std::printf("{\"planned\": false, \"tasks\": []}\n"); return 0; }
  // (an arena that does not start at address 0, which stands for no buffer)
  if (!b2::BuildPlannedTables(q, 1u << 20, &t, &err, &unimpl)) {
    std::fprintf(stderr, "planned: %s\n", err.c_str());
    return 1;
  }
  std::printf("{\"planned\": true, \"gains\": %s, \"families\": %u, \"phases\": %u, \"tasks\": [", b2::PlanGains(t) ? "true" : "false", t.families, st.phases);
  for (uint32_t i = 0; i < t.tasks.size(); ++i) {
    const b2::DTask &d = t.tasks[i];
    const uint64_t *w = &t.desc[d.desc];
    std::printf("%s{\"op\": %u", i ? ", " : "", d.op);
    if (d.op == b2::kTopFuseRows) {
      const b2::DFuse &u = *reinterpret_cast<const b2::DFuse *>(w);
      uint32_t stage = 0;
      for (const b2::DEntry &e : t.entries)
        if (e.task == i && u.pipe.flags) {
          const uint32_t esz = static_cast<uint32_t>(b2::DtypeSize(u.pipe.dt));
          stage = std::max(stage, 2u * b2::pipe_shape(u.pipe.flags, esz, u.vec != 0u, u.cols, std::min(e.tile_hi, u.rows) - e.tile_lo, 512u).buf_bytes);
        }
      std::printf(", \"rows\": %u, \"cols\": %u, \"pipe\": %u, \"flat\": %u, \"steps\": %u, \"stage\": %u, \"room\": %u", u.rows, u.cols, u.pipe.flags, u.flat, u.n_steps, stage, b2::kPlanStageBytes);
    } else if (d.op == b2::kTopSgemm || d.op == b2::kTopSkinny) {
      const b2::DSgemm &g = *reinterpret_cast<const b2::DSgemm *>(w);
      std::printf(", \"mnk\": [%u, %u, %u], \"viewed\": [%u, %u], \"epi\": %u, \"dt1\": %u, \"shape\": %u", g.M, g.N, g.K, g.a.viewed, g.b.viewed, g.epi, g.dt1, g.shape);
    } else if (d.op == b2::kTopGemm) {
      const b2::DGemm &g = *reinterpret_cast<const b2::DGemm *>(w);
      std::printf(", \"prob\": [");
      for (uint32_t k = 0; k < g.n_prob; ++k)
        std::printf("%s{\"mnk\": [%u, %u, %u], \"epi\": %u, \"dt1\": %u, \"form\": %u}", k ? ", " : "", g.prob[k].M, g.prob[k].N, g.prob[k].K, g.prob[k].epi, g.prob[k].dt1, g.prob[k].form);
      std::printf("]");
    }
    std::printf(", \"cut\": [");
    bool first = true;
    for (uint32_t l = 0; l < t.lanes.size(); ++l)
      for (uint32_t k = 0; k < t.lanes[l].count; ++k) {
        const b2::DEntry &e = t.entries[t.lanes[l].off + k];
        if (e.task != i) continue;
        std::printf("%s[%u, %u, %u]", first ? "" : ", ", l, e.tile_lo, e.tile_hi);
        first = false;
      }
    std::printf("]}");
  }
  std::printf("]}\n");
  return 0;
}
