"""Step graphs are captured when a call first needs them, those of its own kind
only: a run that steps through the host call does not also pay for the resident
steps' graphs. step_graph itself, run on the CPU with its captures recorded."""
from tests import host_source as hs

STUBS = r"""
using cudaGraphExec_t = const char*;
struct Engine {
  cudaGraphExec_t graph[2] = {}, graph_up[2] = {}, graph_host[2] = {};
  bool graphs_valid = false, stats_on_device = false;
  int cur = 0, steps = 0, stream = 0;
};
constexpr int FL_OK = 0;
#define TRY(x) if (int st = (x)) return st
int captures = 0, fail_at = -1;
const char* launched = "";
int build_graph(Engine* e, int par, cudaGraphExec_t* out, bool cfl_first, bool host) {
  if (captures++ == fail_at) return 9;
  static const char* names[] = {"resident0", "resident1", "host0", "host1", "", "", "up0", "up1"};
  *out = names[4 * cfl_first + 2 * host + par];
  return FL_OK;
}
void destroy_step_graphs(Engine* e) {
  for (auto* g : {e->graph, e->graph_up, e->graph_host}) g[0] = g[1] = nullptr;
  e->graphs_valid = false;
}
int cudaGraphLaunch(cudaGraphExec_t g, int) { launched = g; return 0; }
int cuda_status(Engine*, int st, const char*) { return st; }
"""

MAIN = r"""
int main(int argc, char** argv) {
  auto calls = [](const char* what) {  // u: host call with fields, h: host call without, r: resident step, d: parameters changed
    Engine e;
    captures = 0;
    std::string line;
    for (const char* c = what; *c; c++) {
      const int before = captures;
      if (*c == 'd') { destroy_step_graphs(&e); continue; }
      if (*c == 'u') e.cur = 0;
      const int st = step_graph(&e, *c == 'u', *c != 'r');
      line += std::string(st ? "failed" : launched) + " " + std::to_string(captures - before) + (c[1] ? ", " : "");
    }
    std::printf("%s\n", line.c_str());
  };
  calls("rrr");
  calls("hhh");
  calls("uu");
  calls("uhr");
  calls("rdr");
  fail_at = 1;
  calls("rrr");
}
"""


def test_a_call_builds_the_graphs_of_its_own_kind(tmp_path):
    text = hs.source("fl_engine.cu")
    out = hs.run(tmp_path, "#include <string>\n" + STUBS + hs.block(text, "int step_graph(Engine* e") + MAIN).splitlines()
    assert out == [
        "resident0 2, resident1 0, resident0 0",  # both parities at the first step
        "host0 2, host1 0, host0 0",
        "up0 1, up0 0",
        "up0 1, host1 2, resident0 2",
        "resident0 2, resident1 2",
        "failed 2, resident0 1, resident1 0",
    ]
