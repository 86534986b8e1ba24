// The autotuner (gpr_tune.cc) against a library that only keeps books: a graph's
// sweeps take as long as the bins it was created with say, so what the search
// compares and what it returns can be read without a device.
//
//   tune_driver single|batch <best chunk> <best hot> <cache>
//
// prints the layouts in the order in which graphs are created ("create ...") and
// the result ("pick ...").  A graph takes 10 ms per sweep, 8 with the given chunk and
// chunk_min, 8 with the given prefix, 6 with both (0: the defaults are the fastest).
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#include "gpr.h"

static int g_chunk, g_hot;

struct gpr_graph {
  gpr_layout_opts l;
};
struct gpr_multigraph {
  gpr_layout_opts l;
};

namespace gpr {
void set_error(const char *, ...) {}
}  // namespace gpr

static void show(const char *what, const gpr_layout_opts &l) {
  printf("%s %d %d %d %d %d\n", what, l.sell_max, l.chunk, l.chunk_min, l.hot_entries, l.flags);
}

static double sweep_ms(const gpr_layout_opts &l) {
  double ms = 10.0;
  if (g_chunk && l.chunk == g_chunk && l.chunk_min == g_chunk) ms -= 2.0;
  if (g_hot && l.hot_entries == g_hot) ms -= 2.0;
  const bool defaults = l.chunk == 0 && l.chunk_min == 0 && l.hot_entries == 0;
  if (!g_chunk && !g_hot && !defaults) ms += 1.0;
  if (l.flags) ms += 20.0;
  return ms;
}

extern "C" {
int gpr_memcpy(void *dst, const void *src, size_t bytes) {
  memcpy(dst, src, bytes);
  return GPR_OK;
}
int gpr_pr_opts_default(gpr_pr_opts *o) {
  memset(o, 0, sizeof(*o));
  return GPR_OK;
}
int gpr_graph_create_ex(int, long long, const int *, const int *, const int *,
                        const gpr_layout_opts *l, gpr_graph **out) {
  show("create", *l);
  *out = new gpr_graph{*l};
  return GPR_OK;
}
int gpr_graph_destroy(gpr_graph *g) {
  delete g;
  return GPR_OK;
}
int gpr_pagerank(gpr_graph *g, float *, const gpr_pr_opts *o, gpr_pr_stats *st) {
  memset(st, 0, sizeof(*st));
  st->iterations = o->max_iter;
  st->loop_ms = sweep_ms(g->l) * o->max_iter;
  return GPR_OK;
}
int gpr_multigraph_create(int, const int *, long long, const int *, const int *, const int *,
                          const gpr_layout_opts *l, gpr_multigraph **out) {
  show("create", l[0]);
  *out = new gpr_multigraph{l[0]};
  return GPR_OK;
}
int gpr_multigraph_destroy(gpr_multigraph *g) {
  delete g;
  return GPR_OK;
}
int gpr_multigraph_pagerank(gpr_multigraph *g, float *, const gpr_pr_opts *o, int *, double *,
                            gpr_pr_stats *st) {
  memset(st, 0, sizeof(*st));
  st->loop_ms = sweep_ms(g->l) * o->max_iter;
  return GPR_OK;
}
}

int main(int argc, char **argv) {
  if (argc != 5) return 2;
  g_chunk = atoi(argv[2]);
  g_hot = atoi(argv[3]);
  const int m = 1000;
  std::vector<int> rp(m + 1), col(8 * m, 0), od(m, 8);
  for (int v = 0; v <= m; ++v) rp[v] = 8 * v;
  gpr_tune_result r;
  gpr_layout_opts lay;
  if (!strcmp(argv[1], "single")) {
    if (gpr_tune_graph(m, 8LL * m, rp.data(), col.data(), od.data(), argv[4], 4, &r) != GPR_OK)
      return 1;
    lay = r.layout;
  } else {
    const int voff[2] = {0, m};
    if (gpr_tune_multigraph(1, voff, 8LL * m, rp.data(), col.data(), od.data(), argv[4], 4, &lay,
                            &r) != GPR_OK)
      return 1;
  }
  show("pick", lay);
  printf("ms %g %g cached %d\n", r.ms_per_sweep, r.default_ms_per_sweep, r.from_cache);
  return 0;
}
