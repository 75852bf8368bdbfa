"""The device memory of a handle (csrc/lpg_devmem.h): parts of slabs are never
freed by themselves.  On the CPU over a recording allocator, with the requests
that lpg_create and lpg_start make for batches in which a temporary buffer is
the first part of its slab; on the GPU such batches against the oracle, bit
for bit."""

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from laser_polio_gb300 import synthetic

CSRC = Path(__file__).resolve().parent.parent / "laser_polio_gb300" / "csrc"

DRIVER = r"""
#include <stdio.h>
#include <stdlib.h>
#include <map>
#include "lpg_devmem.h"

static std::map<uint8_t*, size_t> live;   /* allocations */
static std::map<uint8_t*, size_t> parts;  /* buffers in use */
static int freed_in_use = 0;
static int take(void** p, size_t n) {
  *p = malloc(n);
  live[(uint8_t*)*p] = n;
  return 0;
}
static void release(void* p) {
  const size_t n = live.at((uint8_t*)p);
  auto q = parts.lower_bound((uint8_t*)p);
  if (q != parts.end() && q->first < (uint8_t*)p + n) freed_in_use = 1;
  live.erase((uint8_t*)p);
  free(p);
}
/* p, n bytes: inside one live allocation, beside every other buffer */
static void use(void* p, size_t n) {
  uint8_t* b = (uint8_t*)p;
  auto a = live.upper_bound(b);
  if (a == live.begin()) { puts("a buffer in freed memory"); exit(1); }
  --a;
  if (b + n > a->first + a->second) { puts("a buffer beyond its allocation"); exit(1); }
  auto q = parts.upper_bound(b);
  if (q != parts.end() && b + n > q->first) { puts("buffers overlap"); exit(1); }
  if (q != parts.begin() && (--q)->first + q->second > b) { puts("buffers overlap"); exit(1); }
  if ((uintptr_t)b & 15) { puts("a buffer off its boundary"); exit(1); }
  parts[b] = n;
}
int main(int argc, char** argv) {
  const size_t R = atoi(argv[1]), n = atoi(argv[2]), nt = atoi(argv[3]);
  DevMem m(take, release);
  auto part = [&](size_t bytes) { void* p; m.part(&p, bytes); use(p, bytes); return p; };
  auto back = [&](void* p) { parts.erase((uint8_t*)p); m.give_back(p); };
  auto up = [&](size_t bytes) {
    if (bytes > DevMem::kItemBytes) return part(bytes);
    std::vector<uint8_t> v(bytes, 1);
    void* p;
    m.upload(&p, v.data(), bytes);
    use(p, bytes);
    return p;
  };
  for (size_t r = 0; r < R; ++r) part(16 * n * n), part(8 * n); /* the networks */
  back(part(8 * n * n));
  for (size_t r = 0; r < R; ++r) { void* p; m.own(&p, 29 * 1000); use(p, 29 * 1000); } /* staging */
  void *cnt = part(8 * n), *flags = part(8);
  back(cnt), back(flags);
  for (size_t r = 0; r < R; ++r) {
    for (size_t bytes : {8 * n, 8 * n, 8 * n, 8 * (size_t)3, 8 * n, 8 * nt, 4 * n, 8 * n, 8 * n, 8 * (size_t)101,
                         4 * nt, 4 * nt, 4 * nt, 4 * nt, nt, (size_t)0, (size_t)0})
      up(bytes);
  }
  for (size_t r = 0; r < R; ++r) {
    void *a = up(4 * n), *b = up(8 * n);
    back(a), back(b);
  }
  if (freed_in_use) { puts("an allocation freed that holds buffers in use"); return 1; }
  parts.clear();
  m.clear();
  if (!live.empty()) { puts("memory left"); return 1; }
  return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("devmem")
    (d / "t.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return d / "t"


def test_no_slab_is_freed_before_its_handle(driver):
    batches = [(r, n, nt) for n in (1, 14, 44, 60, 63, 70, 79, 80, 83, 85, 88, 90, 120, 129, 300, 774)
               for r in (1, 2, 8, 9, 10, 12, 13, 16, 18, 24, 28, 33, 37, 56, 64, 99) for nt in (60, 366, 731)]
    for b in batches:
        got = subprocess.run([str(driver), *map(str, b)], capture_output=True, text=True)
        assert got.returncode == 0, (b, got.stdout)


@pytest.mark.gpu
@pytest.mark.parametrize("reps,nodes,dur", [(8, 90, 40), (10, 80, 40), (28, 300, 730)])
def test_gpu_batches_whose_tables_fill_a_slab_equal_the_oracle(reps, nodes, dur):
    from oracle_backend import run_spec_oracle

    from laser_polio_gb300._lib import Handle
    from laser_polio_gb300.engine import build_sim_spec
    from laser_polio_gb300.engine import host_columns

    specs = [build_sim_spec(synthetic.nigeria_like(n_agents=40 * nodes, n_nodes=nodes, dur=dur, seed=r))
             for r in range(reps)]
    n = specs[0].desc.nt - 1
    h = Handle([s.desc for s in specs])
    try:
        for r, s in enumerate(specs):
            h.bind_columns(r, host_columns(s))
        h.start()
        h.step(n)
        h.sync()
        for r, s in enumerate(specs):
            cols, res = host_columns(s), {k: v.copy() for k, v in s.results.items()}
            want_cols, want_res = host_columns(s), {k: v.copy() for k, v in s.results.items()}
            h.read_results(r, res)
            h.read_columns(r, cols)
            st = run_spec_oracle(s, want_cols, want_res, n)
            for k in want_res:
                assert np.array_equal(res[k], want_res[k]), (r, k)
            for k in want_cols:
                assert np.array_equal(cols[k][:st.count], want_cols[k][:st.count]), (r, k)
    finally:
        h.close()
