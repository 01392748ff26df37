"""Rules of the host layer and of the kernels' work split that need no GPU: the headers that hold them are compiled with the host
compiler into a small library and called here."""
import ctypes as C
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "micro-expert-router-ssd-streamed-moe-mer_b200", "csrc")

SOURCE = r"""
#include <cuda_runtime.h>
#include "passes.cuh"
#include "replay_table.h"
using Table = ReplayTable<const char *>;
static int g_destroyed;
static const char *const GRAPH = "graph";
extern "C" {
void *table_new() { return new Table(); }
void table_delete(void *t) { delete static_cast<Table *>(t); }
// One call: 0 plain launches, 1 captured now, 2 replayed.
int table_call(void *t, uint32_t layer, size_t n_tokens, size_t x, size_t out, size_t tag, uint32_t from) {
  Table &tab = *static_cast<Table *>(t);
  auto *c = tab.occurrence(CallKey{layer, n_tokens, (const void *)x, (const void *)out, (const void *)tag, nullptr}, from);
  if (!c) return 0;
  if (c->exec) return 2;
  tab.captured(c, GRAPH, 3, [](const char *) { g_destroyed++; });
  return 1;
}
int table_drop(void *t) {
  g_destroyed = 0;
  static_cast<Table *>(t)->drop([](const char *) { g_destroyed++; });
  return g_destroyed;
}
size_t table_graphs(void *t) { return static_cast<Table *>(t)->graphs(); }
size_t table_size(void *t) { return static_cast<Table *>(t)->size(); }
// The passes of a group of n pairs, as the grouping kernels write them; returns their number.
uint32_t cut(uint32_t n, uint32_t tpp, uint32_t *counts) {
  const PassCut c(n, tpp, 31 - __builtin_clz(tpp));
  uint32_t st = 0;
  for (uint32_t i = 0; i < c.passes; i++) st += counts[i] = c.count(i, n - st);
  return c.passes;
}
size_t max_graphs() { return Table::MAX_GRAPHS; }
size_t max_calls() { return Table::MAX_CALLS; }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src, lib = d / "rules.cpp", d / "librules.so"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC,
                           "-I", "/usr/local/cuda/include", str(src), "-o", str(lib)])
    r = C.CDLL(str(lib))
    r.table_new.restype = C.c_void_p
    for name in ("table_graphs", "table_size", "max_graphs", "max_calls"):
        getattr(r, name).restype = C.c_size_t
    for name in ("table_delete", "table_drop", "table_graphs", "table_size"):
        getattr(r, name).argtypes = [C.c_void_p]
    r.table_call.argtypes = [C.c_void_p, C.c_uint32] + [C.c_size_t] * 4 + [C.c_uint32]
    return r


@pytest.fixture
def table(rules):
    t = rules.table_new()
    yield t
    rules.table_delete(t)


@pytest.mark.parametrize("layers", [48, 61, 94])
@pytest.mark.parametrize("batches", [1, 5])
@pytest.mark.parametrize("device", [False, True])
def test_every_layer_of_a_stack_is_replayed_from_its_fourth_pass_on(rules, table, layers, batches, device):
    # the calls of a model alternate: none may push another one out of the table.  Device calls carry their buffers' addresses.
    calls = [(l, n, *((0x7f0000000000 + (l * 5 + n) * 8192, 0x7f1000000000 + l * 65536, 0) if device else (0, 0, 5)))
             for l in range(layers) for n in (1, 4, 16, 64, 256)[:batches]]
    passes = [[rules.table_call(table, *c, 3) for c in calls] for _ in range(5)]
    assert passes[0] == passes[1] == [0] * len(calls)
    assert passes[2] == [1] * len(calls)
    assert passes[3] == passes[4] == [2] * len(calls)
    assert rules.table_drop(table) == len(calls) and rules.table_graphs(table) == 0
    assert [rules.table_call(table, *c, 3) for c in calls] == [1] * len(calls)  # known calls are captured again at once


def test_calls_with_ever_new_buffers_are_never_captured_and_do_not_grow_the_table(rules, table):
    for i in range(3 * rules.max_calls()):
        assert rules.table_call(table, 0, 1, 4096 * (i + 1), 0, 0, 3) == 0
        assert rules.table_call(table, 7, 1, 1, 0, 0, 3) == min(i // 2, 1) + (i > 2)  # one among them that comes again
        assert rules.table_size(table) <= rules.max_calls()
    assert rules.table_graphs(table) == 1


def test_a_full_table_keeps_what_it_has_until_that_is_idle(rules, table):
    n, more = rules.max_graphs(), rules.max_graphs() + 200
    for _ in range(3):
        for l in range(more):
            rules.table_call(table, l, 1, 0, 0, 1, 3)
    assert rules.table_graphs(table) == n
    for _ in range(3):  # a working set that does not fit: the same calls are replayed, nothing is captured
        assert [rules.table_call(table, l, 1, 0, 0, 1, 3) for l in range(more)] == [2] * n + [0] * (more - n)
    seen = [[rules.table_call(table, 10000 + l, 1, 0, 0, 1, 1) for l in range(100)] for _ in range(60)]  # another model
    assert seen[0] == [0] * 100 and seen[-1] == [2] * 100 and sum(map(sum, ([v == 1 for v in s] for s in seen))) == 100
    assert rules.table_graphs(table) == n


@pytest.mark.parametrize("tpp", [4, 8, 16, 32, 64, 128])
def test_the_passes_of_a_group_share_its_pairs_evenly(rules, tpp):
    counts = (C.c_uint32 * 4096)()
    for n in list(range(0, 2600)) + [4095, 4096, 4097, 10000]:
        k = rules.cut(n, tpp, counts)
        got = counts[:k]
        assert k == -(-n // tpp) and sum(got) == n and all(0 < c <= tpp for c in got), (n, got)
        if tpp < 16:
            assert got[:-1] == [tpp] * (k - 1)
        elif k:
            widths = [(c + 15) // 16 for c in got]  # of an MMA, in units of 16 columns
            assert max(widths) - min(widths) <= 1 and sum(widths) == -(-n // 16), (n, got)


def test_barriers_between_the_ctas_of_a_pair_name_their_scope():
    # an mbarrier operation without one orders memory within its own CTA only; the pair's barriers are signalled by both
    ptx, gemm = (open(os.path.join(CSRC, f)).read() for f in ("ptx.cuh", "kernels_gemm.cu"))
    for arrive in re.findall(r"mbarrier\.arrive[^ ]*shared::cluster[^ ]*", ptx + gemm):
        assert re.match(r"mbarrier\.arrive\.(relaxed|release)\.cluster\.", arrive), arrive
    for name, sem in (("mbar_wait_tmem", "relaxed"), ("mbar_wait_cluster", "acquire")):
        body = ptx[ptx.index(f"bool {name}("):]
        assert f"mbarrier.try_wait.parity.{sem}.cluster." in body[:body.index("\n}\n")]
    kernel = gemm[gemm.index("k_ffn_gemm("):]
    waits = re.findall(r"ok = (mbar_wait\w*)\(&(\w+)\[", kernel)
    crossing = {"a_full": "tmem", "acc_empty": "tmem", "acc_full": "tmem", "b_full": "cluster"}
    assert {b for _, b in waits} == {*crossing, "done", "raw_full", "raw_empty"}
    for wait, barrier in waits:
        assert wait in ({"mbar_wait_tmem", "mbar_wait_cluster"} if barrier == "done" else
                        {"mbar_wait_" + crossing[barrier]} if barrier in crossing else {"mbar_wait"}), (wait, barrier)


ACT_SOURCE = r"""
#include <cuda_runtime.h>
#include "act_rows.h"
extern "C" void act_map(uint32_t rows, uint32_t K, uint32_t box_rows, uint64_t *dims, uint64_t *strides, uint32_t *box) {
  const ActMapShape a(rows, K, box_rows, 2);
  for (int i = 0; i < 4; i++) dims[i] = a.dims[i], box[i] = a.box[i];
  for (int i = 0; i < 3; i++) strides[i] = a.strides[i];
}
extern "C" uint64_t act_byte(uint32_t rows, uint32_t row, uint32_t k, uint32_t part) {
  return (act_rows_hi(rows, row, k / 4) + part * act_rows_lo(rows)) * 8 + k % 4 * 2;
}
extern "C" uint32_t act_row() { return ACT_ROW; }
"""


@pytest.mark.parametrize("rows,K", [(12, 128), (33, 384), (2048 * 8, 2048), (2048 * 8, 768), (37 * 9, 14336), (4096 * 9, 7168), (65536, 16384)])
def test_the_activations_tensor_map_is_one_of_the_documented_kind(tmp_path, rows, K):
    # the encoder's description builds a stride from the one before it: a map whose strides fall may be refused, and the layer with it
    src, lib = tmp_path / "act.cpp", tmp_path / "libact.so"
    src.write_text(ACT_SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, "-I", "/usr/local/cuda/include", str(src), "-o", str(lib)])
    r = C.CDLL(str(lib))
    r.act_byte.restype = C.c_uint64
    dims, strides, box = (C.c_uint64 * 4)(), (C.c_uint64 * 3)(), (C.c_uint32 * 4)()
    for box_rows in range(8, 129, 8):
        r.act_map(rows, K, box_rows, dims, strides, box)
        assert list(box) == [64, box_rows, 2, 2] and box[0] * 2 <= 128 and all(1 <= b <= 256 for b in box)
        assert dims[0] * dims[1] * dims[2] * dims[3] == 2 * rows * K and dims[1] == rows and dims[3] % 2 == 0
        assert strides[0] == dims[0] * 2 and all(strides[i] == strides[i - 1] * dims[i] >= dims[i] for i in (1, 2))
        assert all(s % 16 == 0 and s < 2 ** 40 for s in strides)
    # the kernel that writes the rows puts a value where the map looks for it
    for row in {0, 1, 7, rows // 2, rows - 1}:
        for k in {0, 3, 63, 64, 127, K // 2, K - 1}:
            for part in (0, 1):
                assert r.act_byte(rows, row, k, part) == k % 64 * 2 + row * strides[0] + part * strides[1] + k // 64 * strides[2] < 4 * rows * K
    assert r.act_row() * 8 == strides[0]
