"""How the resident solver deals a system's rows to the CTAs of a team
(csrc/team_plan.h), compiled for the host: every row comes back from the
plan with its own diagonal place and its columns in slot order."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "shyfemcm-ismar_b200" / "csrc"

HARNESS = """
#include "team_plan.h"
using namespace shy;
// the plan of one system, read back: per row of the shares its global row,
// diagonal place, count of the others and their global columns in slot order
extern "C" int deal(int nk, const int *rowptr, const int *col, const float *xy, int T, int rows, int ghosts, int entries,
                    int *cut, int *row, int *place, int *count, int *cols) {
  const TeamShape sh = {rows, ghosts, entries, T};
  TeamBasin B;
  team_basin(rowptr, col, xy, 0, nk, T, sh, B);
  if (B.most > ghosts) return -B.most;
  int n = 0, t = 0;
  for (int r = 0; r <= T; r++) cut[r] = B.cut[r];
  for (int r = 0; r < T; r++)
    for (int j = B.cut[r]; j < B.cut[r + 1]; j++) {
      row[j] = B.rows[j] & 0x7fffffff;
      place[j] = dpos_place(B.dpos[j]);
      count[j] = dpos_count(B.dpos[j]);
      for (int k = 0; k < std::min(count[j], entries) + B.tcount[j]; k++) {
        const int l = k < entries ? B.lcol[(size_t)entries * j + k] / 4 : B.tcol[t++];
        cols[n++] = l < rows ? B.rows[B.cut[r] + l] & 0x7fffffff : B.ghost[B.gptr[r] + l - rows];
      }
    }
  return n;
}
// n pieces of work on nt threads, the one numbered `bad` throwing: how many
// were done, negative when on_threads says that one threw
extern "C" int pieces(int n, int nt, int bad) {
  std::atomic<int> done{0};
  const bool ok = on_threads(n, nt, [&](int i) {
    if (i == bad) throw std::bad_alloc();
    done++;
  });
  return ok ? (int)done : -(int)done;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", f"-I{CSRC}", str(d / "plan.cpp"), "-o",
                    str(d / "plan.so")], check=True)
    lib = C.CDLL(str(d / "plan.so"))
    lib.path = str(d / "plan.so")
    return lib


@pytest.fixture(scope="module")
def deal(lib):
    def call(pattern, xy, T, rows=2048, ghosts=512, entries=8):
        nk = len(pattern)
        rowptr = np.r_[0, np.cumsum([len(p) for p in pattern])].astype(np.int32)
        col = np.concatenate(pattern).astype(np.int32)
        xy = np.ascontiguousarray(xy, np.float32)
        out = [np.zeros(n, np.int32) for n in (T + 1, nk, nk, nk, len(col))]
        p = lambda a: a.ctypes.data_as(C.c_void_p)
        n = lib.deal(nk, p(rowptr), p(col), p(xy), T, rows, ghosts, entries, *[p(a) for a in out])
        return n, out
    return call


def hub_pattern(spokes, n, hub):
    """n rows on a ring, each joined to its two neighbours, `spokes` of them
    to row `hub` as well."""
    ring = [i for i in range(n) if i != hub]
    adj = [{i} for i in range(n)]
    for q, i in enumerate(ring):
        j = ring[(q + 1) % len(ring)]
        adj[i].add(j)
        adj[j].add(i)
    for i in ring[:spokes]:
        adj[i].add(hub)
        adj[hub].add(i)
    a = 2 * np.pi * np.arange(n) / n
    xy = np.stack([np.cos(a), np.sin(a)], 1)
    xy[hub] = 0.0
    return [np.array(sorted(s)) for s in adj], xy


def check(pattern, n, out):
    cut, row, place, count, cols = out
    assert sorted(row) == list(range(len(pattern))) and cut[0] == 0 and cut[-1] == len(pattern)
    at = 0
    for j, i in enumerate(row):
        want = pattern[i]
        assert place[j] == list(want).index(i), (i, place[j])
        assert count[j] == len(want) - 1, (i, count[j])
        assert np.array_equal(cols[at:at + count[j]], want[want != i]), i
        at += count[j]
    assert at == n


@pytest.mark.parametrize("spokes", [8, 9, 254, 255, 256, 257, 300, 1000])
@pytest.mark.parametrize("last", [True, False])
def test_rows_of_any_length(deal, spokes, last):
    """A hub whose neighbours are all numbered below it (the diagonal in the
    last place) or all above it (in the first)."""
    n = 1400
    pattern, xy = hub_pattern(spokes, n, n - 1 if last else 0)
    for T, entries in ((1, 8), (1, 26)):
        check(pattern, *deal(pattern, xy, T, entries=entries))


@pytest.mark.parametrize("T", [2, 3, 7])
def test_shares_of_a_hub(deal, T):
    """The same over several shares: the hub's neighbours in the others are
    ghosts, up to the number a share holds; with more the plan is refused."""
    pattern, xy = hub_pattern(400, 1400, 1399)
    check(pattern, *deal(pattern, xy, T))
    pattern, xy = hub_pattern(1300, 1400, 1399)
    n, _ = deal(pattern, xy, T)
    assert n < -512


@pytest.mark.parametrize("n,nt", [(1, 1), (1, 8), (5, 8), (64, 8), (1000, 3)])
def test_work_on_threads(lib, n, nt):
    """Every piece once; an exception in one is told and ends no other thread's."""
    assert lib.pieces(n, nt, -1) == n
    assert -n < lib.pieces(n, nt, n // 2) <= 0


def test_work_without_threads(lib):
    """A process that cannot start another thread (stacks larger than its
    address space may become) does the work on its own."""
    import resource
    import sys

    def limits():
        resource.setrlimit(resource.RLIMIT_STACK, (1 << 36, resource.RLIM_INFINITY))
        resource.setrlimit(resource.RLIMIT_AS, (1 << 32, 1 << 32))
    code = (f"import ctypes, threading\nlib = ctypes.CDLL({lib.path!r})\n"
            "try:\n    threading.Thread(target=print).start()\n    print('started')\n"
            "except RuntimeError:\n    print(lib.pieces(64, 8, -1))")
    r = subprocess.run([sys.executable, "-c", code], preexec_fn=limits, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.split() == ["64"], (r.returncode, r.stdout, r.stderr)


@pytest.mark.parametrize("T", [2, 7])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_coordinates_that_are_no_numbers(deal, bad, T):
    """Nodes without coordinates (NaN; such as no element uses) are dealt
    like nodes at the origin; infinite ones by their order."""
    pattern, xy = hub_pattern(100, 1400, 1399)
    rng = np.random.default_rng(5)
    xy[rng.random(1400) < 0.3, 0] = bad
    xy[rng.random(1400) < 0.3, 1] = bad
    n, out = deal(pattern, xy, T, ghosts=1024)
    check(pattern, n, out)
    if np.isnan(bad):
        m, want = deal(pattern, np.nan_to_num(xy), T, ghosts=1024)
        assert m == n and all(np.array_equal(a, b) for a, b in zip(out, want))
