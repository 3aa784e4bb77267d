"""The growth of device arrays when allocations fail, over an allocator that
fails where it is told to (compiled here with g++; no GPU): whatever fails, no
capacity claims an array that is not there, the next call makes up for it, and
temporaries are returned."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "icflow_b200" / "csrc"

PROBE = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include "icf_grow.cuh"

struct fake {
  int fail_at = -1, calls = 0;
  std::map<void *, size_t> live;
  bool alloc(void **p, size_t bytes) {
    if (calls++ == fail_at) return false;
    *p = std::malloc(bytes);
    live[*p] = bytes;
    return true;
  }
  void free(void *p) {
    if (!p) return;
    if (!live.erase(p)) std::abort();
    std::free(p);
  }
};

#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); std::exit(1); } } while (0)

static int temps(fake &m, int n) {
  icf_temps<fake> t(m);
  int *a;
  double *b;
  for (int i = 0; i < n; i++)
    if (!(i % 2 ? t.alloc(&a, 10 + i) : t.alloc(&b, 3))) return 1;
  return 0;
}

int main() {
  for (int fail = -1; fail < 3; fail++) {
    fake m;
    int *a = nullptr;
    double *b = nullptr;
    char *c = nullptr;
    long long cap = 0;
    auto have = [&](long long n) {  // what a call that needs n elements finds
      if (n > cap && !icf_grow_all(m, &cap, n, &a, &b, &c)) return false;
      CHECK(m.live.count(a) && m.live[a] >= sizeof(int) * n);
      CHECK(m.live.count(b) && m.live[b] >= sizeof(double) * n);
      CHECK(m.live.count(c) && m.live[c] >= (size_t)n);
      return true;
    };
    CHECK(have(100) && cap == 100);
    CHECK(have(40) && cap == 100 && m.calls == 3);
    m.fail_at = fail < 0 ? -1 : m.calls + fail;
    CHECK(have(1000) == (fail < 0));
    if (fail >= 0) CHECK(cap == 0);
    m.fail_at = -1;
    CHECK(have(40));  // fewer than before the failure
    CHECK(have(1000) && cap == 1000);
    int small_cap = 7;
    CHECK(icf_grow_all(m, &small_cap, 50, &a) && small_cap == 50);
    m.fail_at = fail < 0 ? -1 : m.calls + fail;
    CHECK(icf_grow_all(m, &cap, 20, icf_of(&a, 60), icf_of(&b, 21), icf_of(&c, 20)) == (fail < 0));
    if (fail >= 0) CHECK(cap == 0);
    if (fail < 0) CHECK(cap == 20 && m.live[a] == 60 * sizeof(int) && m.live[b] == 21 * sizeof(double) && m.live[c] == 20);
  }
  for (int n = 0; n <= 9; n++)
    for (int fail = -1; fail < n; fail++) {
      fake m;
      m.fail_at = fail;
      CHECK(temps(m, n) == (fail >= 0 || n > 8));
      CHECK(m.live.empty());
    }
  return 0;
}
"""


def test_failed_allocations(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    (tmp_path / "probe.cpp").write_text(PROBE)
    exe = tmp_path / "probe"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", str(CSRC), str(tmp_path / "probe.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


CAPS = {"icf_pattern.cu": "rows_cap|items_cap|cols_cap|cr_cap|ks_cap|imp_pos_cap|s2m_cap|rhs_cap|slices_cap",
        "icf_solve.cu": "[a-z]+_cap", "icf_broad.cu": r"k?cap|\w+_cap", "icf_contact.cu": r"\w+_cap",
        "icf_api.cu": "pairs_cap|imp_cap|imp_built_cap"}


@pytest.mark.parametrize("name", sorted(CAPS))
def test_arrays_of_one_capacity_grow_together(name):
    """The capacities of the contact buffers, of the structure's merge and of the
    solver are set by the growth of their arrays, never by hand (but to zero)."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    text = re.sub(r"const long long c\w* =|\b(?:halo_cap|cap_cells)\b", "", text)  # (sizes, not capacities)
    assert not re.findall(rf"\b(?:{CAPS[name]})\s*=(?![=]| 0;)[^;]*", text)


def test_solver_allocates_by_capacity():
    """No array of the solver hangs on whether another one is there, and its
    temporaries are held by icf_temps."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "icf_solve.cu").read_text())
    assert not re.findall(r"\bcuda(?:MallocAsync|FreeAsync)\b", text)
    for m in re.finditer(r"cudaMalloc\(&(\S+?),", text):  # each under a check of its own
        assert f"if (!{m.group(1)}) ICF_CUDA(ctx, cudaMalloc(&{m.group(1)}," in text, m.group(1)
