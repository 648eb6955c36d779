"""The per-thread cache of launch plans (csrc/nf4ll_gemm_shared.cuh, KeptPlans), compiled for the host by itself."""
import pathlib
import shutil
import subprocess

import pytest

SOURCE = pathlib.Path(__file__).parent.parent / "decentrik_prime_b200" / "csrc" / "nf4ll_gemm_shared.cuh"
MAIN = r"""
#include <cstdint>
#include <cstdio>
%s
struct P { int v; };
int main() {
  static KeptPlans<P, 2> kept;
  int searches = 0;
  auto get = [&](int64_t a, bool ok) {
    const int64_t key[2] = {a, 7};
    P p{};
    const bool found = kept.get(key, &p, [&](P* q) { ++searches; q->v = static_cast<int>(a); return ok; });
    return found && p.v == a;
  };
  if (get(1, false) || searches != 1) return 1;      // none yet
  if (!get(1, true) || searches != 2) return 2;      // asked again, now kept
  if (!get(1, false) || searches != 2) return 3;
  for (int64_t i = 2; i < 5000; ++i)                 // every set overflows; the plan that stays in use stays kept
    if (!get(i, true) || !get(1, false)) return 4;
  return searches == 2 + 4998 ? 0 : 5;
}
"""


def test_plans_are_kept_once_found(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    text = SOURCE.read_text()
    start = text.index("template <typename P, int KEYS>")
    (tmp_path / "kept.cpp").write_text(MAIN % text[start:text.index("\n};\n", start) + 4])
    exe = tmp_path / "kept"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-o", str(exe), str(tmp_path / "kept.cpp")], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
