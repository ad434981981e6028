"""csrc/index_math.h on the host: the kernels' index arithmetic at the ends of
the int32 range, where no test would allocate the arrays, and on pointers that
no kernel may follow."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "spgemm_b200" / "csrc"


def run_cpp(tmp_path, body):
    src = tmp_path / "check.cpp"
    src.write_text('#include <cstdio>\n#include "index_math.h"\nusing namespace sg;\n' + body)
    exe = tmp_path / "check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover=all",
                    f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()


@pytest.mark.parametrize("nnz", [0, 1, 100, 2 ** 31 - 1])
def test_entry_ranges_stay_inside_the_arrays(tmp_path, nnz):
    ends = [-2 ** 31, -2 ** 31 + 1, -7, -1, 0, 1, 2, 50, 99, 100, 101, 2 ** 30, 2 ** 31 - 2, 2 ** 31 - 1]
    lit = ", ".join(f"(int)({v}ll)" for v in ends)
    out = run_cpp(tmp_path, f"""int main() {{
  const int v[] = {{{lit}}};
  for (int s : v) for (int e : v) {{ EntryRange r = entry_range(s, e, {nnz}); std::printf("%d %d ", r.begin, r.end); }}
}}""")
    got = [(int(out[i]), int(out[i + 1])) for i in range(0, len(out), 2)]
    for (s, e), (b, t) in zip([(s, e) for s in ends for e in ends], got):
        assert 0 <= b <= t <= nnz, (s, e, b, t)
        if 0 <= s <= e <= nnz:
            assert (b, t) == (s, e)


@pytest.mark.parametrize("lo,hi", [(0, 0), (0, 1), (5, 1000), (2 ** 30 - 3, 2 ** 30 + 900), (0, 2 ** 31 - 1),
                                   (2 ** 30 + 1, 2 ** 31 - 1), (2 ** 31 - 40, 2 ** 31 - 1)])
def test_lower_bound_at_any_position(tmp_path, lo, hi):
    """A row of B may begin anywhere below 2^31: lo + hi must not wrap. The
    value at position p is (p - lo) / 2, every value twice."""
    keys = sorted({0, 1, 2, (hi - lo) // 4, (hi - lo) // 2, max((hi - lo) // 2 - 1, 0), (hi - lo) // 2 + 1})
    out = run_cpp(tmp_path, f"""int main() {{
  const int lo = {lo}, hi = {hi}, keys[] = {{{', '.join(map(str, keys))}}};
  for (int key : keys) {{
    bool inside = true;
    const int r = lower_bound_at(lo, hi, key, [&](int p) {{ inside &= p >= lo && p < hi; return (p - lo) / 2; }});
    std::printf("%d %d ", r, (int)inside);
  }}
}}""")
    for k, key in enumerate(keys):
        assert out[2 * k + 1] == "1", key
        assert int(out[2 * k]) == min(lo + 2 * key, hi), key


LAST = 2 ** 31 - 1


@pytest.mark.parametrize("n", [0, 1, 255, 256, 257, LAST - 606208, LAST - 1, LAST, LAST + 1])
@pytest.mark.parametrize("first,stride", [(0, 606208), (606207, 606208), (77, 1 << 20)])
def test_strided_walk_ends(tmp_path, first, stride, n):
    """The walk over an array of n entries, or n - 1 rows and their last
    pointer, meets each position once and stops."""
    out = run_cpp(tmp_path, f"""int main() {{
  long long count = 0, bad = 0; int last = -1;
  strided({first}, {stride}, {n}ll, [&](int p) {{ bad += p < 0 || p >= {n}ll || p % {stride} != {first} % {stride}; ++count; last = p; }});
  std::printf("%lld %lld %d", count, bad, last);
}}""")
    count = len(range(first, n, stride))
    assert out == [str(count), "0", str(range(first, n, stride)[-1] if count else -1)]


@pytest.mark.parametrize("per", [32, 256, 2048, 4096])
@pytest.mark.parametrize("n", [0, 1, 31, 2048, 2049, LAST - 2048, LAST - 1, LAST])
def test_blocks_cover_their_items(tmp_path, per, n):
    out = run_cpp(tmp_path, f"""int main() {{
  const int b = blocks_over({n}, {per});
  std::printf("%d %d %d", b, b ? block_end(0, {per}, {n}) : 0, b ? block_end((b - 1) * {per}, {per}, {n}) : 0);
}}""")
    assert out == [str(-(-n // per)), str(min(per, n)), str(n)]
