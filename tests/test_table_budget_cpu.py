"""The device memory an index may give its k-mer table (csrc/table_budget.hpp,
compiled here): a quarter of the free memory beside nine bytes a node, whatever
the construction's own temporaries take meanwhile."""
import subprocess

import pytest

import sbwt_b200 as S

GIB = 1 << 30
# free bytes before construction, nodes -> budget
CASES = [
    (170 * GIB, 115_000_000), (170 * GIB, 1_000_000_000), (145 * GIB, 1_000_000_000),
    (36_000, 1_000), (9_000, 1_000), (8_999, 1_000), (0, 1), (100, 0), (9_004, 1_000),
    (1 << 40, 1 << 60),
]


@pytest.fixture(scope="module")
def budgets(tmp_path_factory):
    d = tmp_path_factory.mktemp("budget")
    src, exe = d / "budget.cpp", d / "budget"
    src.write_text('#include <cstdio>\n#include <cstdlib>\n#include "table_budget.hpp"\n'
                   'int main(int c, char **v) { for (int i = 1; i + 1 < c; i += 2) std::printf('
                   '"%llu\\n", (unsigned long long)sbwt::kmer_table_budget(strtoull(v[i], 0, 10), '
                   'strtoull(v[i + 1], 0, 10))); }\n')
    subprocess.run(["g++", "-std=c++17", "-I", str(S.HERE / "csrc"), str(src), "-o", str(exe)],
                   check=True)
    args = [str(x) for case in CASES for x in case]
    return [int(x) for x in subprocess.run([str(exe), *args], check=True, capture_output=True,
                                           text=True).stdout.split()]


def test_a_quarter_of_the_free_memory_beside_the_labels(budgets):
    assert budgets == [max(f - 9 * n, 0) // 4 if f // 9 > n else 0 for f, n in CASES]


def test_a_billion_nodes_keep_a_table_of_32_gib(budgets):
    """2^31 slots of 16 bytes and 10 filter bits a k-mer, with 145 GiB free of
    which construction itself takes 36 GB meanwhile."""
    assert budgets[2] >= (1 << 31) * 16 + 1_000_000_000 * 10 // 8
