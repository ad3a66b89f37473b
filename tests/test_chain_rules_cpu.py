"""CPU: the rules by which the chain kernel deals out its work (ttb_chain_rules.cuh), compiled for the host, on grids of every size."""
import ctypes
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "turbotransformers_b200", "csrc")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("chain")
    src, so = d / "rules.cpp", d / "rules.so"
    src.write_text('#include "ttb_chain_rules.cuh"\n'
                   'extern "C" unsigned first_unit(unsigned u, unsigned c, unsigned n) { return ttb::chain::first_unit(u, c, n); }\n'
                   'extern "C" int writes_row(int r, int c) { return ttb::chain::writes_row(r, c); }\n'
                   'extern "C" int rows_have_writers(int r, int n) { return ttb::chain::rows_have_writers(r, n); }\n'
                   'extern "C" long long bias_columns(long long n) { return ttb::chain::bias_columns(n); }\n'
                   'extern "C" int bias_units() { return ttb::chain::kBiasUnits; }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.bias_columns.restype, lib.bias_columns.argtypes = ctypes.c_longlong, [ctypes.c_longlong]
    lib.first_unit.restype = ctypes.c_uint
    return lib


@pytest.mark.parametrize("ctas", [1, 2, 7, 20, 63, 64, 65, 132, 148, 160])
def test_every_row_and_every_unit_belongs_to_one_cta(rules, ctas):
    for rows in range(1, 65):  # a grid that has no CTA for some row is refused
        writers = [sum(rules.writes_row(row, c) for c in range(ctas)) for row in range(rows)]
        assert (writers == [1] * rows) == bool(rules.rows_have_writers(rows, ctas))
    for units in (1, 3, 96, 288, 384, 6283, 1 << 21):
        edges = [rules.first_unit(units, c, ctas) for c in range(ctas + 1)]
        assert edges[0] == 0 and edges[-1] == units and edges == sorted(edges)


@pytest.mark.parametrize("ctas", [1, 20, 132, 148])
def test_a_bias_that_is_accepted_has_room_in_every_cta(rules, ctas):
    units = rules.bias_columns(ctas) // 8
    assert max(rules.first_unit(units, c + 1, ctas) - rules.first_unit(units, c, ctas) for c in range(ctas)) <= rules.bias_units()
    assert units >= 15 * ctas


def test_the_result_of_every_bounded_wait_is_used():
    """A wait that runs out has to reach the status word: none may stand as a statement of its own."""
    source = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "ttb_chain.cu")).read())
    calls = re.findall(r"([^\n]*)\b(?:wait|wait_slots|wait_ahead)\(", source)
    assert len(calls) >= 7
    for before in calls:
        assert re.search(r"(return|=|!|&&|\|\||bool)\s*$", before) or "bool" in before, before
