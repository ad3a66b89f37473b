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
                   'extern "C" int history_fits(long long r, long long h, long long n, long long t) { return ttb::chain::history_fits(r, h, n, t); }\n'
                   'extern "C" int memory_fits(long long r, long long h, long long n, long long k, long long t) { return ttb::chain::memory_fits(r, h, n, k, t); }\n'
                   'extern "C" int bias_units() { return ttb::chain::kBiasUnits; }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.bias_columns.restype, lib.bias_columns.argtypes = ctypes.c_longlong, [ctypes.c_longlong]
    lib.first_unit.restype = ctypes.c_uint
    lib.history_fits.argtypes, lib.memory_fits.argtypes = [ctypes.c_longlong] * 4, [ctypes.c_longlong] * 5
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


# (heads, rows, tokens, us by the chain, us layer by layer) of a decoding step over a cache, and the same over an encoder memory, on 148 SMs
HISTORY = [(12, 1, 30, 289, 404), (12, 24, 30, 408, 427), (12, 24, 1000, 600, 647), (12, 24, 2000, 861, 787), (12, 16, 1000, 511, 607), (12, 16, 2000, 732, 696),
           (12, 16, 2500, 838, 749), (12, 1, 2000, 454, 507), (12, 1, 3000, 552, 513), (12, 1, 4000, 637, 532), (12, 4, 4000, 646, 607), (12, 8, 3000, 592, 656),
           (12, 8, 8000, 1151, 945), (12, 12, 2500, 592, 682), (8, 1, 2000, 395, 459), (8, 1, 4000, 541, 471), (8, 18, 2500, 600, 630), (8, 18, 4000, 766, 743),
           (8, 20, 1000, 501, 510), (8, 20, 1600, 608, 566), (8, 24, 700, 465, 515), (8, 24, 1600, 637, 597), (16, 1, 2500, 911, 1082), (16, 9, 3000, 1284, 1610),
           (16, 10, 1600, 1274, 1362), (16, 16, 1300, 1207, 1384), (16, 18, 1300, 1334, 1423), (16, 18, 3000, 2247, 2123), (16, 16, 4000, 2514, 2330),
           (16, 20, 300, 1005, 1090), (16, 20, 1000, 1518, 1342), (16, 24, 300, 1041, 1172), (16, 24, 1000, 1540, 1485), (16, 24, 1300, 1827, 1706)]
MEMORY = [(8, 64, 200, 436, 532), (8, 64, 400, 498, 532), (8, 64, 700, 600, 550), (8, 64, 1000, 675, 634), (8, 48, 700, 539, 572), (8, 48, 400, 446, 536), (8, 37, 1000, 477, 568),
          (8, 32, 1000, 433, 560), (8, 32, 1600, 517, 2534), (8, 64, 1600, 800, 2600), (8, 18, 3200, 505, 2800), (16, 32, 800, 585, 613), (16, 32, 1600, 813, 5152),
          (16, 24, 1000, 602, 664), (16, 1, 800, 294, 512)]


def test_the_faster_route_is_taken_wherever_both_were_measured(rules):
    """Routes within 4 % of one another count as equal: that is what runs and GPUs differ by."""
    for heads, rows, tokens, chain, layers in HISTORY:
        assert abs(chain - layers) < 0.04 * layers or bool(rules.history_fits(rows, heads, 148, tokens)) == (chain < layers), (heads, rows, tokens)
    for heads, rows, keys, chain, layers in MEMORY:
        assert abs(chain - layers) < 0.04 * layers or bool(rules.memory_fits(rows, heads, 148, keys, 0)) == (chain < layers), (heads, rows, keys)


def test_the_result_of_every_bounded_wait_is_used():
    """A wait that runs out has to reach the status word: none may stand as a statement of its own."""
    source = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "ttb_chain.cu")).read())
    calls = re.findall(r"([^\n]*)\b(?:wait|wait_slots|wait_ahead)\(", source)
    assert len(calls) >= 7
    for before in calls:
        assert re.search(r"(return|=|!|&&|\|\||bool)\s*$", before) or "bool" in before, before
