"""CPU: the two MMA issuers of the tensor-core Linear on their ring of slots, in a model of the barriers.

A barrier wait sees one bit, the parity of the use it waits for. The model keeps the true use numbers beside it, lets loads land,
products finish and warps run in any order, and looks whether an issuer ever takes a slot for filled that is not, or whether the
ring comes to a stop. The rule under test (ttb_ring.cuh) is the kernel's own, compiled for the host."""
import ctypes
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "turbotransformers_b200", "csrc")


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    src, so = d / "rule.cpp", d / "rule.so"
    src.write_text('#include "ttb_ring.cuh"\n'
                   'extern "C" int wait_for_empty_first(int s, int i, int n, int o) { return ttb::ring::wait_for_empty_first(s, i, n, o); }\n'
                   'extern "C" int min_stages() { return ttb::ring::kMinStages; }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def run_ring(stages, blocks, tiles, producers, seed, first):
    """One random order of events. first(offset) says whether an issuer waits for "empty" first. Returns what went wrong, or None."""
    rng = random.Random(seed)
    total = blocks * tiles
    sent = [0] * producers                       # blocks that each producer has sent for
    flying = set()                               # (block, producer) not landed yet
    parts = [0] * total                          # operands landed
    full, empty = [0] * stages, [0] * stages     # completed uses of each slot's two barriers
    own = [[(t, o) for t in range(tiles) for o in range(i, blocks, 2)] for i in range(2)]
    at, passed_empty = [0, 0], [False, False]
    running = [[], []]                           # products issued and not finished, in order, each issuer's
    done = [0] * total
    # each run prefers some actors to others, so that loads and products are held back for long
    weight = {}

    def w(key):
        return weight.setdefault(key, rng.choice([0.01, 0.2, 1.0, 5.0]))

    while sum(done) < total:
        acts = []
        for p in range(producers):
            g = sent[p]
            if g < total and empty[g % stages] % 2 == (g // stages) % 2:
                acts.append((w(("p", p)), ("send", p)))
        for b in flying:
            acts.append((w(("l", b)), ("land", b)))
        for i in range(2):
            if running[i]:
                acts.append((w(("f", i, running[i][0])), ("finish", i)))
            if at[i] == len(own[i]):
                continue
            t, o = own[i][at[i]]
            if t >= 2 and not all(done[(t - 2) * blocks:(t - 1) * blocks]):
                continue                         # two accumulators: the tile before the last one has left its
            g = t * blocks + o
            s, n = g % stages, g // stages
            if first(o) and not passed_empty[i]:
                if empty[s] % 2 == n % 2:
                    acts.append((w(("w", i)), ("see_empty", i)))
            elif full[s] % 2 == (n + 1) % 2:
                acts.append((w(("w", i)), ("issue", i)))
        if not acts:
            return "stalled"
        kind, x = rng.choices([a for _, a in acts], [v for v, _ in acts])[0]
        if kind == "send":
            flying.add((sent[x], x))
            sent[x] += 1
        elif kind == "land":
            flying.discard(x)
            parts[x[0]] += 1
            if parts[x[0]] == producers:
                full[x[0] % stages] += 1
        elif kind == "finish":
            g = running[x].pop(0)
            done[g] = 1
            empty[g % stages] += 1
        elif kind == "see_empty":
            passed_empty[x] = True
        else:
            t, o = own[x][at[x]]
            g = t * blocks + o
            if parts[g] != producers:
                return "read before it landed"
            running[x].append(g)
            at[x] += 1
            passed_empty[x] = False
    return None


# rings of the kernels' sizes (3 and 5: two planes of an operand in one slot), tiles of one to many k-blocks, even and odd
@pytest.mark.parametrize("stages", [3, 4, 5, 6, 8])
@pytest.mark.parametrize("blocks", [1, 2, 3, 5, 7, 8, 12, 31])
def test_issuers_never_read_a_slot_before_its_load_has_landed(rule, stages, blocks):
    assert stages >= rule.min_stages()
    for producers in (1, 2):
        for seed in range(60):
            assert run_ring(stages, blocks, 4, producers, seed, lambda o: rule.wait_for_empty_first(stages, 2, blocks, o)) is None


# What the rule adds is needed where it adds it, and nowhere else: with the wait for "full" alone, odd rings and tiles of an odd
# number of blocks are read too early, and even rings with even tiles never.
@pytest.mark.parametrize("stages,blocks,safe", [(3, 8, False), (5, 12, False), (4, 7, False), (8, 31, False), (4, 8, True), (6, 12, True), (8, 2, True)])
def test_the_model_tells_rings_that_need_the_second_wait(rule, stages, blocks, safe):
    seen = {run_ring(stages, blocks, 4, 1, seed, lambda o: False) for seed in range(400)}
    assert seen == {None} if safe else "read before it landed" in seen
    assert any(rule.wait_for_empty_first(stages, 2, blocks, o) for o in range(blocks)) == (not safe)
    assert not any(rule.wait_for_empty_first(stages, 1, blocks, o) for o in range(blocks))
