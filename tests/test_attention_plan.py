"""Which form of attention a round takes and how the decode form cuts contexts: the rules, compiled for the host."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llama.cu_b200", "csrc")
SMS = 148

MAIN = r"""
#include <cstdio>
#include <vector>
#include "attention_plan.hpp"
struct Req { unsigned pos, len; };
int main() {
    int what, a, b, c, d, e, f;
    while (scanf("%d", &what) == 1) {
        if (what == 0) {  // the split of a decode round
            if (scanf("%d %d %d %d %d %d", &a, &b, &c, &d, &e, &f) != 6) return 1;
            const lcu::AttnPlan p = lcu::attn_plan(a, b, c, d, e, f);
            printf("%d %d\n", p.splits, p.tiles);
        } else if (what == 1) {  // the form of a round: head size, group, KV heads, requests, possible forms
            int n;
            if (scanf("%d %d %d %d %d %d", &a, &b, &c, &d, &e, &n) != 6) return 1;
            std::vector<Req> r(n);
            for (auto &q : r) if (scanf("%u %u", &q.pos, &q.len) != 2) return 1;
            printf("%d\n", (int)lcu::attn_form(a, b, c, r.data(), n, d, e & 1, e >> 1 & 1));
        }
    }
}
"""


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "main")], check=True)

    def run(*words):
        r = subprocess.run([str(d / "main")], input=" ".join(map(str, words)), capture_output=True, text=True, check=True)
        return r.stdout.strip().split("\n")
    return run


def plan(ask, nkvh, dh, n_tok, tiles, clusters=None):
    z, t = map(int, ask(0, nkvh, dh, n_tok, tiles, SMS, int(n_tok < 3 if clusters is None else clusters))[0].split())
    return z, t


@pytest.mark.parametrize("nkvh", [1, 2, 8, 32])
@pytest.mark.parametrize("dh", [64, 128])
@pytest.mark.parametrize("n_tok", [1, 2, 3, 8, 16, 31, 64, 300, 1024])
def test_splits_reach_the_context(ask, nkvh, dh, n_tok):
    for tiles in (1, 2, 4, 8, 12, 16, 32, 64, 512, 1024):
        z, t = plan(ask, nkvh, dh, n_tok, tiles)
        assert z >= 1 and z * t >= tiles and (z == 1 or (z <= 64 and (z - 1) * t < tiles and n_tok * z <= 2048))


@pytest.mark.parametrize("nkvh,dh,n_tok,tiles,most", [
    (1, 128, 16, 64, 31), (1, 128, 31, 32, 11), (8, 128, 2, 64, 22), (8, 128, 4, 32, 16), (8, 128, 8, 16, 8), (8, 64, 4, 32, 16), (32, 128, 1, 32, 16),
    (8, 64, 8, 4, 1), (8, 128, 8, 2, 1), (32, 128, 64, 64, 1)])
def test_no_more_splits_than_their_merge_is_worth(ask, nkvh, dh, n_tok, tiles, most):
    """Rounds that splits for eight CTAs per SM made up to 45 % slower than splits for four."""
    assert plan(ask, nkvh, dh, n_tok, tiles)[0] <= most


def test_short_contexts_are_cut(ask):
    assert plan(ask, 8, 128, 1, 4) == (4, 1) and plan(ask, 8, 128, 16, 8) == (4, 2) and plan(ask, 8, 128, 8, 8) == (8, 1)


SPLIT, ROWS64, ROWS256 = 0, 1, 2


def form(ask, dh, group, nkvh, reqs, possible=3):
    return int(ask(1, dh, group, nkvh, SMS, possible, len(reqs), *[v for r in reqs for v in r])[0])


@pytest.mark.parametrize("dh,group,nkvh,reqs,want", [
    # decoded tokens of short contexts beside a short prompt: 64 rows a CTA (60 sequences of 100, 32 heads: 85 against 119 us)
    (64, 1, 32, [(100, 1)] * 60 + [(0, 2)], ROWS64), (64, 1, 32, [(500, 1)] * 60 + [(0, 2)], ROWS64), (128, 1, 32, [(140, 1)] * 31 + [(0, 2)], ROWS64),
    (64, 4, 8, [(140, 1)] * 60 + [(0, 2)], ROWS64), (128, 4, 8, [(100, 1)] * 31 + [(0, 2)], ROWS64), (64, 1, 32, [(100 + 3 * i, 1) for i in range(60)] + [(0, 300)], ROWS64),
    (64, 4, 8, [(0, 33)], ROWS64), (128, 1, 32, [(5, 1), (0, 2)], ROWS64),
    # long contexts and prompts: 256
    (64, 1, 32, [(1900, 1)] * 60 + [(0, 2)], ROWS256), (128, 1, 32, [(500, 1)] * 60 + [(0, 2)], ROWS256), (128, 4, 8, [(1000, 1)] * 16 + [(0, 2)], ROWS256),
    (64, 4, 8, [(0, 8000)], ROWS256), (128, 4, 8, [(0, 997)], ROWS256), (128, 8, 8, [(0, 500)], ROWS256), (64, 8, 8, [(1900, 2)], ROWS256),
    (128, 4, 8, [(60 + 20 * i, 1) for i in range(31)] + [(512, 481)], ROWS256)])
def test_form_follows_rows_and_contexts(ask, dh, group, nkvh, reqs, want):
    assert form(ask, dh, group, nkvh, reqs) == want
    assert form(ask, dh, group, nkvh, reqs, 1) == ROWS64


@pytest.mark.parametrize("nkvh,reqs,want", [
    (8, [(60000, 4), (5, 1)], SPLIT), (8, [(60000, 16)], SPLIT), (8, [(20000, 8)], SPLIT), (8, [(20000, 16)], SPLIT), (8, [(60000, 1)] * 6 + [(0, 20)], SPLIT), (32, [(60000, 2)], SPLIT),
    (8, [(60000, 64)], ROWS256), (8, [(5000, 128)], ROWS256), (32, [(60000, 16)], ROWS256), (8, [(0, 60000)], ROWS256)])
def test_few_tokens_behind_a_long_context_are_split(ask, nkvh, reqs, want):
    """More pages than the 64-row form takes: without the decode form, four tokens behind 60000 take 1.67 instead of 0.48 ms."""
    assert form(ask, 128, 4 if nkvh == 8 else 1, nkvh, reqs, 2) == want
    assert form(ask, 128, 4 if nkvh == 8 else 1, nkvh, reqs, 0) == SPLIT


def test_plans_of_a_batch_size_are_few(ask):
    """A captured round is kept for each plan, not for each reach: where contexts are not cut, one serves all."""
    def keys(nkvh, dh, n_tok, nctx):
        tiles, got = 1, set()
        while True:
            z, t = plan(ask, nkvh, dh, n_tok, min(tiles, nctx // 64))
            got.add((z, 0 if z == 1 else t))
            if tiles >= nctx // 64:
                return got
            tiles *= 2
    assert len(keys(32, 128, 64, 8192)) == 1
    assert all(len(keys(8, dh, n, 2048)) <= 6 for dh in (64, 128) for n in (1, 4, 16, 64))
