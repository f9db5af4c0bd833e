"""What a pair of CTAs waits for when it gives up (csrc/pair_drain.cuh), against a model of the barriers: the copies of both CTAs and the
expectation of the first count on one barrier a stage.  From every state that two producers can stop in, with the copies that
have landed drawn at random, each wait of the rule ends and no copy is left in flight.  Waiting for the first CTA's fillings alone,
in the same model, leaves copies of the second in flight."""
import os
import subprocess

import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "ternary_llm_b200", "csrc")

MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "pair_drain.cuh"
using namespace tllm;
constexpr int kBytes = 3;
struct Barrier {
    int parity = 0, pending = 1, tx = 0;               // one arrival a phase
    void settle() { while (pending == 0 && tx == 0) { parity ^= 1; pending = 1; } }
    void expect(int n) { tx += n; pending--; settle(); }
    void complete(int n) { tx -= n; settle(); }
    bool done(int p) const { return parity != p; }
};
struct Copy { int stage; };
int main(int argc, char** argv)
{
    const bool first_only = argc > 1;
    long left = 0, stuck = 0, states = 0;
    srand(1);
    for (int stages : {4, 6, 8})
        for (int consumed = 0; consumed <= 3 * stages; consumed++)             // fillings that the MMAs consumed
            for (int a = consumed; a <= consumed + stages; a++)
                for (int b = consumed; b <= consumed + stages; b++)
                    for (int draw = 0; draw < 4; draw++) {
                        states++;
                        std::vector<Barrier> bar(stages);
                        std::vector<Copy> flying;
                        const int end = a > b ? a : b;
                        for (int f = 0; f < end; f++) {
                            const int s = f % stages;
                            std::vector<int> steps;                            // of this filling, in any order
                            if (f < a) bar[s].expect(2 * kBytes), steps.push_back(0);
                            if (f < b) steps.push_back(1);
                            for (size_t i = 0; i < steps.size(); i++) {
                                if (f < consumed || rand() % 2) bar[s].complete(kBytes);
                                else flying.push_back({s});
                            }
                            if (f < consumed && !bar[s].done((f / stages) & 1)) return 2;
                        }
                        const int first = a, second = first_only ? 0 : b;
                        for (int f = pair_fills_begin(first, second, stages); f < pair_fills_end(first, second); f++) {
                            PairFill p = pair_fill(f, first, second, stages);
                            if (first_only) p.unarmed = p.lacks = false;
                            if (p.unarmed) bar[p.stage].expect(kBytes);
                            if (p.lacks) bar[p.stage].complete(kBytes);
                            // the wait: copies land until it ends, or there are none of this stage
                            while (!bar[p.stage].done(p.parity)) {
                                size_t i = 0;
                                while (i < flying.size() && flying[i].stage != p.stage) i++;
                                if (i == flying.size()) { stuck++; break; }
                                flying.erase(flying.begin() + i);
                                bar[p.stage].complete(kBytes);
                            }
                        }
                        left += !flying.empty();
                    }
    printf("%ld %ld %ld\n", states, stuck, left);
    return 0;
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("drain")
    (d / "m.cpp").write_text(MODEL)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-I", SRC, "-o", str(d / "m"), str(d / "m.cpp")])
    return str(d / "m")


def run(*cmd):
    return [int(v) for v in subprocess.check_output(cmd, text=True).split()]


def test_nothing_is_left_in_flight(model):
    states, stuck, left = run(model)
    assert states > 10000 and stuck == 0 and left == 0


def test_the_first_cta_alone_is_not_enough(model):
    _, stuck, left = run(model, "first")
    assert stuck > 0 and left > 0
