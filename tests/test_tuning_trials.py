"""The autotuner's trials (autan_b200/csrc/tuning_trials.hpp) compiled for the host: ranks of unequal
meshes make the same trials, however their cells and blocks lie about the limits, and ask each other
the same number of times."""

import itertools
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent

# Two ranks as threads that meet in every `any`; a rank that asks once more than its peer would wait,
# so a rank that has ended answers for itself and the numbers of questions are compared.
PROGRAM = r"""
#include "tuning_trials.hpp"
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
using namespace autan_b200;
std::mutex guard;
std::condition_variable met;
int ended = 0, asked[2] = {0, 0};
std::vector<bool> flags[2];
struct Rank { long long cells; int fits; TrialScope scope; };
void run(int r, Rank& me, bool second) {
  auto any = [&](bool mine) {
    std::unique_lock<std::mutex> lock(guard);
    flags[r].push_back(mine);
    const size_t k = static_cast<size_t>(asked[r]++);
    met.notify_all();
    met.wait(lock, [&] { return flags[1 - r].size() > k || ended > 0; });
    return mine || (flags[1 - r].size() > k && flags[1 - r][k]);
  };
  me.scope = trial_scope(second, me.cells, 606208, any, [&](int b) { return (me.fits >> (b / 64)) & 1; },
                         [&](int b) { return (me.fits >> (2 + b / 64)) & 1; });
  std::lock_guard<std::mutex> lock(guard);
  ++ended;
  met.notify_all();
}
int main(int argc, char** argv) {
  Rank a{std::atoll(argv[1]), std::atoi(argv[2]), {}}, b{std::atoll(argv[3]), std::atoi(argv[4]), {}};
  const bool second = std::atoi(argv[5]) != 0, fp32 = std::atoi(argv[6]) != 0;
  std::thread t(run, 1, std::ref(b), second);
  run(0, a, second);
  t.join();
  for (int r = 0; r < 2; ++r) {
    const Rank& m = r == 0 ? a : b;
    std::printf("%d|", asked[r]);
    for (const GradTrial& g : grad_trials(m.scope, fp32)) std::printf("%d,%d,%d,%d;", g.mode, g.chunk, g.block, g.minb);
    std::printf("|");
    for (const FaceTrial& f : face_trials(m.scope, false)) std::printf("%d,%d,%d;", f.mode, f.block, f.threads);
    std::printf("\n");
  }
}
"""


@pytest.fixture(scope="module")
def trials(tmp_path_factory):
    d = tmp_path_factory.mktemp("trials")
    src, exe = d / "trials.cpp", d / "trials"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", f"-I{REPO / 'autan_b200' / 'csrc'}", str(src), "-o", str(exe)],
                   check=True)  # fmt: skip

    def run(*args):
        r = subprocess.run([str(exe), *map(str, args)], check=True, capture_output=True, text=True, timeout=60)
        return r.stdout.splitlines()

    return run


SIZES = [5_000, 75_776, 75_777, 303_104, 303_105, 606_208, 606_209, 2_000_000]


@pytest.mark.parametrize("a, b", list(itertools.combinations_with_replacement(SIZES, 2)))
def test_ranks_on_both_sides_of_a_limit_make_the_same_trials(trials, a, b):
    for second, fp32 in ((1, 1), (1, 0), (0, 1)):
        for fits in ((31, 31), (31, 0), (30, 31), (31, 27), (23, 31)):
            one, two = trials(a, fits[0], b, fits[1], second, fp32)
            assert one == two, (second, fp32, fits)
            # the smaller mesh alone would try at least as much: nothing is tried that one cannot run
            own = trials(b, fits[1], b, fits[1], second, fp32)[0]
            assert set(one.split("|")[2].split(";")) <= set(own.split("|")[2].split(";"))


def test_a_mesh_alone_tries_what_fits(trials):
    def modes(cells, fits, second=1):
        _, grads, faces = trials(cells, fits, cells, fits, second, 1)[0].split("|")
        return ({tuple(map(int, t.split(","))) for t in grads.split(";") if t},
                {tuple(map(int, t.split(","))) for t in faces.split(";") if t})  # fmt: skip

    grads, faces = modes(5_000, 31)
    assert {(6, 2, 32, 7), (6, 2, 64, 7), (0, 2, 64, 7), (4, 4, 128, 5)} <= grads
    assert {(0, 64, 256), (3, 32, 256), (3, 64, 256), (3, 128, 256), (2, 128, 256)} <= faces
    grads, faces = modes(5_000, 0)
    assert not any(g[0] == 6 for g in grads) and not any(f[0] == 3 for f in faces)
    grads, faces = modes(100_000, 31)
    assert any(g[0] == 6 for g in grads) and {f[1] for f in faces if f[0] == 3} == {128}
    grads, faces = modes(500_000, 31)
    assert not any(g[0] == 6 for g in grads) and {f[1] for f in faces if f[0] == 3} == {128}
    grads, faces = modes(2_000_000, 31)
    assert not any(g[0] == 6 for g in grads) and not any(f[0] == 3 for f in faces)
