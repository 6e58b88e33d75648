"""The two halves of piece-wise work (autan_b200/csrc/piece_ring.hpp) compiled for the host: every
piece put before it is taken, in order, no more than the ring between them; without a second thread the
same; an exception of either half ends both and comes out."""

import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "piece_ring.hpp"
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <vector>
using namespace autan_b200;
int main(int, char** argv) {
  const long long pieces = std::atoll(argv[1]);
  const int ring = std::atoi(argv[2]), threads = std::atoi(argv[3]);
  const long long bad_put = std::atoll(argv[4]), bad_take = std::atoll(argv[5]);
  std::atomic<long long> put{0}, taken{0};
  std::atomic<int> wrong{0};
  std::vector<long long> slot(ring, -1);
  const char* thrown = "";
  auto start = [&](auto f) {
    if (!threads) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
    return std::thread(f);
  };
  try {
    run_pieces(pieces, ring,
               [&](long long p) {
                 if (p == bad_put) throw std::runtime_error("put");
                 if (p != put || p - taken >= ring) ++wrong;
                 slot[p % ring] = p;
                 ++put;
               },
               [&](long long p) {
                 if (p == bad_take) throw std::runtime_error("take");
                 if (p != taken || slot[p % ring] != p) ++wrong;
                 ++taken;
               },
               start);
  } catch (const std::exception& e) {
    thrown = e.what();
  }
  std::printf("%lld %lld %d %s.\n", put.load(), taken.load(), wrong.load(), thrown);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    (d / "ring.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{REPO / 'autan_b200' / 'csrc'}",
                    str(d / "ring.cpp"), "-o", str(d / "ring")], check=True)  # fmt: skip

    def run(*args):
        r = subprocess.run([str(d / "ring"), *map(str, args)], check=True, capture_output=True, text=True,
                           timeout=60)  # fmt: skip
        put, taken, wrong, thrown = r.stdout.split()
        return int(put), int(taken), int(wrong), thrown.rstrip(".")

    return run


@pytest.mark.parametrize("threads", [1, 0])
@pytest.mark.parametrize("pieces, ring", [(1, 3), (2, 3), (3, 3), (50, 3), (20, 1)])
def test_every_piece_in_order(program, pieces, ring, threads):
    assert program(pieces, ring, threads, -1, -1) == (pieces, pieces, 0, "")


@pytest.mark.parametrize("threads", [1, 0])
@pytest.mark.parametrize("half", ["put", "take"])
@pytest.mark.parametrize("at", [0, 4, 19])
def test_an_exception_ends_both(program, half, at, threads):
    put, taken, wrong, thrown = program(20, 3, threads, at if half == "put" else -1, at if half == "take" else -1)
    assert thrown == half and wrong == 0 and taken <= put <= taken + 4 and (put if half == "put" else taken) == at
