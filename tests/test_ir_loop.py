"""The refinement's host loop (csrc/ir_loop.cuh), compiled for the host with a device of
the test's own: it ends after the last matrix that is being refined, asks rarely, reports
the last residual it formed, and a failing question ends it with the error instead of
being read as "no matrix left"."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "magma_gb300" / "csrc"

MAIN = r"""
#include "ir_loop.cuh"
#include <cstdio>
#include <cstdlib>
#include <string>
// argv: itermax, the residual from which no matrix is left (-1: never), look (0/1),
// the post and the wait that fail (-1: none), and whether a failing wait writes 0
struct Look {
    int last, fail_post, fail_wait, zero, posts = 0, waits = 0, answer = 1;
    int post(int it) { answer = last >= 0 && it >= last ? 0 : 1; return posts++ == fail_post ? -7 : 0; }
    int wait(int *left)
    {
        if (waits++ == fail_wait) { if (zero) *left = 0; return -9; }
        *left = answer;
        return 0;
    }
};
int main(int, char **v)
{
    const int itermax = atoi(v[1]);
    Look look{atoi(v[2]), atoi(v[4]), atoi(v[5]), atoi(v[6])};
    std::string log;
    int done = -1;
    const int rc = mlu::ir_iterate(itermax, atoi(v[3]) ? &look : (Look *)nullptr, [&](int it) { log += " c" + std::to_string(it); },
                                   [&](int it) { log += " r" + std::to_string(it); }, &done);
    printf("%d %d %d %d%s\n", rc, done, look.posts, look.waits, log.c_str());
}
"""


@pytest.fixture(scope="module")
def loop(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("ir_loop")
    (d / "main.cc").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), str(d / "main.cc"), "-o", str(d / "main")], check=True)

    def run(itermax, last, look=1, fail_post=-1, fail_wait=-1, zero=0):
        out = subprocess.run([str(d / "main"), *map(str, (itermax, last, look, fail_post, fail_wait, zero))],
                             capture_output=True, text=True, check=True).stdout.split()
        return [int(x) for x in out[:4]], out[4:]
    return run


def _all(k):
    return [x for it in range(k) for x in (f"c{it}", f"r{it + 1}")]


@pytest.mark.parametrize("itermax", [0, 1, 2, 3, 4, 5, 30])
def test_every_iteration_without_look_or_convergence(loop, itermax):
    assert loop(itermax, -1, look=0) == ([0, itermax, 0, 0], _all(itermax))
    (rc, done, posts, waits), log = loop(itermax, -1)
    assert (rc, done, log) == (0, itermax, _all(itermax))
    assert posts == waits <= 4                    # after 2, 4, 8 and 16 iterations


@pytest.mark.parametrize("last,posts,done", [(0, 1, 3), (2, 1, 3), (3, 2, 5), (4, 2, 5), (5, 3, 9), (16, 4, 17), (17, 4, 30)])
def test_ends_after_the_last_matrix(loop, last, posts, done):
    # the matrix that converges at residual `last` is marked by correct(last), which has run
    (rc, d, p, w), log = loop(30, last)
    assert (rc, d, p, w) == (0, done, posts, posts)
    assert log == _all(done) and f"c{last}" in log


@pytest.mark.parametrize("zero", [0, 1])
def test_a_failing_question_is_an_error(loop, zero):
    (rc, done, _, _), _ = loop(30, 2, fail_wait=0, zero=zero)
    assert rc == -9 and done == -1
    (rc, done, _, _), _ = loop(30, 2, fail_post=0)
    assert rc == -7 and done == -1
