"""CPU tests of the worker threads behind the large host arrays (csrc/host_pool.hpp), compiled on their own.

- Every share of [0, n) is taken once, whatever n and the grain, from several pools at once too.
- A process forked after the pool started has none of its threads: dropping the pool there ends, and work
  given to it is done by the caller.
"""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "skirt9-gpu_b200", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <cstring>
#include <memory>
#include <sys/wait.h>
#include <unistd.h>
#include "host_pool.hpp"

static bool covers(skg::HostPool& pool, size_t n, size_t grain)
{
    std::vector<std::atomic<int>> hits(n);
    pool.run(n, grain, [&](size_t a, size_t b) { for (size_t i = a; i < b; ++i) ++hits[i]; });
    for (auto& h : hits)
        if (h != 1) return false;
    return true;
}

int main(int, char** argv)
{
    alarm(20);  // a wait that does not end ends the process
    if (!std::strcmp(argv[1], "shares"))
    {
        std::atomic<bool> ok{true};
        auto all = [&] {
            skg::HostPool pool;
            for (size_t n : {1, 2, 15, 16, 17, 1000, 1001, 4096})
                for (size_t grain : {1, 3, 64, 5000}) ok = covers(pool, n, grain) && ok;
        };
        std::vector<std::thread> callers;
        for (int i = 0; i < 3; ++i) callers.emplace_back(all);
        for (auto& t : callers) t.join();
        return ok ? 0 : 1;
    }
    auto pool = std::make_unique<skg::HostPool>();
    if (!covers(*pool, 1000, 1)) return 1;
    pid_t child = fork();
    if (child == 0)
    {
        alarm(5);
        const bool good = std::strcmp(argv[1], "work") || covers(*pool, 1000, 1);
        pool.reset();
        _exit(good ? 0 : 1);
    }
    int status = 0;
    waitpid(child, &status, 0);
    return WIFEXITED(status) && WEXITSTATUS(status) == 0 && covers(*pool, 1000, 1) ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("pool")
    src, exe = d / "pool.cpp", d / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("what", ["shares", "drop", "work"])
def test_host_pool(program, what):
    assert subprocess.run([program, what]).returncode == 0
