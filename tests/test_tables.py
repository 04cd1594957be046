"""The host-built twiddle tables (bigint_b200/csrc/tables.cu): every entry
against its definition, and the time all of them take, which a program pays in
bgpu_init."""
from __future__ import annotations

import os
import re
import subprocess

import numpy as np
import pytest

from conftest import ROOT, load_recipe

CSRC = os.path.join(ROOT, "bigint_b200", "csrc")

# Writes every set's table; prints its parameters, then the time of all sets
# and the time of the two three-prime sets with a division for each product,
# quotient and remainder (both the shortest of several).
HARNESS = r"""
#include <chrono>
#include <cstdio>
#include <vector>
#include "tables.h"
using namespace bgpu;
static double us(std::chrono::steady_clock::time_point a) {
    return std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - a).count();
}
int main(int argc, char** argv) {
    std::vector<std::vector<uint2>> t;
    FILE* f = fopen(argv[1], "wb");
    for (int s = 0; s < kNumSets; ++s) {
        t.emplace_back(table_entries(s, stage_log_of(s)));
        build_tables(s, stage_log_of(s), t[s].data());
        fwrite(t[s].data(), sizeof(uint2), t[s].size(), f);
        printf("%d %d %d", stage_log_of(s), kPrimeSets[s].log_max, kPrimeSets[s].split);
        for (int q = 0; q < kPrimeSets[s].np; ++q) printf(" %u %u", kPrimeSets[s].p[q], kPrimeSets[s].g[q]);
        printf("\n");
    }
    fclose(f);
    double all = 1e30, plain = 1e30;
    for (int k = 0; k < 7; ++k) {
        auto t0 = std::chrono::steady_clock::now();
        for (int s = 0; s < kNumSets; ++s) build_tables(s, stage_log_of(s), t[s].data());
        all = std::min(all, us(t0));
        t0 = std::chrono::steady_clock::now();
        for (int s = 0; s < 2; ++s) {
            const size_t per = t[s].size() / kPrimeSets[s].np;
            for (int q = 0; q < kPrimeSets[s].np; ++q) {
                const uint32_t p = kPrimeSets[s].p[q], r = kPrimeSets[s].g[q];
                uint64_t v = 1;
                for (size_t i = 0; i < per; ++i) {
                    t[s][q * per + i] = make_uint2((uint32_t)(v % p), (uint32_t)((v << 32) / p));
                    v = v * r % p;
                }
            }
        }
        plain = std::min(plain, us(t0));
    }
    printf("%.1f %.1f\n", all, plain);
}
"""


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    d = tmp_path_factory.mktemp("tables")
    src, exe, out = d / "harness.cu", d / "harness", d / "tables.bin"
    src.write_text(HARNESS)
    nvcc = load_recipe("bigint_b200/build.py").NVCC
    subprocess.run([nvcc, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC, str(src),
                    os.path.join(CSRC, "tables.cu"), "-o", str(exe)], check=True)
    lines = subprocess.run([str(exe), str(out)], check=True, capture_output=True, text=True).stdout.splitlines()
    sets = []
    for line in lines[:-1]:
        v = [int(x) for x in re.findall(r"\d+", line)]
        sets.append((v[0], v[1], v[2], list(zip(v[3::2], v[4::2]))))
    return sets, np.fromfile(out, dtype=np.uint32).reshape(-1, 2).astype(np.uint64), [float(x) for x in lines[-1].split()]


def powers(root, n, p):
    v = np.ones(n, dtype=np.uint64)
    k = 1
    while k < n:  # v[k .. 2k) = v[0 .. k) root^k
        v[k : 2 * k] = v[: min(k, n - k)] * np.uint64(pow(root, k, p)) % np.uint64(p)
        k *= 2
    return v


def test_entries(built):
    sets, table, _ = built
    at = 0
    for stage_log, log_max, split, primes in sets:
        for p, g in primes:
            pinv = np.uint64(pow(p, -1, 1 << 32))
            for sign in (1, -1):
                def root(log):
                    return pow(pow(g, (p - 1) >> log, p), sign, p)

                want = [powers(root(j + 1), 1 << j, p) for j in range(stage_log)]
                stage = np.concatenate([[np.uint64(1)], *want])
                got = table[at : at + stage.size]
                assert np.array_equal(got[:, 0], stage)
                assert np.array_equal(got[:, 1], (stage << np.uint64(32)) // np.uint64(p))
                at += stage.size
                for step, n in ((1 << split, 1 << (log_max - split)), (1, 1 << split)):
                    v = powers(pow(root(log_max), step, p), n, p)
                    mont = (v << np.uint64(32)) % np.uint64(p)
                    got = table[at : at + n]
                    assert np.array_equal(got[:, 0], mont)
                    assert np.array_equal(got[:, 1], mont * pinv & np.uint64(0xFFFFFFFF))
                    at += n
    assert at == len(table)


def test_time(built):
    """The tables of all 42 primes in at most three times what the six primes of
    the three-prime sets take with divisions (0.8 times; five times with them)."""
    all_us, plain_us = built[2]
    assert all_us < 3 * plain_us
