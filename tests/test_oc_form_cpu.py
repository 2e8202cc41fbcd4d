"""The launch form of the optimality-criteria update (stokes_to_gb300/csrc/oc_form.h), compiled
for the host: for every design size, on devices of 1 to 1300 multiprocessors, with and without
the cluster, the block sums fit the OC_PARTS doubles that a handle has for them, every cell
has a thread, and registers hold the cells where the form says so. (28^3 and 32^3 are the sizes
whose second buffer of sums once began too far into the array.)
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_block_sums_fit_for_every_size(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "form.cpp"
    src.write_text(r'''
#include <cstdio>
#include <initializer_list>
#include "oc_form.h"
using namespace stg;
int main() {
    long long bad = 0, seen = 0;
    auto check = [&](long long nc, int sms, bool can) {
        const OcForm f = oc_form(nc, sms, can);
        const long long threads = (long long)f.blocks * f.threads, held = f.cluster ? OC_CR : OC_GR;
        seen++;
        bad += f.parts() > OC_PARTS || f.parts() != (f.cluster ? 0 : 2 * f.blocks);
        bad += f.blocks < 1 || f.blocks > (f.cluster ? OC_CB : sms < OC_MAX_BLOCKS ? sms : OC_MAX_BLOCKS);
        bad += f.held && threads * held < nc;
        bad += f.cluster && (!can || nc > OC_CLUSTER_MAX || f.threads != OC_T<OC_CR>);
        bad += !f.cluster && f.threads != (f.held ? OC_T<OC_GR> : OC_T<0>);
        bad += !f.cluster && (f.blocks - 1ll) * f.threads >= nc;  // a block without cells
    };
    for (int sms : {1, 2, 76, 148, 152, 304, 607, 608, 609, 1300})
        for (int can = 0; can < 2; can++) {
            for (long long n = 4; n <= 1024; n += 4) check(n * n * n, sms, can);
            for (long long n = 8; n <= 16384; n += 8) check(n * n, sms, can);
            for (long long nc : {1, 127, 128, 129, 16383, 16384, 16385}) check(nc, sms, can);
        }
    std::printf("%lld %lld\n", seen, bad);
    return bad != 0;
}
''')
    exe = tmp_path / "form"
    subprocess.run([gxx, "-std=c++17", "-I", os.path.join(ROOT, "stokes_to_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    seen, bad = map(int, out.stdout.split())
    assert out.returncode == 0 and bad == 0 and seen > 40000
