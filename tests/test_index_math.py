"""Index arithmetic of the kernels with several threads per item, compiled for
the host: batches reach 2^31 - 16 items, so thread numbers pass 32 bits."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CHECK = r"""
#include "swb_index.h"
#include <cstdio>
#include <initializer_list>
int main() {
    const size_t items[] = {0, 1, 31, 32, (size_t(1) << 29) - 1, size_t(1) << 29, (size_t(1) << 29) + 33, 0x7FFFFFEFu};
    for (size_t it : items)
        for (unsigned per : {1u, 8u, 32u})
            for (unsigned lane : {0u, per - 1}) {
                const size_t t = it * per + lane;
                if (swb::group_item((unsigned)(t / 256), 256, (unsigned)(t % 256), per) != it) {
                    std::printf("item %zu, %u threads each\n", it, per);
                    return 1;
                }
            }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_group_item_is_exact_over_the_accepted_batches(tmp_path):
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "swiftbwa_b200", "csrc"), "-o", str(exe), str(src)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
