"""The status words that kernels write into host memory: one per device, in one page,
none shared (two threads may call scComputeVertexNormalsNoAlloc on two devices)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "solidcloth_b200" / "csrc"

PROGRAM = r"""
#include "host_words.h"
#include <cstdint>
#include <cstdio>
static sc::HostWords w;
int main()
{
    for (int d = 0; d < 2; d++) *w.of(d) = 10 + d;              // two devices' kernels, then their readers
    for (int d = 0; d < 2; d++) if (*w.of(d) != 10 + d) return 1;
    for (int d = 0; d < sc::HostWords::DEVICES; d++)
    {
        if (!sc::HostWords::has(d) || w.of(d) < w.word || w.of(d) >= w.word + sizeof(w.word) / sizeof(int)) return 2;
        for (int e = 0; e < d; e++) if (w.of(d) == w.of(e)) return 3;
    }
    if (sc::HostWords::has(-1) || sc::HostWords::has(sc::HostWords::DEVICES)) return 4;
    if (reinterpret_cast<uintptr_t>(w.word) % 4096 || sizeof(w.word) > 4096) return 5;
    puts("ok");
}
"""


def test_one_word_per_device(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    (tmp_path / "w.cpp").write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-I", str(CSRC), str(tmp_path / "w.cpp"), "-o", str(tmp_path / "w")], check=True)
    r = subprocess.run([str(tmp_path / "w")], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.returncode


def test_the_call_uses_its_devices_word():
    """every use of the page in noalloc.cu goes through the device's word (or registers the whole page)"""
    src = (CSRC / "noalloc.cu").read_text()
    uses = re.findall(r"g_noalloc_host(?!_word)([^;,)]*)", src)
    assert uses and all(u == "" or u.startswith((".word", ".of(dev")) for u in uses), uses
