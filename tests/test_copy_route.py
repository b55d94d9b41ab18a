"""Which fields of a state the copy kernel takes (csrc/copy_route.hpp): whole
words on the context's device while that device is current.  The rule is host
code and compiles without CUDA."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "aquagpusph_gb300", "csrc")
CHECK = r"""
#include <cstdio>
#include <cstdlib>
#include "copy_route.hpp"
int main(int argc, char** argv) {
    if (argc != 6) return 2;
    std::printf("%d", (int)aqua::copied_by_kernel(
        std::atoi(argv[1]) != 0, std::atoi(argv[2]), std::atoi(argv[3]), std::atoi(argv[4]),
        reinterpret_cast<const void*>(std::strtoull(argv[5], nullptr, 0))));
    return 0;
}
"""


@pytest.fixture(scope="module")
def route(tmp_path_factory):
    d = tmp_path_factory.mktemp("route")
    src, exe = d / "check.cpp", d / "check"
    src.write_text(CHECK)
    subprocess.run([os.environ.get("CXX") or shutil.which("g++") or "g++", "-std=c++17",
                    "-I", CSRC, str(src), "-o", str(exe)], check=True)

    def call(device_memory, memory, context, current, address=0x7f0000000100):
        out = subprocess.run([str(exe), str(int(device_memory)), str(memory), str(context),
                              str(current), hex(address)], check=True, capture_output=True)
        return out.stdout == b"1"
    return call


def test_own_device_current(route):
    assert route(True, 0, 0, 0) and route(True, 1, 1, 1)
    assert route(True, 0, 0, 0, 0x7f0000000104)


def test_another_device_current(route):
    """A kernel would run on the wrong device: copies, as for any device."""
    assert not route(True, 0, 0, 1)
    assert not route(True, 1, 1, 0)
    assert not route(True, 1, 1, -1)


def test_other_memory(route):
    assert not route(False, 0, 0, 0)      # host, managed or unknown
    assert not route(True, 1, 0, 0)       # another device's
    assert not route(True, 0, 0, 0, 0x7f0000000102)
    assert not route(True, 0, 0, 0, 0x7f0000000101)
