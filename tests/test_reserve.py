"""The reservation of shared memory (csrc/reserve.h), compiled for the host with stand-ins for the three CUDA calls."""

import re
import subprocess
from pathlib import Path

from models_b200.kernels import build

PROGRAM = r"""
#include "reserve.h"
#include <cstdio>
static int device = 0, calls = 0, last = -1;
static cudaError_t answer = cudaSuccess;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes) { ++calls; last = bytes; return answer; }
#define EXPECT(what) if (!(what)) { std::printf("line %d: %s\n", __LINE__, #what); return 1; }
int main() {
    mb::DeviceSet done{0};
    int kernel = 0;
    EXPECT(mb::reserve_on_device(&kernel, 100, done) == cudaSuccess && calls == 1 && last == 100);
    EXPECT(mb::reserve_on_device(&kernel, 100, done) == cudaSuccess && calls == 1);
    device = 1;  // the attribute of device 0 says nothing about this one
    answer = cudaErrorInvalidValue;
    EXPECT(mb::reserve_on_device(&kernel, 100, done) == cudaErrorInvalidValue && calls == 2);
    answer = cudaSuccess;  // a call that failed is made again
    EXPECT(mb::reserve_on_device(&kernel, 100, done) == cudaSuccess && calls == 3);
    EXPECT(mb::reserve_on_device(&kernel, 100, done) == cudaSuccess && calls == 3);
    device = 64;
    EXPECT(mb::reserve_on_device(&kernel, 100, done) == cudaSuccess && mb::reserve_on_device(&kernel, 100, done) == cudaSuccess && calls == 5);
    device = 0;
    EXPECT(mb::reserve_on_device(&kernel, 100, done) == cudaSuccess && calls == 5);
    return 0;
}
"""


def test_shared_memory_is_reserved_on_every_device(tmp_path):
    source, program = tmp_path / "reserve.cpp", tmp_path / "reserve"
    source.write_text(PROGRAM)
    include = Path(build._nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-I", str(build.CSRC), "-I", str(include), str(source), "-o", str(program)], check=True)
    result = subprocess.run([str(program)], capture_output=True, text=True)
    assert result.returncode == 0, result.stdout


def test_no_launcher_keeps_the_first_answer_for_every_device():
    for path in sorted(build.CSRC.glob("*.cu")):
        text = path.read_text()
        assert not re.search(r"static\s+const\s+cudaError_t", text), f"{path.name}: an attribute of one device is kept for all"


def test_no_launcher_remembers_a_reservation_for_every_device():
    """What a launcher keeps about attributes it keeps for each device: in a DeviceSet, or in an array that the device's number indexes."""
    for path in sorted(build.CSRC.glob("*.cu")):
        for kept, count in re.findall(r"static\s+(?:bool|int|size_t)\s+(\w+)(?:\[(\w+)\])?\s*=", path.read_text()):
            assert count in ("64", "kMaxDevices"), f"{path.name}: {kept} is kept for all devices"
