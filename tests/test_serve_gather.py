"""The render server's batch forming (gather_ms of csrc/server.h): a burst of
requests is not cut into fragments while the device is busy anyway."""

import os
import subprocess

import pytest

import build as native

PROGRAM = r"""
#include <cstdio>
#include "server.h"
int main() {
  double now, oldest, newest; int busy, full;
  while (std::scanf("%lf %lf %lf %d %d", &now, &oldest, &newest, &busy, &full) == 5)
    std::printf("%.17g\n", gsr::gather_ms(now, oldest, newest, busy, full));
}
"""


@pytest.fixture(scope="module")
def gather(tmp_path_factory):
    d = tmp_path_factory.mktemp("gather")
    (d / "gather.cpp").write_text(PROGRAM)
    subprocess.run([native.CXX, "-std=c++17", "-I", native.CSRC, "-I", native.INCLUDE, "-I",
                    os.path.join(native.CUDA_HOME, "include"), str(d / "gather.cpp"), "-o",
                    str(d / "gather")], check=True)

    def ask(now, oldest, newest, busy, full):
        line = f"{now} {oldest} {newest} {int(busy)} {int(full)}\n"
        return float(subprocess.run([str(d / "gather")], input=line, capture_output=True,
                                    text=True, check=True).stdout)

    return ask


def test_a_burst_is_gathered_while_the_device_is_busy(gather):
    # submits 5 us apart: the lane waits for them to end ...
    assert 0.0 < gather(10.005, 10.0, 10.005, True, False) < 0.1
    # ... and launches when they have
    assert gather(10.2, 10.0, 10.005, True, False) == 0.0


def test_nothing_waits_that_need_not(gather):
    assert gather(10.0, 10.0, 10.0, False, False) == 0.0  # an idle device
    assert gather(10.005, 10.0, 10.005, True, True) == 0.0  # a full batch
    # an endless stream of submits holds the oldest request up for a bounded time
    assert gather(10.6, 10.0, 10.6, True, False) == 0.0
    assert gather(10.499, 10.0, 10.499, True, False) <= 0.0011
