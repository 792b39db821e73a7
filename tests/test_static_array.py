"""What the library's device image reserves for cipsi_run_pt2_static is the one
array that the header promises: a program that hands the device's memory to its
own pool counts on it."""
import os
import re

from conftest import ROOT


def test_device_image_holds_the_promised_array_alone():
    arrays = []
    csrc = os.path.join(ROOT, "cipsi_gb300", "csrc")
    for name in sorted(os.listdir(csrc)):
        with open(os.path.join(csrc, name)) as fh:
            text = fh.read()
        for m in re.finditer(r"^(?:static )?__device__ (?:__align__\(\d+\) )?[\w ]+ (\w+)\[(\w+)\];", text, re.M):
            size = re.search(r"%s = \(size_t\)(\d+) << 20;" % m.group(2), text)
            arrays.append((m.group(1), int(size.group(1)) if size else m.group(2)))
    with open(os.path.join(ROOT, "include", "cipsi_gb300.h")) as fh:
        promised = re.search(r"besides one (\d+) MiB array", fh.read())
    assert arrays == [("g_pt2_scratch", int(promised.group(1)))]
