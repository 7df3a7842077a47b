"""Kernels that start while their predecessor runs read its output by ordinary
loads (the rule stated at lux::after_previous), checked on the sources."""
import os
import re

import pytest

import bevy_penumbra_b200

CSRC = os.path.join(os.path.dirname(bevy_penumbra_b200.__file__), "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


# What a chained kernel reads of the launch just before it: the children pass
# the own pass's list and the next level's records, the resolve the pack's
# tables.
@pytest.mark.parametrize("buffer", ["merged", "pass_list", "tables"])
def test_output_of_the_previous_launch_is_read_by_ordinary_loads(buffer):
    text = source("view.cu")
    assert re.search(r"\bV\.%s\b" % buffer, text)
    pointers = {"V." + buffer, "J.V." + buffer}
    pointers |= set(re.findall(r"\*\s*(\w+)\s*=\s*V\.%s\b" % buffer, text))
    loads = re.findall(r"__ldg\(\s*&?([\w.]+)", text)
    assert not [p for p in loads if p in pointers]


@pytest.mark.parametrize("name", ["view.cu", "screen.cu", "scene.cu"])
def test_every_chained_kernel_waits_first(name):
    text = source(name)
    started = set()
    for call in re.findall(r"lux::launch\(\s*(\([^;]*?\)|[^,;]*?),", text):
        started |= {k for k in re.findall(r"\w+_kernel", call)}
    assert started
    for kernel in started:
        body = re.search(r"\b%s\((?:[^()]|\([^()]*\))*\)\s*\{(.{0,60})" % kernel, text, re.S)
        assert body, kernel
        assert body.group(1).split(";")[0].strip() == "lux::after_previous()", kernel
