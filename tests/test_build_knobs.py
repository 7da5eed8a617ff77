"""The tuning defines that the build names are read by some source."""
import os
import re

ROOT = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "denrimrendererkit_gb300")


def test_named_defines_are_read():
    with open(os.path.join(ROOT, "build.py")) as f:
        named = set(re.findall(r"\b(DK_[A-Z0-9_]+)=\d", f.read()))
    assert named
    sources = ""
    for name in os.listdir(os.path.join(ROOT, "csrc")):
        with open(os.path.join(ROOT, "csrc", name)) as f:
            sources += f.read()
    for define in named:
        assert re.search(rf"#ifndef {define}\b", sources), define
