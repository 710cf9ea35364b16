"""A launch that can be refused (no tensor map: the brick gather) is never taken for done: its result is used at
every call, and the declaration has the compiler say so."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "cube2_b200", "csrc")


def test_gather_launch_is_checked():
    calls = []
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        if name == "common.cuh":
            assert re.search(r"\[\[nodiscard\]\]\s+bool launch_pm3_force_gather\(", text)
        else:
            calls += [(name, m.group(1).strip()) for m in re.finditer(r"([^;{}]*)\blaunch_pm3_force_gather\(a?", text)
                      if not m.group(1).strip().endswith("bool")]
            # a call through a lambda: its result is returned, and used where the lambda is called
            bare = re.findall(r"[;{})]\s*gather\(\w+\);", text)
            assert not bare, (name, bare)
    assert len(calls) >= 2
    for name, before in calls:
        assert before.endswith(("return", "!", "=")), (name, before)
