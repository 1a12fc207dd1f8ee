"""Setup that belongs to a kernel on one device (no GPU needed: the source is read)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kyojin_mac_b200", "csrc")


def test_shared_memory_limits_are_set_per_device():
    """cudaFuncSetAttribute acts on the current device only: a flag per process would leave a second GPU of the process with the 48 KB default, and launches there
    fail. Every call therefore stands in a function that asks for the current device and remembers it."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for body in re.findall(r"^(?:template|static|int|extern)[^\n]*(?:\n(?!\}).*)*", text, re.M):
            calls = body.count("cudaFuncSetAttribute(")
            if calls:
                seen += calls
                assert "cudaGetDevice(&dev)" in body and re.search(r"(<<|>>) \(?dev\b", body), (os.path.basename(path), body[:120])
                assert not re.search(r"static bool \w*configured", body), (os.path.basename(path), body[:120])
        assert not re.search(r"static bool \w*configured", text), os.path.basename(path)
    assert seen >= 4
