"""No launcher sets a kernel's limit of dynamic shared memory to a size that
depends on the input: the limit belongs to the kernel, not to the call, and
contexts on several host threads launch the same kernels, so one thread could
lower it between another's setting and its launch."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imagestackalignator_b200", "csrc")


def limits():
    """(file, expression) of every value that a limit is set to."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            text = f.read()
        for m in re.finditer(r"cudaFuncAttributeMaxDynamicSharedMemorySize\s*,", text):
            depth, i = 0, m.end()
            while depth >= 0:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            yield os.path.basename(path), " ".join(text[m.end():i - 1].split())


def test_limits_are_constants():
    """Constants by this code's naming: capitals, and members of a layout struct L."""
    found = list(limits())
    assert found
    for path, expr in found:
        names = re.findall(r"[A-Za-z_]\w*", re.sub(r"\(int\)", "", expr))
        assert all(n.isupper() for n in names), (path, expr)
