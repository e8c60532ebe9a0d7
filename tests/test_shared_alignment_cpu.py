"""Shared arrays that a kernel reads or writes as vectors say how they are aligned, read off the source."""
import glob
import os
import re

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fuselink_b200", "csrc", "kernels")
VECTOR = r"reinterpret_cast<(?:const |volatile )*(?:float|uint|int|longlong|ulonglong)[24]\s*\*>\(\s*&?\s*(\w+)"


def test_shared_arrays_used_as_vectors_state_their_alignment():
    """An array of floats is aligned to 4 bytes, wherever the compiler puts it; a 16-byte access to another address faults."""
    used = []
    for path in sorted(glob.glob(os.path.join(KERNELS, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        declared = {}
        for m in re.finditer(r"\b__shared__([^;]*);", text):
            for name in re.findall(r"(\w+)\s*(?:\[|,|$)", m.group(1)):
                declared.setdefault(name, []).append(m.group(1))
        for name in re.findall(VECTOR, text):
            for d in declared.get(name, []):
                used.append(name)
                assert re.search(r"__align__\((16|32|64|128|1024)\)", d), f"{os.path.basename(path)}: {name}"
    assert "qk_angle" in used
