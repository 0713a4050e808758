"""A kernel's shared-memory limit is an attribute of one device: no function keeps
whether it has set it (or the result) for the process, where the second device
of a program would be left with the limit it starts with."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "cola_halo_b200", "csrc")


def test_no_limit_is_set_once_per_process():
    found = []
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = open(path).read()
        # initialisers of function-level statics, up to the end of the statement
        for m in re.finditer(r"^[ \t]+static\s+(?:const\s+)?(\w+)\s+(\w+)\s*=", text, re.M):
            rest = text[m.end():]
            end = rest.index("}();") if rest.lstrip().startswith("[") else rest.index(";")
            near = rest[:end + 400] if m.group(1) == "bool" else rest[:end]
            if "FuncSetAttribute" in near or "smem_attr" in near:
                found.append((os.path.basename(path), m.group(2)))
    assert not found, found
