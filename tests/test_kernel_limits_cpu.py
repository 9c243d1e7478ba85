"""The shared-memory limit of a kernel belongs to the process, not to a context: contexts run in
threads of their own, so a limit may not depend on one context's sizes (read as source)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "waterscapes_gb300", "csrc")

# sizes that are compile-time constants of the instantiation
CONSTANT = re.compile(r"^(?:[A-Z][A-Z_]*|[\d\s*]+)$")


def test_dynamic_shared_memory_limits_are_constants():
    found = 0
    for f in sorted(os.listdir(CSRC)):
        s = open(os.path.join(CSRC, f)).read()
        for v in re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*(.*?)\)\);", s):
            found += 1
            if v == "(int)sm" and "const size_t sm = staged_smem_bytes<T>();" in s:
                continue  # (the staged kernel: a constant of its type)
            assert CONSTANT.match(v), (f, v)
    assert found >= 5
