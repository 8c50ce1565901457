"""Device memory that the library keeps for photon maps must not make another of its
calls fail: every allocation goes through device_malloc, which gives the kept
memory back and tries again."""
import re

from encore_b200.build import CSRC


def test_every_allocation_can_take_the_kept_memory_back():
    direct = []
    for f in sorted(CSRC.iterdir()):
        if f.suffix in (".cu", ".cpp", ".h"):
            body = ""
            for line in f.read_text().splitlines():
                if re.match(r"^\w.*\(.*\{$", line):  # a function begins
                    body = line
                code = re.sub(r'"[^"]*"', "", line.split("//")[0])
                if re.search(r"\bcudaMalloc\s*\(", code) and not re.search(
                        r"\b(device_malloc|keep_small)\(", body):
                    direct.append(f"{f.name}: {line.strip()}")
    assert not direct, direct
