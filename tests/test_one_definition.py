"""A struct of namespace scope that several source files define has one definition: the files are
linked together and pass such structs to each other."""
import collections
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rbmongpu_gb300", "csrc")


def definitions(text):
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    for m in re.finditer(r"^(?:struct|class) (\w+)[^;{()]*\{", text, flags=re.M):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield m.group(1), "".join(text[m.start():end].split())


def test_structs_shared_by_files_agree():
    found = collections.defaultdict(dict)
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            for name, body in definitions(open(os.path.join(CSRC, f)).read()):
                found[name].setdefault(body, []).append(f)
    assert "Chunk" in found and "TcNet" in found
    assert not {n: list(b.values()) for n, b in found.items() if len(b) > 1}
