"""The library's translation units are linked into one library: a class of a namespace they share
has one definition."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "monc_b200", "csrc")
TOKEN = re.compile(r"namespace\s+(\w*)\s*\{|\b(?:struct|class|union)\s+(\w+)\s*(?:<[^<>;{]*>)?\s*(?::[^;{]*)?\{|[{}]")


def definitions(path):
    """(scope, name) of every class defined at namespace scope; unnamed namespaces are left out."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/|\"(?:\\.|[^\"\\\n])*\"|'(?:\\.|[^'\\\n])'", "", open(path).read(), flags=re.S)
    scope, out = [], []
    for m in TOKEN.finditer(text):
        t = m.group(0)
        if t == "}":
            if scope:
                scope.pop()
        elif t.startswith("namespace"):
            scope.append(m.group(1) or os.path.basename(path))  # an unnamed one is the file's own
        elif m.group(2):
            if None not in scope:
                out.append(("::".join(scope), m.group(2)))
            scope.append(None)
        else:
            scope.append(None)
    return out


def test_classes_of_shared_namespaces_are_defined_once():
    seen = {}
    for f in sorted(os.listdir(CSRC)):
        for d in definitions(os.path.join(CSRC, f)):
            seen.setdefault(d, set()).add(f)
    assert ("mgpu", "Scalars") in seen and len(seen) > 30
    assert not {d: f for d, f in seen.items() if len(f) > 1}
