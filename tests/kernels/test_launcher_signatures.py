"""The argument types that ops/_lib.py passes to the launchers, against the declarations in the CUDA sources."""

import re
from pathlib import Path

from nanonemo_b200.csrc import build
from nanonemo_b200.ops import _lib

CODES = {"int": "i", "long long": "q", "float": "f", "double": "d"}


def _declared() -> dict:
    out = {}
    for path in build.sources():
        text = re.sub(r"//[^\n]*", "", Path(path).read_text())
        for name, args in re.findall(r'extern "C"\s+int\s+(nnb_\w+)\s*\(([^)]*)\)\s*\{', text):
            args = [a.strip() for a in args.split(",") if a.strip() not in ("", "void")]
            out[name] = "".join("p" if "*" in a or a.startswith("cudaStream_t") else CODES[re.sub(r"\s*\w+$", "", a).strip()] for a in args)
    return {n: sig for n, sig in out.items() if not n.endswith("_prof_read")}  # compiled in with -DNNB_PROFILE only


def test_signatures_are_those_of_the_sources():
    assert _lib._SIGNATURES == _declared()


def test_every_launcher_that_is_called_by_name_has_a_signature():
    root = Path(_lib.__file__).resolve().parents[1]
    called = {n for f in root.rglob("*.py") for n in re.findall(r'"(nnb_\w+)"', f.read_text())}
    assert called <= set(_lib._SIGNATURES), called - set(_lib._SIGNATURES)


def test_the_native_binding_declares_the_launchers_as_the_sources_do():
    text = (Path(_lib.__file__).resolve().parents[1] / "csrc" / "binding.cpp").read_text()
    protos = re.findall(r"^int (nnb_\w+)\(([^)]*)\);", text, re.M)
    assert protos
    for name, args in protos:
        args = [a.strip() for a in args.split(",") if a.strip()]
        sig = "".join("p" if "*" in a or a == "cudaStream_t" else CODES[a] for a in args)
        assert sig == _lib._SIGNATURES[name], name
