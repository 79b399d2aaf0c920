"""Kernels started with programmatic dependent launch may run before their predecessor on the stream is complete:
each of them has to wait for it (pdl_wait) before anything else, early returns included.  Checked in the sources."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "ipeps.jl_b200" / "csrc"


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def _kernels():
    """name -> whether pdl_wait() is the first statement, for every __global__ function"""
    out = {}
    for f in sorted(CSRC.glob("*.cu*")):
        text = _code(f)
        for m in re.finditer(r"__global__\b", text):
            head = re.match(r"[^{;]*\{", text[m.start():]).group(0)
            while True:  # launch bounds and cluster sizes
                new = re.sub(r"__(?:launch_bounds|cluster_dims)__\s*\((?:[^()]|\([^()]*\))*\)", "", head)
                if new == head:
                    break
                head = new
            name = re.search(r"(\w+)\s*\(", head).group(1)
            body = text[m.start() + len(re.match(r"[^{;]*\{", text[m.start():]).group(0)):]
            out.setdefault(name, []).append(body.lstrip().startswith("pdl_wait();"))
    return out


def test_dependent_launches_wait():
    kernels = _kernels()
    started = set()
    for f in sorted(CSRC.glob("*.cu")):
        text = _code(f)
        aliases = dict(re.findall(r"auto\s+(\w+)\s*=\s*(\w+_kernel)\b", text))
        for name in re.findall(r"\blaunch(?:_clusters)?\(c\.stream,\s*(\w+)", text):
            started.add(aliases.get(name, name))
    assert len(started) > 50
    for name in sorted(started):
        assert kernels[name] and all(kernels[name]), name


def test_other_launches_are_plain():
    """The attribute is set in one place only."""
    hits = [f.name for f in CSRC.glob("*.cu*") if "ProgrammaticStreamSerialization" in f.read_text()]
    assert hits == ["ctx.cuh"]
