"""Libraries of a shipped mechanism with its generated header changed, for GPU
tests of forms that only a larger mechanism takes."""

from mkpp_gb300 import api, build
from mkpp_gb300.emitter import cuda_emitter
from mkpp_gb300.emitter.plan import load


def make(tmp, monkeypatch, name, mech, table=None, change=lambda text: text):
    """Builds and loads `name`: the header of `mech`, through `change`."""
    text = cuda_emitter.emit_mechanism(load(mech), table=table)
    (tmp / f"{name}.cuh").write_text(change(text.replace(f"mkpp_{mech}", f"mkpp_{name}")))
    monkeypatch.setattr(build, "GEN", tmp)
    monkeypatch.setattr(build, "LIB", tmp)
    monkeypatch.setattr(api, "LIB_DIR", tmp)
    build.compile_mechanism(name)
    api.load_library(name)
    return name
