"""What a built tree holds (CPU): the large tables of a generated header only
in the translation units whose kernels use them, and no objects beside the
libraries that were linked from them."""

import re

import pytest

from mkpp_gb300 import build

GENERATED = sorted(build.GEN.glob("*.cuh"))
LARGE = 512          # elements of a table that every unit may hold a copy of


@pytest.mark.parametrize("path", GENERATED, ids=lambda p: p.name)
def test_large_tables_are_made_per_use(path):
    lines = path.read_text().splitlines()
    large = 0
    for before, line in zip(lines, lines[1:]):
        m = re.match(r"(?:alignas\(16\) )?static __device__ const [\w ]+ \w+\[(\d+)\] = \{", line)
        if m and int(m.group(1)) > LARGE:
            large += 1
            assert before == "template <int = 0>", line[:80]
    assert large >= 1


def test_no_objects_stay_beside_the_libraries(tmp_path, monkeypatch):
    def unit(mech, name, verbose):
        obj = tmp_path / f"{name}.o"
        obj.write_bytes(b"object")
        return obj

    monkeypatch.setattr(build, "LIB", tmp_path)
    monkeypatch.setattr(build, "_compile_unit", unit)
    monkeypatch.setattr(build, "_link", lambda mech, objs: tmp_path / "lib.so" if all(o.exists() for o in objs) else None)
    assert build.compile_mechanism("chapman") == tmp_path / "lib.so"
    assert not list(tmp_path.glob("*.o"))


def test_host_only_programs_stay_out_of_device_code():
    """The evaluation program of a table-driven mechanism serves host checks
    of its tables; no kernel walks it."""
    text = (build.GEN / "ts1.cuh").read_text()
    for what in ("eval_prog[", "static void eval_step("):
        at = text.index(what)
        assert text.rindex("#ifndef __CUDACC__", 0, at) > text.rfind("#endif", 0, at)


def test_device_code_is_compressed():
    assert "--compress-mode=size" in build._flags("chapman", False)
