"""Chapman with every reaction split into parts of equal rate: a mechanism of
thousands of reactions (slots beyond 14 bits, more rates and partial
derivatives than a block's shared memory holds) with Chapman's solution."""

import copy

from mkpp_gb300.emitter import cuda_emitter
from mkpp_gb300.emitter.plan import load_raw, reduce_plan

NAME = "chapman_split"


def raw(parts):
    out = copy.deepcopy(load_raw("chapman"))
    one = out["reactions"]
    out["reactions"] = []
    for part in range(parts):
        for r in one:
            x = copy.deepcopy(r)
            x.update(index=len(out["reactions"]), k=f"({r['k']})/{parts}.0")
            x["dk_dfixed"] = [[s, f"({e})/{parts}.0"] for s, e in r["dk_dfixed"]]
            out["reactions"].append(x)
    out["num_reactions"] = len(out["reactions"])
    out["name"] = NAME
    return out


def write_header(directory, parts):
    """The table-driven header of the split mechanism; returns its plan."""
    plan = reduce_plan(raw(parts))
    (directory / f"{NAME}.cuh").write_text(cuda_emitter.emit_mechanism(plan, table=True))
    return plan
