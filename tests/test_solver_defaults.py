"""BatchSolver.set_solver's defaults are the library's."""
import inspect
import os
import re

import gcfg

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_set_solver_defaults():
    text = open(os.path.join(ROOT, "gc-fg_gb300", "csrc", "engine.cuh")).read()
    fields = re.findall(r"^    int (\w+(?:, \w+)*);", text[text.index("struct SolveParams {"):], re.M)
    names = [n for f in fields for n in f.split(", ")]
    values = re.search(r"kDefaultSolveParams\{([^}]*)\}", text).group(1).split(",")
    lib = dict(zip(names, (eval(v) for v in values)))  # noqa: S307 (integers and shifts)
    py = {k: p.default for k, p in inspect.signature(gcfg.BatchSolver.set_solver).parameters.items()}
    for key, field in dict(push_rounds_per_gr="push_rounds", max_tile_sweeps="max_sweeps",
                           sweeps_per_local_relabel="bfs_every", local_relabel_first="bfs_first",
                           push_only="push_only", threads_y="warps").items():
        assert py[key] == lib[field], key
