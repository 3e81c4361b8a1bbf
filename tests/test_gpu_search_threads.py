"""The search's block size is the one that was asked for, in each of its forms,
and the lists do not depend on it.  The sizes are read from the launches, as the
profiler of the installed torch records them, in a process of its own so that
the other tests run without it."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FORMS = [(0.8e-3, 1), (0.8e-3, 2), (0.25e-3, 1)]   # eight lanes, twice, and one thread per particle
THREADS = (64, 128, 256)


def main(folder):
    import numpy as np
    import torch
    from torch.profiler import ProfilerActivity, profile

    from mcmtop_b200 import _abi
    from mcmtop_b200.deck import taylor_bar
    from mcmtop_b200.solver import Solver

    torch.cuda.init()
    trace = os.path.join(folder, "trace.json")
    out = []
    for dx, kind in FORMS:
        deck, first = taylor_bar(dx=dx), None
        for threads in THREADS:
            sol = Solver(deck, _abi.PREC_FP64_EXACT)
            sol.set_tuning(search_threads=threads, search_kind=kind)
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                sol.step()
                torch.cuda.synchronize()
            prof.export_chrome_trace(trace)
            with open(trace) as f:
                events = json.load(f)["traceEvents"]
            blocks = {e["args"]["block"][0] for e in events if e.get("cat") == "kernel" and "k_search" in e["name"]}
            lists = sol.neighbours()[:2]
            first = first or lists
            out.append([sol.tuning()["search_threads"], sorted(blocks),
                        all(bool(np.array_equal(a, b)) for a, b in zip(lists, first))])
            sol.close()
    print(json.dumps(out))


def test_blocks_as_asked(tmp_path):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([ROOT] + [p for p in [os.environ.get("PYTHONPATH")] if p]))
    r = subprocess.run([sys.executable, os.path.abspath(__file__), str(tmp_path)], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    got = json.loads(r.stdout.strip().splitlines()[-1])
    assert got == [[t, [t], True] for _ in FORMS for t in THREADS]


if __name__ == "__main__":
    main(sys.argv[1])
