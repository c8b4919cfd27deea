"""qlp_last_launch_count against the kernels that the CUDA profiler sees, one evaluation and
a batch replayed from graphs, on both paths and with the outside-surface-brightness prior.
In a process of its own: the profiler has to be there before the first CUDA call."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = r"""
import json, sys
import numpy as np, torch
from torch.profiler import ProfilerActivity, profile
from goldens import Golden
from qlens_gb300 import PixelLikelihood

def kernels(f):
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    return sum(e.count for e in p.key_averages() if "qlpix" in e.key)

with profile(activities=[ProfilerActivity.CUDA]):
    torch.zeros(8, device="cuda").add_(1)
    torch.cuda.synchronize()
g = Golden("tiny_sie")
out = []
for precision in (0, 1):
    for osb in (False, True):
        pl = PixelLikelihood.from_opts(g.image, g.psf, g.opts, precision=precision)
        pl.set_lens_model(g.lenses, *g.zbeta())
        if osb:
            pl.set_outside_sb_prior(True)
        P = np.array([g.params()] * 3)
        for name, f in (("one", pl.invert_image_surface_brightness_map), ("batch", lambda: pl.eval_batch(P))):
            f()
            out.append((precision, osb, name, kernels(f), pl.last_launch_count()))
        pl.close()
print(json.dumps(out))
"""


def test_count_is_what_ran():
    pytest.importorskip("torch")
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests")]))
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    if not any(seen for _p, _o, _n, seen, _c in out):
        pytest.skip("the profiler sees no kernels here")
    assert [x for x in out if x[3] != x[4]] == []
