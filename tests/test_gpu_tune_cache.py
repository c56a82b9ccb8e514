"""The persisted tuning choices (CSIPM_TUNE_CACHE): lines that no tuning of the
present kernels wrote are passed over and their sizes tuned again, and a width
that does not fit leaves the heuristic's configuration."""
import json
import os
import re
import subprocess
import sys

import pytest

from conftest import ORACLE, PKG

pytestmark = pytest.mark.gpu

CODE = """import sys; sys.path[:0] = [%r, %r]; import numpy as np, torch, csipm, oracle as O
size = %r
N = int(np.prod(size))
rng = np.random.default_rng(0)
op = csipm.FFTOperator(csipm.FFTParameters(len(size), size, torch.zeros(N, dtype=torch.float64, device='cuda'), 0.1, None))
x = rng.standard_normal(N)
y = op.M_perpt_M_perp_vec(torch.tensor(x, device='cuda')).cpu().numpy()
r = O.Operator(size).AtA(x)
assert np.linalg.norm(y - r) <= 1e-12 * np.linalg.norm(r)
op.close()
"""


def _open(path, size):
    subprocess.run([sys.executable, "-c", CODE % (PKG, ORACLE, size)], env=dict(os.environ, CSIPM_TUNE_CACHE=str(path)),
                   check=True, timeout=600)
    return [json.loads(line) for line in path.read_text().splitlines()]


def _write(path, entry):
    path.write_text(json.dumps(entry) + "\n")


def test_lines_of_other_kernels_are_tuned_again(cuda, tmp_path):
    size = (48, 40, 36)
    own = tmp_path / "own.jsonl"
    written = _open(own, size)
    assert len(written) == 1 and len(_open(own, size)) == 1   # its own line is taken
    old = dict(written[0])
    gen = old.pop("gen")                                      # before generations were written
    older = {k: v for k, v in old.items() if k != "s2_two"}   # before dim 2 was tuned
    wide = dict(written[0], s3_tb=3, row_rb=5)                # widths no tuning chooses
    for k, entry in enumerate([old, older, dict(old, gen=gen - 1), wide]):
        path = tmp_path / f"f{k}.jsonl"
        _write(path, entry)
        lines = _open(path, size)
        assert len(lines) == 2 and lines[0] == entry and lines[1]["gen"] == gen, entry


@pytest.mark.parametrize("size,fits_not", [((4, 4, 1000), {"s3_two": 0, "s3_tb": 16}), ((6, 2000), {"s2_two": 0, "s2_tb": 8}),
                                           ((3000, 64), {"row_two": 0, "row_rb": 16}), ((12804, 4), {"row_two": 0, "row_rb": 1})],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "")
def test_a_choice_that_does_not_fit(cuda, tmp_path, size, fits_not):
    """The heuristic's configuration stays, so the product runs and is right."""
    with open(os.path.join(PKG, "csrc", "tune.cuh")) as f:
        gen = int(re.search(r"TUNE_GEN = (\d+)", f.read()).group(1))
    n = list(size) + [1] * (3 - len(size))
    entry = dict(elem=8, dim=len(size), n=n, masked=0, s3_two=1, s3_tb=0, s2_tb=0, row_two=1, row_rb=0, s2_two=1, gen=gen)
    path = tmp_path / "f.jsonl"
    entry.update(fits_not)
    _write(path, entry)
    assert len(_open(path, size)) == 1   # taken, not tuned again
