"""The persisted tuning choices (CSIPM_TUNE_CACHE): lines that no tuning of the
present kernels wrote are passed over and their sizes tuned again."""
import json
import os
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
