"""A stored tuning choice is an index into a list of candidates: it is used with that list alone.  A
choice whose result differs in the last bits from the heuristic's (another K split) is taken from
a file that this build wrote, and not from the same line without its list or with another one."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# one product of ~1.2 GFLOP with few output tiles: its candidates split K differently
CODE = r"""
import sys
import hashlib
import torch
from dirac_caspt2_gb300 import api
m, n, k = 128, 96, 12288
g = torch.Generator(device="cuda").manual_seed(5)
rnd = lambda a, b: torch.complex(torch.randn((a, b), generator=g, device="cuda", dtype=torch.float64),
                                 torch.randn((a, b), generator=g, device="cuda", dtype=torch.float64))
A, B, C = rnd(k, m), rnd(n, k), rnd(n, m)
torch.cuda.synchronize()
with api.Caspt2Session(0) as ses:
    ses.lib.dcg_set_autotune_trials(ses.h, int(sys.argv[1]))
    ses.zgemm(api.DCG_PREC_FP64, m, n, k, 1, A.data_ptr(), 1, m, 0, B.data_ptr(), k, False, C.data_ptr(), 1, m, 0)
print(hashlib.sha256(C.cpu().numpy().tobytes()).hexdigest())
"""


def _product(path, trials):
    env = dict(os.environ, DCG_TUNE_FILE=str(path), PYTHONPATH=ROOT)
    out = subprocess.run([sys.executable, "-c", CODE, str(int(trials))], capture_output=True, text=True, env=env, cwd=ROOT)
    assert out.returncode == 0, out.stderr
    return out.stdout.strip()


def test_choice_belongs_to_its_list(gpu_lib, tmp_path):
    pytest.importorskip("torch")
    f = tmp_path / "tune.txt"
    heuristic = _product(f, False)
    assert not f.exists()
    _product(f, True)
    (line,) = f.read_text().splitlines()
    key, ncand, ms, ident = line.split()[:6], int(line.split()[7]), line.split()[8:10], line.split()[10]
    assert ncand > 1 and int(ident) != 0
    used = 0
    for choice in range(1, ncand):
        fields = [*key, str(choice), str(ncand), *ms]
        f.write_text(" ".join([*fields, ident]) + "\n")
        if _product(f, False) == heuristic:
            continue
        used += 1   # the choice shows in the bits: without its list, or with another, it must not
        for other in (fields, [*fields, str(int(ident) ^ 1)]):
            f.write_text(" ".join(other) + "\n")
            assert _product(f, False) == heuristic
        break
    assert used
