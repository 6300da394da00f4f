"""A K build that fails halfway leaves nothing running beside its caller's
stream.  The failure is a cuBLAS call that returns an error without doing
anything (a preloaded stand-in, in a process of its own).  The build is called
under stream capture, and ending a capture is an error while a stream that was
forked from it has not been joined."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

FAKE = '''
int cublasGemmEx() { return 13; }                   /* execution failed */
int cublasGemmStridedBatchedEx() { return 13; }
'''

CHILD = '''
import sys
sys.path[:0] = [%(root)r, %(here)r]
import numpy as np
import torch
from helpers import density, dimer
from pyscf_wb97mv_fast_gb300 import _native, cosx
from pyscf_wb97mv_fast_gb300.cosx import CosxBatch, CosxEngine

kind, engine, omegas = sys.argv[1], sys.argv[2], [float(w) for w in sys.argv[3].split(',')]
cosx.set_f_engine(engine)
mol = dimer('synthetic-svp')
dev = torch.device('cuda', torch.cuda.current_device())
rng = np.random.default_rng(1)
engines = [CosxEngine(mol) for _ in range(1 if kind == 'single' else 6)]
grids, qd = [], []
for k, eng in enumerate(engines):
    n = 500 + 64 * k
    grids.append((eng.relative(rng.normal(size=(n, 3))),
                  torch.ones(n, dtype=torch.float64, device=dev)))
    qd.append(torch.as_tensor(density(mol.nao, 10, k), device=dev))
    eng.workspace(eng.workspace_bytes(n))
if kind == 'single':
    def call():
        engines[0].get_k_multi(*grids[0], qd[0], omegas, stats=False)
else:
    batch = CosxBatch(engines, grids, omegas)
    def call():
        batch.run(qd)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
failed = False
with torch.cuda.stream(torch.cuda.Stream()):
    graph.capture_begin(capture_error_mode='thread_local')
    try:
        call()
    except _native.NativeError as e:
        failed = 'GEMM failed' in str(e)
    graph.capture_end()
torch.cuda.synchronize()
raise SystemExit(0 if failed else 5)
'''


# engine 'library': the F product fails; 'tc', which calls no cuBLAS, the K product
@pytest.mark.parametrize('kind,engine,omegas', [
    ('single', 'library', '0.0'), ('single', 'library', '0.0,0.3'),
    ('batch', 'library', '0.0,0.3'), ('batch', 'tc', '0.0'), ('batch', 'tc', '0.0,0.3')])
def test_failed_build_is_joined(tmp_path, kind, engine, omegas):
    src = tmp_path / 'fake.c'
    src.write_text(FAKE)
    fake = tmp_path / 'fake.so'
    subprocess.run(['gcc', '-shared', '-fPIC', '-o', str(fake), str(src)], check=True)
    child = CHILD % dict(root=os.path.dirname(HERE), here=HERE)
    r = subprocess.run([sys.executable, '-c', child, kind, engine, omegas],
                       env=dict(os.environ, LD_PRELOAD=str(fake)), capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout[-2000:], r.stderr[-4000:])
