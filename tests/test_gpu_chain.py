"""The chained launches of operators and solves, whose kernels may start while
the one before drains, against the same calls with CUDA_LAUNCH_BLOCKING=1, where
no two kernels are ever in flight together.  Every sum has a fixed order, so
solutions, iteration counts and reliable updates have to agree bit for bit over
whole solves; a kernel that read a field before the launch that writes it had
finished would leave other digits.

The sizes take each route: FP64 with four threads per site and with one, the CG
step in the update kernel and in a launch of its own, int16 second passes that
wait with their links requested and those that wait first, batches of 1, 2 and 4
systems per thread, a hopping parameter per system."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import hashlib, json, sys
import numpy as np
sys.path[:0] = [%(root)r, %(root)r + "/bqcd-r399-quda_b200"]
import bqcdg as bq

def links(L, rng):
    m = rng.standard_normal((4, 2, L[0] * L[1] * L[2] * L[3] // 2, 3, 3, 2))
    m = m[..., 0] + 1j * m[..., 1]      # rows: two of a unitary matrix and their cross product
    a = m[..., 0, :] / np.linalg.norm(m[..., 0, :], axis=-1, keepdims=True)
    b = m[..., 1, :] - (a.conj() * m[..., 1, :]).sum(-1, keepdims=True) * a
    b /= np.linalg.norm(b, axis=-1, keepdims=True)
    return np.ascontiguousarray(np.stack([a, b, np.cross(a, b).conj()], -2))

out = {}
def put(name, xs, infos):
    h = hashlib.sha256()
    for x in xs:
        h.update(np.ascontiguousarray(x).tobytes())
    out[name] = [h.hexdigest()] + [[i.niter, i.reliable_updates, i.converged] for i in infos]

HALF, SINGLE, DOUBLE = bq.PREC_HALF, bq.PREC_SINGLE, bq.PREC_DOUBLE
kappa = 0.115
for L, csw, runs in [((8, 8, 8, 8), 1.9, [DOUBLE, SINGLE, HALF]), ((16, 16, 16, 20), 0.0, [DOUBLE, SINGLE, HALF]),
                     ((16, 16, 16, 20), 1.9, [DOUBLE, SINGLE, HALF, "batch", "kappa"])]:
    rng = np.random.default_rng(3)
    volh = L[0] * L[1] * L[2] * L[3] // 2
    para = bq.HmcPara(kappa=kappa, csw=csw, rho=0.05)
    with bq.Lattice(L, (1, 1, 1, -1)) as lat:
        lat.load_gauge(links(L, rng), flipped=False)
        if csw:
            lat.clover_init(para.csw_kappa)
        bs = [rng.standard_normal((volh, 3, 4, 2)).view(np.complex128)[..., 0] for _ in range(8)]
        put("W+W %%s %%s" %% (L, csw), [lat.w_dagger_w(bs[0], para)], [])
        for prec in runs:
            name = "%%s %%s %%s" %% (L, csw, prec)
            if prec == "batch":
                hb, hx = [lat.field(b) for b in bs], [lat.field() for b in bs]
                for p in (HALF, SINGLE):
                    for nbt in (1, 2, 4):
                        for n in (3, 8):
                            for x, b in zip(hx, hb):
                                lat.field_caxpby(x, 0.0, 0.0, b)
                            i = lat.solve_batch(hx[:n], hb[:n], para, precision=p, block=n, rhs_per_thread=nbt)
                            put("%%s %%d %%d %%d" %% (name, p, nbt, n), [lat.field_get(x) for x in hx[:n]], i)
            elif prec == "kappa":
                lat.clover_init_t(csw)
                for x, b in zip(hx, hb):
                    lat.field_caxpby(x, 0.0, 0.0, b)
                i = lat.solve_batch_kappa(hx[:5], hb[:5], para, [0.11 + 0.001 * k for k in range(5)], precision=HALF,
                                          block=5)
                put(name, [lat.field_get(x) for x in hx[:5]], i)
            else:
                x, i = lat.solve(np.zeros_like(bs[0]), bs[0], para, precision=prec)
                put(name, [x], [i])
print(json.dumps(out))
"""


def run(blocking):
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1" if blocking else "0")
    r = subprocess.run([sys.executable, "-c", CHILD % dict(root=ROOT)], env=env, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_chained_equals_one_kernel_at_a_time():
    want = run(True)
    assert len(want) == 3 + 9 + 12 + 1
    for k, v in want.items():
        assert all(i[2] for i in v[1:]), (k, v)  # every solve converged
    for _ in range(3):
        assert run(False) == want
