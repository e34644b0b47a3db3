"""A host call of few rays that fails leaves the caller's arrays alone. The
failure is a host-side one: the call waits for its stream, which CUDA refuses
while the stream is being captured (the capture is invalidated, nothing runs).
In a process of its own, since CUDA keeps the refusal as the thread's last
error."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
    import ctypes as C, sys
    import numpy as np, torch
    from kazen_proto_gb300 import _native as N, scenes

    query, n = sys.argv[1], 100
    drv = C.CDLL("libcuda.so.1")
    s = scenes.soup_desc(scenes.triangle_soup(3000, seed=5)).build()
    rays = scenes.soup_rays(n, seed=1)
    stream = torch.cuda.Stream()
    s.set_stream(stream)
    out = {k: np.empty(n, t) for k, t in (("t", np.float32), ("prim_id", np.uint32), ("geom_id", np.uint32),
                                          ("u", np.float32), ("v", np.float32), ("occ", np.uint8))}

    def call():
        for a in out.values():
            a.view(np.uint8)[:] = 0xA5
        p = rays.ctypes.data_as(C.c_void_p)
        if query == "any":
            return N.lib().kz_intersect_any(s.handle, p, n, out["occ"].ctypes.data_as(C.c_void_p), N.KZ_MEM_HOST)
        hits = N.KzHits(*(out[k].ctypes.data for k in ("t", "prim_id", "geom_id", "u", "v")))
        return N.lib().kz_intersect_closest(s.handle, p, n, hits, N.KZ_MEM_HOST)

    def written():
        return [k for k, a in out.items() if (a.view(np.uint8) != 0xA5).any()]

    N.check(call())
    assert written() == (["occ"] if query == "any" else ["t", "prim_id", "geom_id", "u", "v"])
    handle, graph = C.c_void_p(stream.cuda_stream), C.c_void_p()
    assert drv.cuStreamBeginCapture_v2(handle, 1) == 0  # thread-local mode
    rc = call()
    drv.cuStreamEndCapture(handle, C.byref(graph))
    assert rc == N.KZ_ERR_CUDA, rc
    assert written() == [], written()
    print("arrays untouched")
"""


@pytest.mark.parametrize("query", ["closest", "any"])
def test_failed_call_writes_nothing(gpu, query):
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(CHILD), query], capture_output=True, text=True, cwd=ROOT,
                       timeout=300)
    assert r.returncode == 0 and "arrays untouched" in r.stdout, r.stdout + r.stderr
