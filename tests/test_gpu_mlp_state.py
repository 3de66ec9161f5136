"""What the proposal's entry points keep between calls: a workspace per thread and
device.  It has to survive a reset of the device, and threads may not share it."""
import subprocess
import sys
import threading
from pathlib import Path

import numpy as np
import pytest

from oracle import mlp as om

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

# no torch in this process: the reset takes the whole context, whoever uses it
RESET = r"""
import ctypes as C, glob, os, sys
import numpy as np
import spray_gb300 as sg
from oracle import mlp as om

rt = C.CDLL(sorted(glob.glob(os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "lib64", "libcudart.so.*")))[0])


def dev(a):
    p = C.c_void_p()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)) == 0
    assert rt.cudaMemcpy(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 1) == 0
    return p.value


def host(p, like):
    a = np.zeros_like(like)
    assert rt.cudaMemcpy(a.ctypes.data_as(C.c_void_p), C.c_void_p(p), C.c_size_t(a.nbytes), 2) == 0
    return a


rng = np.random.default_rng(5)
n, norm = 700, (0.0, 0.0, 0.0, 1.0)
lo = rng.uniform(-1, 0.5, (64, 3))
boxes = np.concatenate([lo, lo + 0.4], 1).astype(np.float32)
s = np.zeros(n, om.SAMPLE_DTYPE)
s["org"], s["dir"], s["ncand"] = rng.uniform(-2, 2, (n, 3)), rng.normal(size=(n, 3)), 8
s["cand"], s["label"] = rng.integers(0, 64, (n, 8)), rng.integers(0, 8, n)
params = om.init_params(5)


def calls():
    logits, pred, grad = np.zeros((n, 8), np.float32), np.zeros(n, np.int32), np.zeros(om.PARAMS + 2, np.float32)
    db, ds, dp = dev(boxes), dev(s), dev(params)
    dl, dq, dg, dm, dv, dw = dev(logits), dev(pred), dev(grad), dev(0 * params), dev(0 * params), dev(np.zeros(3, np.float32))
    sg.mlp_forward(dp, db, norm, ds, n, dl, dq)
    sg.mlp_grad(dp, db, norm, ds, n, dg)
    out = [host(dl, logits), host(dq, pred), host(dg, grad)]
    sg.mlp_train(dp, dm, dv, db, norm, ds, n, 256, 1e-3, 3, 1, dw)
    return out + [host(dp, params), host(dw, np.zeros(3, np.float32))]


want = calls()
for _ in range(2):
    assert rt.cudaDeviceReset() == 0
    got = calls()
    assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(want, got))
print("same after a reset")
"""


def test_calls_after_a_device_reset(lib_built):
    r = subprocess.run([sys.executable, "-c", RESET], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode == 0 and "same after a reset" in r.stdout, (r.returncode, r.stdout[-500:], r.stderr[-2000:])


def test_threads_side_by_side(lib_built):
    torch = pytest.importorskip("torch")
    import spray_gb300 as sg
    rng = np.random.default_rng(6)
    norm = (0.0, 0.0, 0.0, 1.0)
    lo = rng.uniform(-1, 0.5, (64, 3))
    boxes = torch.from_numpy(np.concatenate([lo, lo + 0.4], 1).astype(np.float32)).cuda()

    def job(seed):
        r = np.random.default_rng(seed)
        n = 5000 + 611 * seed
        s = np.zeros(n, om.SAMPLE_DTYPE)
        s["org"], s["dir"], s["ncand"] = r.uniform(-2, 2, (n, 3)), r.normal(size=(n, 3)), 8
        s["cand"], s["label"] = r.integers(0, 64, (n, 8)), r.integers(0, 8, n)
        ts = torch.from_numpy(s.view(np.uint8)).cuda()
        p = torch.from_numpy(om.init_params(seed)).cuda()
        m, v = torch.zeros_like(p), torch.zeros_like(p)
        loss = torch.zeros(6, device="cuda")
        torch.cuda.synchronize()

        def run():
            sg.mlp_train(p.data_ptr(), m.data_ptr(), v.data_ptr(), boxes.data_ptr(), norm, ts.data_ptr(), n, 2048, 1e-3, 6, 1,
                         loss.data_ptr())

        return run, lambda: np.concatenate([p.cpu().numpy(), loss.cpu().numpy()]).view(np.uint32)

    want = []
    for k in range(4):
        run, result = job(k)
        run()
        want.append(result())
    jobs = [job(k) for k in range(4)]
    threads = [threading.Thread(target=run) for run, _ in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, (_, result) in enumerate(jobs):
        assert np.array_equal(result(), want[k]), k
