"""Tiles of the proposal's kernels: several tiles per group and per CTA, ragged
ends, domains beyond the box records kept on chip, buffers aligned to four bytes
only.  Tolerances are those of the single-tile tests."""
import numpy as np
import pytest

from oracle import mlp as om

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

NORM = (8.0, 8.0, 8.0, 0.125)
DOMAINS = 1500  # records are kept for the first 1024


def case(n, seed):
    rng = np.random.default_rng(seed)
    lo = rng.uniform(0.0, 15.0, (DOMAINS, 3))
    boxes = np.concatenate([lo, lo + rng.uniform(0.1, 2.0, (DOMAINS, 3))], axis=1).astype(np.float32)
    s = np.zeros(n, om.SAMPLE_DTYPE)
    s["org"] = rng.uniform(-2.0, 18.0, (n, 3))
    d = rng.normal(size=(n, 3))
    s["dir"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    s["ncand"] = rng.integers(0, 9, n)
    s["cand"] = (rng.integers(0, DOMAINS, (n, 1)) + np.arange(8) * 173) % DOMAINS
    s["label"] = np.where(rng.uniform(size=n) < 0.8, rng.integers(0, 8, n) % np.maximum(s["ncand"], 1), -1)
    s["label"][s["ncand"] == 0] = -1
    p = om.init_params(seed)
    p[om.B1:om.W2] = 0.02
    return s, boxes, p


def dev(a, shift=0):
    """`a` on the device, `shift` bytes past an aligned address."""
    raw = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
    t = torch.zeros(raw.size + shift, dtype=torch.uint8, device="cuda")
    t[shift:] = torch.from_numpy(raw.copy()).cuda()
    return t, t.data_ptr() + shift


@pytest.mark.parametrize("n", [1, 129, 128 * 8 * 2 + 7, 128 * 152 * 9 + 31])
def test_forward_rows_do_not_depend_on_their_tile(lib_built, n):
    import spray_gb300 as sg
    s, boxes, p = case(n, 21)
    tb, db = dev(boxes, 4)
    tp, dp = dev(p, 4)
    out = []
    for shift in (0, 4):
        ts, ds = dev(s, shift)
        tl, dl = dev(np.zeros(n * 8, np.float32), shift)
        pred = torch.zeros(n, dtype=torch.int32, device="cuda")
        sg.mlp_forward(dp, db, NORM, ds, n, dl, pred.data_ptr())
        out.append((tl[shift:].cpu().numpy().view(np.float32).reshape(n, 8), pred.cpu().numpy()))
    assert np.array_equal(out[0][0].view(np.uint32), out[1][0].view(np.uint32))
    assert np.array_equal(out[0][1], out[1][1])
    got, pred = out[0]
    some = np.unique(np.concatenate([np.arange(min(n, 300)), np.arange(max(0, n - 300), n)]))
    want, _ = om.forward(p, s[some], boxes, NORM)
    fin = np.isfinite(want)
    assert np.array_equal(np.isfinite(got[some]), fin)
    assert np.allclose(got[some][fin], want[fin], atol=2e-2, rtol=2e-2)
    has = s["ncand"] > 0
    assert np.array_equal(pred[has], np.argmax(got, axis=1)[has])


@pytest.mark.parametrize("n", [129, 128 * 152 + 1, 128 * 152 * 2 + 77, 128 * 152 * 4])
def test_gradient_over_several_tiles_a_cta(lib_built, n):
    import spray_gb300 as sg
    s, boxes, p = case(n, 33)
    tb, db = dev(boxes, 4)
    tp, dp = dev(p, 4)
    grads = []
    for shift in (0, 4):
        ts, ds = dev(s, shift)
        grad = torch.zeros(om.PARAMS + 2, dtype=torch.float32, device="cuda")
        sg.mlp_grad(dp, db, NORM, ds, n, grad.data_ptr())
        grads.append(grad.cpu().numpy())
    assert np.array_equal(grads[0].view(np.uint32), grads[1].view(np.uint32))
    g = grads[0]
    want, loss, cnt = om.grad(p, s, boxes, NORM)
    assert g[om.PARAMS + 1] == cnt
    assert abs(g[om.PARAMS] - loss) <= 1e-3 * max(1.0, abs(loss))
    for a, b in ((om.W1, om.B1), (om.B1, om.W2), (om.W2, om.B2), (om.B2, om.W3), (om.W3, om.B3), (om.B3, om.W4),
                 (om.W4, om.B4), (om.B4, om.PARAMS)):
        err = np.linalg.norm(g[a:b] - want[a:b]) / max(np.linalg.norm(want[a:b]), 1e-12)
        assert err < 3e-2, (a, err)
