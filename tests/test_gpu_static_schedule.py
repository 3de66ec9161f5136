"""spray_gpu_schedule_static on rays with components that are not finite, against the
oracle's exact slab tests: the group test in front of them may not turn away a
domain that they accept (a NaN component is dropped by their comparisons)."""
import numpy as np
import pytest

import spray_gb300 as sg
from conftest import small_config

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("domains", [1, 3, 27, 30])
@pytest.mark.parametrize("where", ["org", "dir", "both"])
def test_rays_that_are_not_finite(lib_built, oracle_mod, domains, where):
    rng = np.random.default_rng(domains)
    lo = rng.uniform(-4, 3, (domains, 3))
    bounds = np.concatenate([lo, lo + rng.uniform(0.5, 3, (domains, 3))], 1).astype(np.float32)
    n = 4001
    org = rng.uniform(-6, 6, (n, 3)).astype(np.float32)
    dr = rng.normal(size=(n, 3)).astype(np.float32)
    dr = (dr / np.linalg.norm(dr, axis=1, keepdims=True)).astype(np.float32)
    odd = np.array([np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-39, -1e-42, 3e38], np.float32)
    for a in ((org,) if where == "org" else (dr,) if where == "dir" else (org, dr)):
        hit = rng.random((n, 3)) < 0.3
        a[hit] = rng.choice(odd, hit.sum())
        a[:40] = odd[0]  # every component
        a[40:80] = odd[1]
    doms = [sg.Domain(np.array([b[:3], b[3:], b[:3]], np.float32), np.array([[0, 1, 2]], np.uint32), bounds=b) for b in bounds]
    o = oracle_mod.Oracle(small_config(), sg.Scene(doms, [sg.Light(0, (0, 0, 9))]))
    want, _ = o.schedule(org, dr)
    o.close()
    want = want[np.lexsort((want["depth"], want["ray"], want["domain"]))]
    to4 = lambda a: torch.from_numpy(np.concatenate([a, np.zeros((len(a), 1), np.float32)], 1)).cuda()
    bnd, o4, d4 = torch.from_numpy(bounds).cuda(), to4(org), to4(dr)
    cap = len(want) + 64
    entries = torch.zeros((cap, 2), dtype=torch.int32, device="cuda")
    starts = torch.zeros(domains + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    k = sg.schedule_static(bnd.data_ptr(), domains, o4.data_ptr(), d4.data_ptr(), n, 16, entries.data_ptr(), cap,
                           starts.data_ptr())
    e = entries[:k].cpu().numpy().view(np.uint32)
    dom = np.repeat(np.arange(domains), np.diff(starts.cpu().numpy().astype(np.int64)))
    assert k == len(want)
    assert np.array_equal(dom, want["domain"])
    assert np.array_equal(e[:, 0] & ((1 << 26) - 1), want["ray"])
    assert np.array_equal((e[:, 0] >> 26) & 31, want["depth"])
    assert np.array_equal(e[:, 1], want["tdom"].view(np.uint32))
