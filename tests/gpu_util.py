"""Shared helpers of the GPU parity tests."""
import numpy as np
import torch


def gate(actual, reference, what="", rel_bound=1e-3, nrmse_bound=3e-5):
    """The reference project's acceptance criterion (docs/GPU_TESTS.md:126-131):
    maxabs <= 5e-4*max(1,max|ref|) and NRMSE <= 3e-5, no non-finite value; plus a
    per-output relative bound of 1e-3 whose denominator is floored at 1e-2*max|ref| of
    the row.  The floor is needed because every output is a +-sum of 128 core values
    (the output H128), so its error scales with the block, not with the output itself:
    outputs that cancel to ~0 have unbounded plain relative error under ANY
    re-association of the fp32 sum (measured: 1e-2 for a plain re-ordered CPU sum)."""
    a = np.asarray(actual, dtype=np.float64)
    r = np.asarray(reference, dtype=np.float64)
    assert a.shape == r.shape, (what, a.shape, r.shape)
    assert np.isfinite(a).all(), what
    err = np.abs(a - r)
    maxref = np.abs(r).max() if r.size else 0.0
    assert err.max(initial=0.0) <= 5e-4 * max(1.0, maxref), (what, err.max(), maxref)
    nrmse = np.sqrt((err ** 2).sum() / max((r ** 2).sum(), 1e-30))
    assert nrmse <= nrmse_bound, (what, nrmse)
    if r.ndim == 2 and r.size:
        floor = 1e-2 * np.abs(r).max(axis=1, keepdims=True)
        rel = err / np.maximum(np.abs(r), np.maximum(floor, 1e-30))
        assert rel.max() <= rel_bound, (what, rel.max())


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    return t.detach().cpu().numpy()


def linear64(w, layer, x):
    """The linear of prepared weights `w` with the sums in 64 bits: the decoded weights and the core input
    are the device's own (bit-exact by their own tests), everything after them is float64."""
    h = torch.ones(1, 1, dtype=torch.float64)
    while h.shape[0] < 128:
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
    h = (h / 128 ** 0.5).cuda()
    core = w.input_stages(x)[2].double() @ w.dequantize().double()
    y = (core.view(x.shape[0], -1, 128) @ h).view(x.shape[0], -1) * dev(np.asarray(layer.svh).view(np.float16)).double()
    return y if layer.bias is None else y + dev(layer.bias).double()
