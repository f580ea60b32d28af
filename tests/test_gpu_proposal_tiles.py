"""The proposal network's blocked layers at the batch sizes where their tiles
change or end (24 samples per item; the last three convolutions take smaller
tiles below 296, 592 and 1184 samples, which lie between 12 and 13, 24 and 25,
and 49 and 50 items), against plain torch in float64 with the same BF16
weights.  Tolerances: an FP32 sum of n terms is off by at most about n * 2^-24
of the sum of magnitudes; the longest forward chain is 1,728 terms and its
magnitudes stay within 50 times the result's scale, so 1e-4 of the largest
logit; gradients sum up to 6.3 million signed terms in partial sums, 2e-3 of a
layer's largest gradient, as in test_gpu_proposal.
"""
import numpy as np
import pytest

from oracle import psb_proposal_oracle as P

pytestmark = pytest.mark.gpu


def _reference(flat, grids, hm, mask, target):
    import torch
    p, off = {}, 0
    for name, shape in P.LAYERS:
        n = int(np.prod(shape))
        v = torch.from_numpy(flat[off:off + n]).reshape(shape)
        off += n
        v = v if name.endswith(".b") else v.bfloat16()
        p[name] = v.double().cuda().requires_grad_()
    names = [n for n, _ in P.LAYERS]
    x = grids.double().reshape(-1, 1, 32, 32, 32)
    feats = []
    for c in x.split(192):
        for k in range(4):
            w = p[names[2 * k]].reshape(-1, c.shape[1], 3, 3, 3)
            c = torch.relu(torch.nn.functional.conv3d(c, w, p[names[2 * k + 1]], stride=2, padding=1))
        feats.append(torch.relu(torch.nn.functional.linear(c.reshape(c.shape[0], -1), p[names[8]], p[names[9]])))
    t = torch.relu(torch.nn.functional.linear(hm.double(), p[names[10]], p[names[11]])).repeat_interleave(24, 0)
    h = torch.relu(torch.nn.functional.linear(torch.cat([torch.cat(feats), t], 1), p[names[12]], p[names[13]]))
    logits = torch.nn.functional.linear(h, p[names[14]], p[names[15]]).reshape(-1, 24)
    logp = torch.log_softmax(logits.masked_fill(mask == 0, -np.inf), 1)
    has = (target.sum(1) > 0) & (mask.sum(1) > 0)
    loss = -(target.double() * logp.masked_fill(mask == 0, 0.0))[has].sum() / max(1, int(has.sum()))
    g = torch.autograd.grad(loss, [p[n] for n in names])
    return logits.detach().cpu().numpy(), loss.item(), [v.reshape(-1).cpu().numpy() for v in g]


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("B", [1, 2, 12, 13, 24, 25, 49, 50])
def test_layers_match_float64(gpu_core, B, offset):
    """offset 1: the grids start 4 bytes past an aligned address."""
    import torch
    from psacking_b200 import proposal
    if offset and B > 2:
        pytest.skip("alignment does not depend on the batch")
    rng = np.random.default_rng(100 + B)
    flat = P.init_params(4).astype(np.float32)
    buf = torch.zeros(B * 24 * 32 ** 3 + offset, dtype=torch.float32, device="cuda")
    grids = buf[offset:].reshape(B * 24, 32 ** 3)
    grids.copy_(torch.from_numpy((rng.random((B * 24, 32 ** 3)) < 0.1).astype(np.float32)))
    hm = torch.from_numpy(rng.random((B, 1024)).astype(np.float32)).cuda()
    mask = torch.ones((B, 24), device="cuda")
    mask[0, 20:] = 0
    target = torch.zeros((B, 24), device="cuda")
    for b in range(B):
        target[b, int(rng.integers(0, 20))] = 1.0
    torch.cuda.synchronize()
    net = proposal.Proposal(flat)
    logits, loss = net.run(grids, hm, mask, target)
    got = net.grads()
    net.close()
    want_logits, want_loss, want = _reference(flat, grids, hm, mask, target)
    assert np.abs(logits.cpu().numpy() - want_logits).max() <= 1e-4 * np.abs(want_logits).max()
    assert abs(loss - want_loss) <= 1e-4 * abs(want_loss)
    off, gmax = 0, max(np.abs(w).max() for w in want)
    for (name, _), w in zip(P.LAYERS, want):
        scale = max(np.abs(w).max(), 1e-3 * gmax)
        assert np.abs(got[off:off + w.size] - w).max() <= 2e-3 * scale, name
        off += w.size


@pytest.mark.parametrize("offset", [0, 1, 2])
def test_item_grids_any_destination(gpu_core, offset):
    """Extents that end inside a group of four cells, and destinations that
    start 0, 4 and 8 bytes past a 16-byte boundary: equal to the oracle, and
    nothing written before or behind."""
    import torch
    from psacking_b200 import proposal
    from psacking_b200.rotations import orientation_maps
    rng = np.random.default_rng(9)
    maps = np.ascontiguousarray(orientation_maps(24), np.int32)
    items = [(rng.random(s) < 0.5).astype(np.int32) for s in [(1, 2, 3), (5, 7, 6), (33, 9, 31), (2, 64, 1)]]
    n = len(items) * 24 * 32 ** 3
    buf = torch.full((n + 8,), -1.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    arr, dims = proposal._ptrs(items)
    proposal.check(proposal.lib().psb_prop_item_grids(arr, dims.ctypes.data, len(items), maps.ctypes.data, len(maps),
                                                      buf.data_ptr() + 4 * offset))
    got = buf.cpu().numpy()
    assert (got[:offset] == -1).all() and (got[offset + n:] == -1).all()
    got = got[offset:offset + n].reshape(len(items), 24, 32, 32, 32)
    for k, it in enumerate(items):
        assert np.array_equal(got[k], P.oriented_grids(it, maps)), k
