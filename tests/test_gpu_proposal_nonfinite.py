"""Infinite weights and inputs in the proposal network's convolutions, against
float64 sums of the layers' own terms: a tap that falls outside its input is no
term (not 0 times the weight), and a zero gradient adds nothing to the weights'
(whatever the input there).  In every case all results are finite that way.
Tolerances as in test_gpu_proposal_tiles, derived there.
"""
import numpy as np
import pytest

from oracle import psb_proposal_oracle as P

pytestmark = pytest.mark.gpu

TAPS = [(d, h, w) for d in range(3) for h in range(3) for w in range(3)]


def _window(n, tap):
    """Outputs for which the tap lies inside, and the inputs it reads there."""
    o = [slice(1 if k == 0 else 0, n) for k in tap]
    i = [slice(1 if k == 0 else k - 1, 2 * n - 1 + k, 2) for k in tap]
    return (slice(None), slice(None), *o), (slice(None), slice(None), *i)


def _conv(x, w, b):
    import torch
    n = x.shape[2] // 2
    y = b.reshape(1, -1, 1, 1, 1) + torch.zeros((x.shape[0], len(b), n, n, n), dtype=x.dtype, device=x.device)
    for t, tap in enumerate(TAPS):
        o, i = _window(n, tap)
        y[o] += (x[i][:, None] * w[None, :, :, t, None, None, None]).sum(2)
    return torch.where(y > 0, y, 0.0)


def _conv_grads(x, w, dy):
    import torch
    n = x.shape[2] // 2
    dx, dw = torch.zeros_like(x), torch.zeros_like(w)
    for t, tap in enumerate(TAPS):
        o, i = _window(n, tap)
        dx[i] += (dy[o][:, :, None] * w[None, :, :, t, None, None, None]).sum(1)
        for c in range(w.shape[1]):
            g = dy[o]
            dw[:, c, t] = torch.where(g == 0, 0.0, g * x[i][:, c:c + 1]).sum((0, 2, 3, 4))
    return torch.where(x > 0, dx, 0.0), dw, dy.sum((0, 2, 3, 4))


def _reference(flat, grids, hm, mask, target):
    import torch
    p, off = {}, 0
    for name, shape in P.LAYERS:
        n = int(np.prod(shape))
        v = torch.from_numpy(flat[off:off + n]).reshape(shape)
        off += n
        p[name] = (v if name.endswith(".b") else v.bfloat16()).double().cuda()
    a = [grids.double().reshape(-1, 1, 32, 32, 32)]
    for k in range(4):
        a.append(_conv(a[-1], p[f"c{k}.w"], p[f"c{k}.b"]))
    head = [n for n, _ in P.LAYERS[8:]]
    for n in head:
        p[n].requires_grad_()
    top = a[4].reshape(-1, 512).requires_grad_()
    lin = torch.nn.functional.linear
    f = torch.relu(lin(top, p["f1.w"], p["f1.b"]))
    t = torch.relu(lin(hm.double(), p["f2.w"], p["f2.b"])).repeat_interleave(24, 0)
    h = torch.relu(lin(torch.cat([f, t], 1), p["h1.w"], p["h1.b"]))
    logits = lin(h, p["h2.w"], p["h2.b"]).reshape(-1, 24)
    logp = torch.log_softmax(logits.masked_fill(mask == 0, -np.inf), 1)
    loss = -(target.double() * logp.masked_fill(mask == 0, 0.0)).sum() / len(target)
    g = dict(zip(head + ["top"], torch.autograd.grad(loss, [p[n] for n in head] + [top])))
    dy = torch.where(top > 0, g["top"], 0.0).reshape(a[4].shape)
    for k in (3, 2, 1, 0):
        dy, g[f"c{k}.w"], g[f"c{k}.b"] = _conv_grads(a[k], p[f"c{k}.w"], dy)
    return (logits.detach().cpu().numpy(), loss.item(),
            {n: g[n].detach().reshape(-1).cpu().numpy() for n, _ in P.LAYERS})


def _case(which, rng):
    import torch
    p = P.unpack(P.init_params(6).astype(np.float32))
    p = {k: v.copy() for k, v in p.items()}
    grids = rng.random((24, 32, 32, 32)).astype(np.float32) * 0.2
    if which.startswith("weight"):
        # an infinite weight on the first tap, over an input that is zero
        # wherever that tap reads it: outputs at the near faces do without it
        k = int(which[-1])
        p[f"c{k}.w"][1, 0, 0] = np.inf
        if k == 0:
            grids[:, 1::2, 1::2, 1::2] = 0
        else:
            p[f"c{k - 1}.w"][0] = 0
            p[f"c{k - 1}.b"][0] = 0
        p[f"c{k}.b"][1] = 0.3
    elif which == "gradient":
        # the same tap in the second layer, its input alive at the far face
        # only, which no output reads through it
        p["c1.w"][1, 0, 0] = np.inf
        p["c0.w"][0] = np.abs(p["c0.w"][0])
        p["c0.b"][0] = 0
        p["c0.b"][1:] = 0.1
        grids[:, :30] = 0
    else:
        # infinite inputs that only dead outputs read
        p["c0.w"] = -np.abs(p["c0.w"]) - np.float32(0.01)
        p["c0.b"][:] = 1.5
        for g in grids:
            for _ in range(3):
                g[tuple(rng.integers(0, 32, 3))] = np.inf
            g[0, 0, int(rng.integers(0, 32))] = np.inf
    return P.pack(p).astype(np.float32), torch.from_numpy(grids).cuda()


@pytest.mark.parametrize("which", ["weight0", "weight1", "weight2", "weight3", "gradient", "input"])
def test_terms_that_do_not_exist(gpu_core, which):
    import torch
    from psacking_b200 import proposal
    rng = np.random.default_rng(len(which))
    flat, grids = _case(which, rng)
    hm = torch.from_numpy(rng.random((1, 1024)).astype(np.float32)).cuda()
    mask = torch.ones((1, 24), device="cuda")
    target = torch.zeros((1, 24), device="cuda")
    target[0, 5] = 1.0
    torch.cuda.synchronize()
    net = proposal.Proposal(flat)
    logits, loss = net.run(grids.reshape(24, -1), hm, mask, target)
    got = net.grads()
    net.close()
    want_logits, want_loss, want = _reference(flat, grids, hm, mask, target)
    assert np.isfinite(want_logits).all() and all(np.isfinite(w).all() for w in want.values())
    assert np.abs(logits.cpu().numpy() - want_logits).max() <= 1e-4 * np.abs(want_logits).max()
    assert abs(loss - want_loss) <= 1e-4 * abs(want_loss)
    off, gmax = 0, max(np.abs(w).max() for w in want.values())
    for name, _ in P.LAYERS:
        w = want[name]
        scale = max(np.abs(w).max(), 1e-3 * gmax)
        assert np.abs(got[off:off + w.size] - w).max() <= 2e-3 * scale, name
        off += w.size
