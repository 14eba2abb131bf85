"""Pruner.fit's host side on the CPU: a library that only records its calls stands in for the kernels."""
import numpy as np
import pytest
import torch


class _Recorder:
    """Entry points that return 0; the addresses of every grouped Adam step."""

    def __init__(self):
        self.adam = []

    def __getattr__(self, name):
        if name == "vk_adam_group":
            return self._adam_group
        return lambda *a: 0

    def _adam_group(self, ref, n, *_):
        self.adam.append([(t.n, t.p, t.g, t.m, t.v, t.p_bf16) for t in ref._obj[:n]])
        return 0


@pytest.fixture
def pruner(monkeypatch):
    from vulcan.gpu import _lib as K
    from vulcan.gpu import prune as PR
    rec = _Recorder()
    monkeypatch.setattr(K, "lib", lambda: rec)
    monkeypatch.setattr(K, "ptr", lambda t: None if t is None else t.data_ptr())
    monkeypatch.setattr(K, "stream", lambda: None)
    return PR, PR.Pruner("cpu"), rec


def _addresses(PR, pr):
    return [(pr.w[k].numel(), pr.w[k].data_ptr(), pr._grad[k].data_ptr(), pr._adam[k][0].data_ptr(),
             pr._adam[k][1].data_ptr(), pr.bf[k].data_ptr() if k in pr.bf else None) for k in PR._PARAMS]


def test_adam_takes_the_tensors_of_its_step(pruner):
    """Weights loaded by fit's callback, and gradients of a validation pass of another size, are what the next epoch's
    steps update: no address of the tensors before them."""
    PR, pr, rec = pruner
    n, batch = 96, 32
    feat, y = torch.zeros(n, PR.N_IN, dtype=torch.bfloat16), torch.zeros(n)
    seen, keep = [], []

    def log(_):
        seen.append(_addresses(PR, pr))
        keep.append((dict(pr.w), pr._adam, pr._grad, pr.bf))   # alive, so that no address comes again
        pr.load_state_dict({k: np.array(v) for k, v in pr.state_dict().items()})
        pr.forward_train(torch.zeros(7, PR.N_IN), 7)
    pr.fit(feat, y, epochs=3, batch=batch, log=log)
    assert len(rec.adam) == 9
    for ep in range(3):
        assert all(step == seen[ep] for step in rec.adam[3 * ep:3 * ep + 3])
    flat = [{a for t in s for a in t[1:] if a} for s in seen]
    assert not flat[0] & flat[1] and not flat[1] & flat[2]


def test_adam_takes_gradients_replaced_between_steps(pruner):
    PR, pr, rec = pruner
    grads = []

    class Clipped(PR.Pruner):
        def backward(self, *a):
            out = super().backward(*a)
            self._grad = {k: v.clamp(-1, 1) for k, v in self._grad.items()}
            grads.append(self._grad)
            return out

        def adam_step(self, lr, b1=0.9, b2=0.999, eps=1e-8, wd=0.0):
            super().adam_step(lr, b1, b2, eps, wd)
    Clipped("cpu").fit(torch.zeros(64, PR.N_IN, dtype=torch.bfloat16), torch.zeros(64), epochs=1, batch=32)
    assert [[t[2] for t in step] for step in rec.adam] == [[g[k].data_ptr() for k in PR._PARAMS] for g in grads]


@pytest.mark.parametrize("shape,ok", [((64,), True), ((70,), True), ((64, 1), True), ((63,), False), ((1,), False),
                                      ((1, 64), False), ((), False)])
def test_weights_have_a_row_per_target(pruner, shape, ok):
    PR, pr, rec = pruner
    args = (torch.zeros(64, PR.N_IN, dtype=torch.bfloat16), torch.zeros(64), torch.ones(shape))
    if ok:
        assert len(pr.fit(*args, epochs=1, batch=32)) == 1
    else:
        with pytest.raises(ValueError):
            pr.fit(*args, epochs=1, batch=32)
        assert not rec.adam
