"""The solvers that lambda_max keeps per input shape hold a bounded amount of C = A·Aᵀ between them: past
the limit those used longest ago give theirs back, and go on returning the same λ and gradients (within
FP32 rounding, 2e-6 of λ and 1e-5 of the largest gradient entry, at tolerance 1e-6)."""
import pytest
import torch


class _Fake:
    def __init__(self, held):
        self.held, self.released = held, 0

    def c_bytes(self):
        return self.held

    def release_c(self):
        self.held, self.released = 0, self.released + 1


def test_longest_unused_give_back_first(monkeypatch):
    from collections import OrderedDict
    from eigenvaluecomputation_by_amm_b200 import autograd as G
    a, b, c, other, none = _Fake(40), _Fake(50), _Fake(30), _Fake(500), _Fake(0)
    monkeypatch.setattr(G, "_SOLVERS", OrderedDict(
        [((0, "none"), none), ((0, "a"), a), ((1, "other"), other), ((0, "b"), b), ((0, "c"), c)]))
    monkeypatch.setattr(G, "_c_limit", lambda device: 80)
    G._bound_c(0)
    assert (a.released, b.released, c.released, other.released) == (1, 0, 0, 0)
    G._bound_c(0)
    assert (a.released, b.released, c.released) == (1, 0, 0)
    monkeypatch.setattr(G, "_c_limit", lambda device: 20)     # the one in use gives back its own too
    G._bound_c(0)
    assert b.held == c.held == 0 and other.released == 0


@pytest.mark.gpu
def test_results_after_c_is_given_back(amm_lib, monkeypatch):
    from eigenvaluecomputation_by_amm_b200 import autograd as G
    monkeypatch.setattr(G, "_SOLVERS", type(G._SOLVERS)())
    g = torch.Generator(device="cuda").manual_seed(3)
    shapes = [(8, 256, 2600), (8, 260, 2600), (8, 264, 2600)]
    inputs = []
    for B, m, n in shapes:
        A = torch.randn(B, m, n, device="cuda", generator=g)
        A[:, :, 0] *= 12.0                    # a gap above the rest
        inputs.append(A)

    def call(A):
        A = A.detach().requires_grad_(True)
        lam = G.lambda_max(A)
        lam.sum().backward()
        return lam.detach(), A.grad

    first = [call(A) for A in inputs]
    held = [s.c_bytes() for s in G._SOLVERS.values()]
    assert min(held) >= 8 * 256 * 256 * 4     # the autotuner kept C at these sizes
    late = G.lambda_max(inputs[0].detach().requires_grad_(True))   # its backward comes after
    monkeypatch.setattr(G, "_c_limit", lambda device: max(held))
    call(torch.randn(8, 268, 2600, device="cuda", generator=g))
    assert sum(s.c_bytes() for s in G._SOLVERS.values()) <= max(held)
    late.sum().backward()
    for A, (lam, grad) in zip(inputs, first):
        lam2, grad2 = call(A)
        assert float(((lam2 - lam).abs() / lam).max()) < 2e-6
        assert float((grad2 - grad).abs().max()) < 1e-5 * float(grad.abs().max())
