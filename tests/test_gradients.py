"""Gradients: the module's come from the backward kernels (csrc/ma_backward.cu), or from a recomputation in tensor operations
where those do not apply (monarch_attention_b200/backward.py); the reference differentiates its eager implementation with
autograd.  tests/golden holds the reference's own
gradients on seeded cases (generated by tests/golden/make_golden.py)."""
import numpy as np
import pytest
import torch

from cases import GRAD_CASES, grad_weights
from helpers import bits_to_float, error_metrics, golden, make_inputs
from make_golden import grad_sample_positions, to_bits

# relative Frobenius bounds for gradients against the reference's (same inputs, same cotangent): the CPU
# recomputation runs the same operations in the same order, the GPU one sums in a different order
GRAD_TOL_CPU = {"f32": 1e-6, "bf16": 1e-6, "f16": 1e-6}
GRAD_TOL_GPU = {"f32": 1e-4, "bf16": 3e-2, "f16": 1e-2}


def _stored(name, key, dtype):
    return bits_to_float(golden()[f"{name}/{key}"], dtype)


def _sampled(t, dtype):
    flat = to_bits(t.detach().cpu()).reshape(-1)
    return bits_to_float(flat[grad_sample_positions(flat.size)], dtype)


@pytest.mark.parametrize("case", GRAD_CASES, ids=lambda c: c["name"])
def test_recomputation_on_cpu_gives_the_reference_output_and_gradients(case):
    """The differentiable restatement the backward pass uses, run on the CPU: the bits of the reference's
    output, and its gradients."""
    from monarch_attention_b200.backward import differentiable_forward
    q, k, v, mask = make_inputs(case)
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    out = differentiable_forward(q, k, v, mask, case["T"], case["B"], case["pre_pad"])
    assert np.array_equal(_sampled(out, case["vdtype"]), _stored(case["name"], "out", case["vdtype"]))
    out.backward(grad_weights(case).to(out.dtype))
    for key, t, dt in (("dq", q.grad, case["dtype"]), ("dk", k.grad, case["dtype"]), ("dv", v.grad, case["vdtype"])):
        _, _, fro = error_metrics(_sampled(t, dt), _stored(case["name"], key, dt))
        assert fro <= GRAD_TOL_CPU[dt], (key, fro)


@pytest.mark.parametrize("case", GRAD_CASES, ids=lambda c: c["name"])
def test_oracle_autograd_gives_the_reference_gradients(case):
    """The CPU oracle is differentiable too; its gradients pin the same numbers from the test side."""
    from oracle.monarch_oracle import monarch_attention_oracle
    q, k, v, mask = make_inputs(case)
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    out = monarch_attention_oracle(q, k, v, mask, case["T"], case["B"], case["pre_pad"])
    out.backward(grad_weights(case).to(out.dtype))
    for key, t, dt in (("dq", q.grad, case["dtype"]), ("dk", k.grad, case["dtype"]), ("dv", v.grad, case["vdtype"])):
        _, _, fro = error_metrics(_sampled(t, dt), _stored(case["name"], key, dt))
        assert fro <= GRAD_TOL_CPU[dt], (key, fro)


@pytest.mark.gpu
@pytest.mark.parametrize("case", GRAD_CASES, ids=lambda c: c["name"])
def test_module_gradients_match_the_reference(case):
    """Through the module API on the GPU: the forward result is the kernels' (bit for bit the result of a call
    without gradients), the gradients are the reference's within the tolerance of the storage type."""
    import monarch_attention_b200 as ma
    dev = torch.device("cuda:0")
    q, k, v, mask = make_inputs(case)
    q, k, v = (t.to(dev).requires_grad_(True) for t in (q, k, v))
    mask = None if mask is None else mask.to(dev)
    mod = ma.MonarchAttention(case["B"], case["T"], "pre" if case["pre_pad"] else "post")
    out = mod(q, k, v, mask)
    assert out.requires_grad
    with torch.no_grad():
        plain = mod(q, k, v, mask)
    assert torch.equal(out.detach(), plain)
    out.backward(grad_weights(case).to(dev).to(out.dtype))
    for key, t, dt in (("dq", q.grad, case["dtype"]), ("dk", k.grad, case["dtype"]), ("dv", v.grad, case["vdtype"])):
        assert t is not None and torch.isfinite(t.float()).all()
        _, _, fro = error_metrics(_sampled(t, dt), _stored(case["name"], key, dt))
        assert fro <= GRAD_TOL_GPU[dt], (key, fro)


@pytest.mark.gpu
def test_only_the_requested_gradients_are_computed():
    import monarch_attention_b200 as ma
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(3)
    q, k, v = (torch.randn(1, 2, 40, 16, generator=g).to(dev) for _ in range(3))
    v.requires_grad_(True)
    out = ma.MonarchAttention(8, 2, "post")(q, k, v)
    out.sum().backward()
    assert q.grad is None and k.grad is None and v.grad is not None
    with pytest.raises(ValueError, match="out="):
        ma.monarch_attention_b200(q, k, v, None, 2, 8, False, out=torch.empty_like(v))
