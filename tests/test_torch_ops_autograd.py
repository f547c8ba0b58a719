"""Backward through the torch operators, on the CPU: kernels that stand in for the CUDA ones are
registered for the duration of a test (they return zeros of the result's shape and type)."""

import warnings

import pytest
import torch

import mosaicist_b200.torch_ops  # noqa: F401  (registers torch.ops.mosaicist_sm100a.*)

NS = "mosaicist_sm100a"
BF16, F32, U8, I32 = torch.bfloat16, torch.float32, torch.uint8, torch.int32


def _z(*shape, dtype=F32):
    return torch.zeros(shape, dtype=dtype)


#: operator -> (arguments, results); the floating-point arguments are the ones that can ask for gradients
CASES = {
    "grouped_gemm_nvfp4": ((_z(2, 128, 32, dtype=U8), _z(2, 1, 1, 32, 16, dtype=U8), _z(2, 128, 32, dtype=U8),
                            _z(2, 1, 1, 32, 16, dtype=U8), _z(2), None), (_z(2, 128, 128, dtype=BF16),)),
    "grouped_gemm_nvfp4_ragged": ((_z(128, 32, dtype=U8), _z(1, 1, 32, 16, dtype=U8), _z(1, 128, 32, dtype=U8),
                                   _z(1, 1, 1, 32, 16, dtype=U8), _z(1, dtype=I32), _z(1, dtype=I32), _z(1), None),
                                  (_z(128, 128, dtype=BF16),)),
    "quantize_nvfp4": ((_z(1, 128, 64), _z(1), None), (_z(1, 128, 32, dtype=U8), _z(1, 1, 1, 32, 16, dtype=U8))),
    "silu_mul_quantize_nvfp4": ((_z(1, 128, 128, dtype=BF16), _z(1), None),
                                (_z(1, 128, 32, dtype=U8), _z(1, 1, 1, 32, 16, dtype=U8))),
    "global_scale_for": ((_z(2, 8),), (_z(2),)),
    "quantize_mxfp8": ((_z(128, 128),), (_z(128, 128, dtype=U8), _z(1, 1, 32, 16, dtype=U8))),
    "grouped_gemm_mxfp8_ragged": ((_z(128, 128, dtype=U8), _z(1, 1, 32, 16, dtype=U8), _z(1, 128, 128, dtype=U8),
                                   _z(1, 1, 1, 32, 16, dtype=U8), _z(1, dtype=I32), _z(1, dtype=I32), None, _z(128)),
                                  (_z(128, 128, dtype=BF16),)),
    "gemm_f16": ((_z(8, 8, dtype=BF16), _z(8, 8, dtype=BF16)), (_z(8, 8, dtype=BF16),)),
    "grouped_gemm_bf16_int4_ragged": ((_z(128, 64, dtype=BF16), _z(1, 256, 32, dtype=U8), _z(1, 256, 1, dtype=BF16),
                                       _z(1, dtype=I32), _z(1, dtype=I32), None, 64), (_z(128, 256, dtype=BF16),)),
    "moe_masked": ((_z(1, 128, 128, dtype=BF16), _z(1, 256, 64, dtype=U8), _z(1, 2, 2, 32, 16, dtype=U8), _z(1), _z(1),
                    _z(1, 128, 64, dtype=U8), _z(1, 1, 2, 32, 16, dtype=U8), _z(1), _z(1), _z(1, dtype=I32), _z(1), _z(1)),
                   (_z(1, 128, 128, dtype=BF16),)),
}


@pytest.fixture()
def on_cpu():
    lib = torch.library.Library(NS, "IMPL")
    for name, (_, results) in CASES.items():
        def kernel(*args, _results=results):
            fresh = tuple(torch.zeros_like(r) for r in _results)
            return fresh if len(fresh) > 1 else fresh[0]
        lib.impl(name, kernel, "CPU")
    yield
    lib._destroy()


@pytest.mark.parametrize("name", sorted(CASES))
def test_backward_raises_instead_of_leaving_the_gradient_out(on_cpu, name):
    args, results = CASES[name]
    op = getattr(torch.ops.mosaicist_sm100a, name)
    plain = op(*args)
    assert not any(r.requires_grad for r in (plain if isinstance(plain, tuple) else (plain,)))
    leaves = [a.clone().requires_grad_() if isinstance(a, torch.Tensor) and a.is_floating_point() else a for a in args]
    assert any(getattr(a, "requires_grad", False) for a in leaves)
    out = op(*leaves)
    out = out if isinstance(out, tuple) else (out,)
    for got, want in zip(out, results):
        assert got.shape == want.shape and got.dtype == want.dtype
        if not want.is_floating_point():          # bytes carry no gradient
            assert not got.requires_grad
            continue
        assert got.requires_grad
        other = next(a for a in leaves if getattr(a, "requires_grad", False))
        with pytest.raises(RuntimeError, match="not implemented|no autograd formula"):
            (got.float().sum() + other.float().sum()).backward()


def test_a_formula_can_still_be_registered(on_cpu):
    """torch.library.register_autograd gives an operator a derivative, as for any custom operator."""
    lib = torch.library.Library(NS, "FRAGMENT")
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")           # torch notes that an autograd kernel is replaced
        torch.library.register_autograd(f"{NS}::global_scale_for", lambda ctx, g: torch.full((2, 8), 3.0), lib=lib)
    try:
        x = torch.zeros(2, 8, requires_grad=True)
        torch.ops.mosaicist_sm100a.global_scale_for(x).sum().backward()
        assert torch.equal(x.grad, torch.full((2, 8), 3.0))
    finally:
        lib._destroy()
    with pytest.raises(RuntimeError):
        torch.ops.mosaicist_sm100a.global_scale_for(x).sum().backward()
