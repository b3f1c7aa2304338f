"""Host-side logic that needs no GPU: the module-name shim, argument / device checks that must raise before any
kernel is launched, and the checkpoint-side weight packer (checked against the oracle's quantiser and layout)."""
import importlib
import sys

import numpy as np
import pytest
import torch

from oracle import nvfp4_oracle as O


def test_shim_registers_and_removes_the_reference_module_names(b200):
    shim = b200.compat_shim
    names = ["flashinfer.cute_dsl.rmsnorm_fp4quant", "flashinfer.cute_dsl.add_rmsnorm_fp4quant",
             "flashinfer.fused_moe.cute_dsl.b12x_moe", "dense_blockscaled_gemm_persistent_cooperative"]
    before = {n: sys.modules.get(n) for n in names + ["flashinfer"]}
    assert not shim.installed()                       # nothing is shadowed without an explicit install()
    shim.install()
    try:
        assert shim.installed()
        # the reference's loader calls (tests/python/support/flashinfer_verbatim.py:101-108,111-162)
        assert shim.load_operator("rmsnorm_fp4quant").rmsnorm_fp4quant is b200.rmsnorm_fp4quant
        assert shim.load_operator("add_rmsnorm_fp4quant").add_rmsnorm_fp4quant is b200.add_rmsnorm_fp4quant
        assert shim.load_b12x_operator().b12x_fused_moe is b200.b12x_fused_moe
        assert shim.ensure_loaded() is sys.modules["flashinfer.cute_dsl"]
        # plain imports by module path resolve too
        m = importlib.import_module("flashinfer.cute_dsl.rmsnorm_fp4quant")
        assert m.rmsnorm_fp4quant is b200.rmsnorm_fp4quant
        from flashinfer.fused_moe.cute_dsl.b12x_moe import B12xMoEWrapper, b12x_fused_moe
        assert b12x_fused_moe is b200.b12x_fused_moe and B12xMoEWrapper is b200.B12xMoEWrapper
        bs = importlib.import_module("dense_blockscaled_gemm_persistent_cooperative")
        assert bs.run is b200.gemm.run and bs.Sm120BlockScaledGemmKernel is b200.Sm120BlockScaledGemmKernel
        with pytest.raises(ImportError):
            shim.load_operator("layernorm")
        shim.install()                                # idempotent
    finally:
        shim.uninstall()
    assert not shim.installed()
    for n, old in before.items():
        assert sys.modules.get(n) is old


def _cpu_moe_args(experts=2, hidden=256, inter=128, tokens=4, top_k=1):
    w1 = torch.zeros(experts, 2 * inter, hidden // 2, dtype=torch.uint8)
    w2 = torch.zeros(experts, hidden, inter // 2, dtype=torch.uint8)
    s1 = torch.zeros(experts, (2 * inter // 128) * (hidden // 64) * 512, dtype=torch.uint8)
    s2 = torch.zeros(experts, (hidden // 128) * (inter // 64) * 512, dtype=torch.uint8)
    x = torch.zeros(tokens, hidden, dtype=torch.bfloat16)
    ids = torch.zeros(tokens, top_k, dtype=torch.int32)
    w = torch.ones(tokens, top_k)
    return x, w1, s1, w2, s2, ids, w


def test_operators_refuse_cpu_tensors_before_any_launch(b200):
    """No CPU fallback and no pointer of a CPU tensor ever reaches a kernel."""
    x, w1, s1, w2, s2, ids, w = _cpu_moe_args()
    with pytest.raises(ValueError):
        b200.b12x_fused_moe(x, w1, s1, w2, s2, ids, w, 2, 1)
    with pytest.raises(ValueError):
        b200.rmsnorm_fp4quant(torch.zeros(4, 128, dtype=torch.bfloat16), torch.ones(128, dtype=torch.bfloat16))
    with pytest.raises(ValueError):
        b200.nvfp4_gemm(torch.zeros(128, 64, dtype=torch.uint8), torch.zeros(128, 64, dtype=torch.uint8),
                        torch.zeros(512, dtype=torch.uint8), torch.zeros(512, dtype=torch.uint8))
    with pytest.raises(ValueError):
        b200.topk_route(torch.zeros(4, 8), 2)


def test_moe_device_check_names_the_offending_argument(b200):
    from cutedsl_fully_opensourced_b200.moe import _on_device
    dev = torch.device("cuda", 0)
    with pytest.raises(ValueError, match="token_selected_experts"):
        _on_device(dev, token_selected_experts=torch.zeros(2, 2, dtype=torch.int32))
    with pytest.raises(ValueError, match="w1_alpha"):
        _on_device(dev, x=None, w1_alpha=torch.ones(2))
    _on_device(dev, fc2_input_scale=None)            # optional tensors may be absent


def _fake(*shape, dtype=torch.uint8, gpu=0):
    """A tensor that says it lives on a GPU and has no memory: what the checks before a launch look at."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        return torch.empty(*shape, dtype=dtype, device=f"cuda:{gpu}")


def _gemm_args(**changed):
    args = {"a": _fake(128, 128), "b": _fake(256, 128), "sfa": _fake(2048), "sfb": _fake(4096),
            "out": _fake(128, 256, dtype=torch.bfloat16), "alpha": _fake(1, dtype=torch.float32)}
    args.update(changed)
    return args


@pytest.mark.parametrize("name", ["b", "sfa", "sfb", "out", "alpha"])
def test_gemm_refuses_a_tensor_of_another_gpu(b200, name):
    good = _gemm_args()
    other = _fake(*good[name].shape, dtype=good[name].dtype, gpu=1)
    with pytest.raises(ValueError, match="must be a CUDA tensor on cuda:0"):
        b200.nvfp4_gemm(**_gemm_args(**{name: other}))
    with pytest.raises(ValueError, match="must be a CUDA tensor on cuda:0"):
        b200.nvfp4_gemm(**_gemm_args(**{name: other}), sf_vec_size=32)
    fp8 = {n: t.view(torch.float8_e4m3fn) for n, t in (("a", good["a"]), ("b", good["b"]))}
    if name == "b":
        other = other.view(torch.float8_e4m3fn)
    with pytest.raises(ValueError, match="must be a CUDA tensor on cuda:0"):
        b200.mxfp8_gemm(**_gemm_args(**{**fp8, name: other}))
    with pytest.raises(RuntimeError):                  # the same call with every tensor on its GPU gets past the checks
        b200.nvfp4_gemm(**good)


def test_gemm_refuses_scale_factors_with_gaps(b200):
    for name, n in (("sfa", 2048), ("sfb", 4096)):
        with pytest.raises(ValueError, match="one run of memory"):
            b200.nvfp4_gemm(**_gemm_args(**{name: _fake(2 * n)[::2]}))
        with pytest.raises(ValueError, match="one run of memory"):
            b200.nvfp4_gemm(**_gemm_args(**{name: _fake(n // 16, 32)[:, :16]}))
        for view in (_fake(n // 512, 32, 4, 4).permute(1, 2, 3, 0), _fake(16, n // 16).t(), _fake(1, 2 * n)[:, :n]):
            with pytest.raises(RuntimeError):          # one run, whatever the order of its dimensions
                b200.nvfp4_gemm(**_gemm_args(**{name: view}))


def _norm_args(**changed):
    bf16 = torch.bfloat16
    args = {"input": _fake(8, 256, dtype=bf16), "residual": _fake(8, 256, dtype=bf16), "weight": _fake(256, dtype=bf16),
            "y_fp4": _fake(8, 128), "block_scale": _fake(128, 16), "block_scale_unswizzled": _fake(8, 16),
            "global_scale": _fake(1, dtype=torch.float32), "output_both_sf_layouts": True}
    args.update(changed)
    return args


@pytest.mark.parametrize("view", [lambda: _fake(8, 32)[:, :16], lambda: _fake(16, 8).t(), lambda: _fake(256)[::2]])
def test_norm_refuses_row_major_scales_that_are_no_run_of_rows(b200, view):
    with pytest.raises(ValueError, match="block_scale_unswizzled must be a contiguous"):
        b200.add_rmsnorm_fp4quant(**_norm_args(block_scale_unswizzled=view()))
    with pytest.raises(RuntimeError):                  # a contiguous one, also at an odd offset, gets past the checks
        b200.add_rmsnorm_fp4quant(**_norm_args(block_scale_unswizzled=_fake(200)[1:129].view(8, 16)))


def _moe_args(**changed):
    """hidden 256, intermediate 128, 2 experts, 4 tokens, top-1"""
    f32 = torch.float32
    args = {"x": _fake(4, 256, dtype=torch.bfloat16), "w1_weight": _fake(2, 256, 128), "w1_weight_sf": _fake(2, 2 * 4 * 512),
            "w2_weight": _fake(2, 256, 64), "w2_weight_sf": _fake(2, 2 * 2 * 512),
            "token_selected_experts": _fake(4, 1, dtype=torch.int32), "token_final_scales": _fake(4, 1, dtype=f32),
            "num_experts": 2, "top_k": 1, "w1_alpha": _fake(2, dtype=f32), "w2_alpha": _fake(2, dtype=f32),
            "fc2_input_scale": _fake(1, dtype=f32), "router_logits": _fake(4, 2, dtype=f32),
            "output": _fake(4, 256, dtype=torch.bfloat16), "workspace": _fake(1 << 22)}
    args.update(changed)
    return args


@pytest.mark.parametrize("name", ["w1_weight", "w1_weight_sf", "w2_weight", "w2_weight_sf", "token_selected_experts",
                                  "token_final_scales", "w1_alpha", "w2_alpha", "fc2_input_scale", "router_logits", "output",
                                  "workspace"])
def test_moe_operator_refuses_a_tensor_of_another_gpu_or_the_cpu(b200, name):
    """The single-GPU operator checks for itself (the test above covers what the expert-parallel classes call)."""
    good = _moe_args()
    for other in (_fake(*good[name].shape, dtype=good[name].dtype, gpu=1), torch.zeros(good[name].shape, dtype=good[name].dtype)):
        with pytest.raises(ValueError, match=f"{name} must be a CUDA tensor on cuda:0"):
            b200.b12x_fused_moe(**_moe_args(**{name: other}))
    with pytest.raises(RuntimeError):                  # with every tensor on its GPU the call gets past the checks
        b200.b12x_fused_moe(**good)


def test_argument_forms_that_python_takes_for_the_same(b200):
    """16.0 is 16, a result type is not looked at beside the result's tensor, and None is torch's default type."""
    past_the_checks = pytest.raises(RuntimeError)
    for call in (lambda: b200.add_rmsnorm_fp4quant(**_norm_args(block_size=16.0)),
                 lambda: b200.nvfp4_gemm(**_gemm_args(), sf_vec_size=16.0),
                 lambda: b200.nvfp4_gemm(**_gemm_args(), sf_vec_size=32.0),
                 lambda: b200.nvfp4_gemm(**_gemm_args(), out_dtype=None),
                 lambda: b200.nvfp4_gemm(**_gemm_args(out=None), out_dtype=None),
                 lambda: b200.b12x_fused_moe(**_moe_args(local_expert_offset=0.0))):
        with past_the_checks:
            call()
    with pytest.raises(NotImplementedError):
        b200.add_rmsnorm_fp4quant(**_norm_args(block_size=16.5))
    with pytest.raises(NotImplementedError):
        b200.nvfp4_gemm(**_gemm_args(), sf_vec_size=16.5)
    with pytest.raises(TypeError):
        b200.nvfp4_gemm(**_gemm_args(out=None), out_dtype="bf16")
    z = _fake(128, 128)
    with pytest.raises(NotImplementedError):
        b200.mm_fp4(z, z.t(), _fake(2048), _fake(2048), out_dtype=None)
    x, w1, s1, w2, s2, ids, w = _cpu_moe_args()
    with pytest.raises(NotImplementedError):
        b200.b12x_fused_moe(x, w1, s1, w2, s2, ids, w, 2, 1, output_dtype=None)


def test_pack_moe_weights_matches_the_oracle_quantiser_and_layout(b200):
    torch.manual_seed(0)
    e, inter, hidden = 3, 128, 256
    w1 = 0.02 * torch.randn(e, 2 * inter, hidden)
    w2 = 0.02 * torch.randn(e, hidden, inter)
    packed = b200.pack_moe_weights(w1, w2, fc2_input_scale=2.0)
    for name, w, extra in (("w1", w1, 1.0), ("w2", w2, 2.0)):
        for i in range(e):
            gs = float(448.0 * 6.0 / w[i].abs().max())
            codes, sf = O.quantize_nvfp4(w[i].numpy(), gs)
            assert np.array_equal(packed[f"{name}_weight"][i].numpy(), O.pack_e2m1(codes))
            storage = b200.layout.six_mode_to_storage(packed[f"{name}_weight_sf"])[i].numpy()
            assert np.array_equal(storage, O.swizzle_sf(sf))
            assert abs(float(packed[f"{name}_alpha"][i]) * gs * extra - 1.0) < 1e-6
    assert tuple(packed["w1_weight_sf"].shape) == (32, 4, 2, 4, 4, e)
    with pytest.raises(ValueError):
        b200.pack_moe_weights(w1, w2[:2])


def test_mm_fp4_refuses_other_block_formats(b200):
    z = torch.zeros(1, dtype=torch.uint8)
    with pytest.raises(NotImplementedError):
        b200.mm_fp4(z, z, z, z, block_size=32)
    with pytest.raises(NotImplementedError):
        b200.mm_fp4(z, z, z, z, use_8x4_sf_layout=True)
