"""A bounded wait that ran out is reported by the module whose function launched the kernel."""
import types

import pytest


def test_layer_norm_reports_its_own_waits(monkeypatch):
    from torchmpi_b200._lib import TorchMPIError
    from torchmpi_b200.ops import gemm, layernorm
    fake = types.SimpleNamespace(tmpi_layernorm_status=lambda: 4001, tmpi_gemm_status=lambda: 0, tmpi_conv_status=lambda: 0)
    monkeypatch.setattr(layernorm, "lib", fake)
    monkeypatch.setattr(gemm, "lib", fake)
    with pytest.raises(TorchMPIError, match="layer norm.*4001"):
        layernorm.check_status()
    gemm.check_status()


def test_linear_reports_waits_of_its_split_weight_gradient(monkeypatch):
    from torchmpi_b200._lib import TorchMPIError
    from torchmpi_b200.ops import gemm
    monkeypatch.setattr(gemm, "lib", types.SimpleNamespace(tmpi_gemm_status=lambda: 0, tmpi_conv_status=lambda: 2006))
    with pytest.raises(TorchMPIError, match="2006"):
        gemm.check_status()


def test_attention_reports_its_waits(monkeypatch):
    from torchmpi_b200._lib import TorchMPIError
    from torchmpi_b200.ops import attention
    monkeypatch.setattr(attention, "lib", types.SimpleNamespace(tmpi_attention_status=lambda: 3011))
    with pytest.raises(TorchMPIError, match="3011"):
        attention.check_status()


def _function(file, name):
    """Source of a device function of the kernels, and of the macros of its file."""
    import pathlib
    import re

    import torchmpi_b200
    src = (pathlib.Path(torchmpi_b200.__file__).parent / "csrc" / "kernels" / file).read_text()
    start = src.index(f"__device__ void {name}(")
    macros = dict(re.findall(r"#define (\w+)\([^)]*\) \\\n(.*)", src))
    return src[start:src.index("\n}\n", start)], macros


@pytest.mark.parametrize("file,name", [("attention.cu", "softmax_rows"), ("attention_bwd.cu", "softmax_rows"), ("attention_bwd.cu", "drain")])
def test_lanes_of_an_attention_warp_leave_together(file, name):
    """A wait may run out for some lanes of a warp and succeed for others; whoever left alone would be missing at the warp's next barrier,
    which knows no budget.  (Read from the source: a wait that runs out in one lane only cannot be brought about.)"""
    body, macros = _function(file, name)
    leaving = 0
    for line in body.splitlines():
        used = [m for m in macros if m + "(" in line]
        for text in [line] + [macros[m] for m in used]:
            if "return;" in text:
                assert any(vote in text for vote in ("__all_sync(~0u", "__any_sync(~0u", "mbar_wait_warp(")), text
                leaving += 1
        assert "mbar_wait(" not in line
    assert leaving
