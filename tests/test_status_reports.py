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
