"""QLinear's input shapes, with the launches replaced (no GPU): what is accepted, what is refused."""
import types

import pytest
import torch

from nvfp4_v100_b200.pipeline import _qwen38_infer as Q

K, M = 64, 32


@pytest.fixture
def layer(monkeypatch):
    done = lambda *a: 0
    monkeypatch.setattr(Q, "GEMV_T1", done)
    monkeypatch.setattr(Q, "GEMV", types.SimpleNamespace(launch_nvfp4_gemv2=done))
    monkeypatch.setattr(Q, "V5", types.SimpleNamespace(launch_nvfp4_gemm_w4a16_ex=done))
    monkeypatch.setattr(Q, "_stream_handle", lambda: 0)
    return Q.QLinear(0, 0, M, K)


@pytest.mark.parametrize("shape", [(K,), (1, K), (2, K), (5, K), (1, 1, K), (2, 3, K), (3, 1, 2, K)])
def test_output_shape(layer, shape):
    assert layer(torch.zeros(shape, dtype=torch.float16)).shape == (*shape[:-1], M)
    assert layer(torch.zeros(shape)).shape == (*shape[:-1], M)
    strided = torch.zeros((*shape[:-1], 2 * K), dtype=torch.float16)[..., ::2]
    assert layer(strided).shape == (*shape[:-1], M)


@pytest.mark.parametrize("lead", [(2,), (3,), (4,), (2, 2), (1, 3, 2)])
@pytest.mark.parametrize("width", [2 * K, K // 2, 3 * K, K + 1])
def test_wrong_feature_width_is_refused(layer, lead, width):
    with pytest.raises(RuntimeError):
        layer(torch.zeros((*lead, width), dtype=torch.float16))


@pytest.mark.parametrize("shape", [(0, K), (2, 0, K)])
def test_no_tokens_is_refused(layer, shape):
    with pytest.raises(IndexError):
        layer(torch.zeros(shape, dtype=torch.float16))
