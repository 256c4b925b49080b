"""The bindings import and find the current stream whatever private names torch has (no GPU needed)."""
import importlib
import types

import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("missing", ["_cuda_getCurrentRawStream", "_cuda_getDevice"])
def test_public_call_where_a_private_name_is_missing(lkb, monkeypatch, missing):
    api = importlib.import_module("lfm2-ampere_b200.api")
    monkeypatch.delattr(torch._C, missing, raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=0xBEEF))
    try:
        importlib.reload(api)
        assert api.stream() == 0xBEEF
    finally:
        monkeypatch.undo()
        importlib.reload(api)


@pytest.mark.gpu
def test_handle_is_the_current_streams(lkb):
    api = importlib.import_module("lfm2-ampere_b200.api")
    assert api.stream() == torch.cuda.current_stream().cuda_stream
    with torch.cuda.stream(torch.cuda.Stream()):
        assert api.stream() == torch.cuda.current_stream().cuda_stream != 0
