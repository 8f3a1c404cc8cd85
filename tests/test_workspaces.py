"""Which workspace a call gets that does not bring its own: never one that another call may be using at the same time.  The
library and the streams are stand-ins, so this runs without a GPU."""
import types

import pytest

import fp8_quant_matmul_b200 as f
from fp8_quant_matmul_b200 import api

torch = pytest.importorskip("torch")


class Operand:
    """As much of a CUDA tensor as gemm looks at; its device is the CPU, where the workspaces of this test are."""
    is_cuda = True
    device = torch.device("cpu")

    def get_device(self):
        return 0

    def data_ptr(self):
        return 4096


class Library:
    """Records the workspace of every call."""

    def __init__(self):
        self.calls, self.zeroed, self.capture, self.held, self.gone = [], [], 0, [], []

    def fp8bs_workspace_bytes(self, M, N, K):
        return M << 10

    def fp8bs_workspace_init(self, ptr, nbytes, stream):
        self.zeroed.append((ptr, stream))
        return 0

    def fp8bs_gemm_ex(self, *args):
        self.calls.append((args[13], args[15]))           # workspace, stream
        assert args[14] >= args[5] << 10
        return 0

    def fp8bs_capture_id(self, stream, out):
        out._obj.value = self.capture
        return 0

    def fp8bs_capture_hold(self, stream, token):
        self.held.append(token)
        return 0

    def fp8bs_capture_released(self, out, n):
        tokens, self.gone = self.gone[:n], self.gone[n:]
        for i, t in enumerate(tokens):
            out[i] = t
        return len(tokens)


@pytest.fixture
def box(monkeypatch):
    lib, now = Library(), types.SimpleNamespace(stream=11)
    monkeypatch.setattr(api, "lib", lambda: lib)
    monkeypatch.setattr(api, "_stream", lambda index: now.stream)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: types.SimpleNamespace(cuda_stream=now.stream))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: lib.capture != 0)
    for name in ("_workspaces", "_graph_workspaces", "_needs"):
        monkeypatch.setattr(api, name, {}, raising=False)
    monkeypatch.setattr(api, "_set_up", set())
    return lib, now


def call(box, stream, capture=0, M=1024):
    lib, now = box
    now.stream, lib.capture = stream, capture
    x = Operand()
    f.gemm(x, x, x, x, C=x, M=M, N=512, K=7168)
    assert lib.calls[-1][1] == stream
    return lib.calls[-1][0]


def test_every_stream_has_a_workspace_of_its_own(box):
    a, b = call(box, 11), call(box, 12)
    assert a != b
    assert box[0].zeroed == [(a, 11), (b, 12)]            # zeroed on the stream that uses it
    assert call(box, 11) == a and call(box, 12) == b


def test_a_grown_workspace_is_zeroed_on_its_stream_and_touches_no_other(box):
    a, b = call(box, 11), call(box, 12)
    c = call(box, 11, M=4096)
    assert box[0].zeroed[-1] == (c, 11) and c != b
    assert call(box, 11) == c and call(box, 12) == b


def test_a_captured_graph_shares_its_workspace_with_nobody(box):
    a = call(box, 11)
    g1 = call(box, 11, capture=7)
    assert g1 != a and call(box, 11, capture=7) == g1     # one per capture and stream
    g1_other = call(box, 12, capture=7)
    g2 = call(box, 11, capture=8)
    assert len({a, g1, g1_other, g2}) == 4
    assert [s for _, s in box[0].zeroed] == [11, 11, 12, 11]
    assert call(box, 11) == a                             # the eager one is as it was


def test_workspaces_are_given_back(box):
    for stream in range(100, 100 + 3 * api.MAX_WORKSPACES):
        call(box, stream)
    assert len(api._workspaces) == api.MAX_WORKSPACES
    call(box, 11, capture=7)
    call(box, 11, capture=8)
    first, second = box[0].held
    assert set(api._graph_workspaces) == {first, second}
    box[0].gone = [first]
    call(box, 11, capture=9)
    assert set(api._graph_workspaces) == {second, box[0].held[2]}


def test_another_build_is_asked_again(monkeypatch):
    monkeypatch.setattr(api, "_needs", {})
    monkeypatch.setattr(api, "_set_up", {0})
    monkeypatch.setattr(api, "_lib", None)
    key = (0, 1024, 512, 7168, f.PATH_MN_SMALL, 3, 128 | f.SPLIT_WORKSPACE)
    need = api._workspace_need(key)
    api._set_up.add(0)
    assert need > 0 and api._workspace_need(key) == need and api._needs == {key: need}
    api.load(api._LIB_PATH)
    assert not api._needs and not api._set_up
