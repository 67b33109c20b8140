"""Which split-K workspace a decode launch is given: the one of the stream it runs on, whatever stream the plan was built
on, and the caller's own where one is handed in.  The launch itself is a stand-in that records its arguments, so no GPU
is needed."""

import ctypes as C

import pytest
import torch

from hyquant_b200 import _lib
from hyquant_b200 import decode_d_stage as dd
from hyquant_b200.d_stage_kv_cache import DStageLayerCache

B, H_KV, R = 1, 2, 4


class Machine:
    """The current stream, whether it is capturing, one workspace per stream, and the launches that were made."""

    def __init__(self, monkeypatch):
        self.stream, self.capturing, self.spaces, self.launches = 11, False, {}, []
        monkeypatch.setattr(_lib, "stream_ptr", lambda device=None: self.stream)
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: self.capturing)
        monkeypatch.setattr(dd, "decode_workspace", lambda device, heads, repeat: self.space(self.stream))

    def space(self, stream):
        return self.spaces.setdefault(stream, torch.zeros(256, dtype=torch.uint8))

    def launch(self, args, stream):
        self.launches.append((stream, args._obj.workspace, args._obj.flags))
        return 0


@pytest.fixture
def machine(monkeypatch):
    return Machine(monkeypatch)


def layer_on(machine):
    plan = dd.DecodePlan.__new__(dd.DecodePlan)
    plan.device, plan.BH_KV, plan.kv_repeat = torch.device("cpu"), B * H_KV, R
    plan.args = _lib.DecodeArgs()
    plan._args_ref, plan._fn = C.byref(plan.args), machine.launch
    plan.stream, plan.ws = machine.stream, machine.space(machine.stream)
    plan.args.workspace, plan.args.workspace_bytes = plan.ws.data_ptr(), plan.ws.numel()
    layer = DStageLayerCache(0)
    layer._plan, layer._B, layer._H_KV, layer._D, layer.phase = plan, B, H_KV, 128, "decode"
    layer._staging_buf_k = torch.zeros(B * H_KV, 128, 128, dtype=torch.bfloat16)
    return layer


def query(contiguous):
    q = torch.zeros(B, 1, H_KV * R, 128, dtype=torch.bfloat16).transpose(1, 2)
    return q.contiguous() if contiguous else torch.zeros(B, H_KV * R, 1, 256, dtype=torch.bfloat16)[..., ::2]


@pytest.mark.parametrize("contiguous", [True, False])       # the direct route, and the general one
def test_a_launch_takes_the_workspace_of_its_stream(machine, contiguous):
    layers = [layer_on(machine), layer_on(machine)]
    for stream, layer in ((11, 0), (22, 0), (11, 1), (22, 1), (22, 0), (11, 0)):
        machine.stream = stream
        layers[layer].decode_attention(query(contiguous), R)
        assert machine.launches[-1][:2] == (stream, machine.space(stream).data_ptr())
        assert layers[layer]._plan.ws is machine.space(stream)      # what decode_status reads
    assert machine.space(11).data_ptr() != machine.space(22).data_ptr()


def test_nothing_is_allocated_for_a_launch_under_capture(machine):
    layer = layer_on(machine)
    machine.stream, machine.capturing = 33, True
    layer.decode_attention(query(True), R)
    assert machine.launches[-1][1] == machine.space(11).data_ptr() and 33 not in machine.spaces


def test_a_workspace_of_the_callers_serves_one_launch(machine):
    layer = layer_on(machine)
    layer._lengths = torch.zeros(2, dtype=torch.int32)
    own, k = torch.zeros(256, dtype=torch.uint8), torch.zeros(B, H_KV, 1, 128, dtype=torch.bfloat16)
    machine.stream = 22
    layer.capture_decode_step(query(True), k, k, R, torch.empty(B, H_KV * R, 1, 128, dtype=torch.bfloat16), overlap=False,
                              num_splits=4, workspace=own)
    assert machine.launches[-1] == (22, own.data_ptr(), _lib.HQ_DECODE_SHARED_CHIP)
    machine.stream = 11
    layer.decode_attention(query(True), R)
    assert machine.launches[-1] == (11, machine.space(11).data_ptr(), 0)
    assert layer._plan.args.num_splits == 0
