"""One mixture-of-experts layer called by several threads on one stream: the gather (or quantiser) and the
grouped GEMM that reads its scratch stay together in the stream.  The order of the launches is checked on the
CPU with a library that records them, the results on the GPU."""

import threading
import time

import pytest
import torch

from flydsl_b200 import _lib, pertoken_quant
from flydsl_b200.expert_parallel import ExpertParallelMoe
from flydsl_b200.kernels.moe.moe_gemm_2stage import compile_moe_gemm1, compile_moe_gemm2


class Recorder:
    """Stands for the library and the host extension: notes a chain that enters while another one still
    holds the same scratch."""

    def __init__(self):
        self.holders, self.overlaps, self.guard = {}, 0, threading.Lock()

    def enter(self, *scratch):
        with self.guard:
            for s in scratch:
                self.overlaps += self.holders.get(s, 0)
                self.holders[s] = self.holders.get(s, 0) + 1
        time.sleep(0.01)

    def leave(self, *scratch):
        with self.guard:
            for s in scratch:
                self.holders[s] -= 1

    def chain(self, *scratch):
        self.enter(*scratch)
        self.leave(*scratch)
        return 0

    def moe_stage(self, *a):
        return self.chain(a[9].data_ptr())

    def moe_layer(self, *a):
        self.chain(a[9].data_ptr(), a[11].data_ptr())
        return a[0]

    def flyb200_moe_quant_sorted(self, *a):
        self.enter(a[0])
        return 0

    def flyb200_moe_gemm(self, *a):
        self.leave(a[2])
        return 0


@pytest.fixture
def recorder(monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(_lib, "ops", lambda: rec)
    monkeypatch.setattr(_lib, "load", lambda: rec)
    monkeypatch.setattr(_lib, "current_stream", lambda dev: 0)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: None)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return rec


def run(work, n=4):
    errors = []

    def guarded(i):
        try:
            work(i)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


KW = dict(model_dim=256, inter_dim=128, experts=4, topk=2, tile_m=16, tile_n=128, tile_k=128, in_dtype="fp8")


@pytest.mark.parametrize("stage", [1, 2])
def test_stage_launches_stay_together(recorder, stage):
    fn = compile_moe_gemm1(**KW, doweight_stage1=False) if stage == 1 else compile_moe_gemm2(**KW, doweight_stage2=False)
    t = torch.zeros(16)
    for blocks in (2, 3):  # the second size replaces the buffer
        run(lambda i, b=blocks: fn._launch(t, t, t, t, t, t, t, t, t, 8, b, None))
    run(lambda i: fn._launch(t, t, t, t, t, t, t, t, t, 8, 1 + i, None))
    assert recorder.overlaps == 0 and len(fn._scratch) == 1


def test_quantising_launches_stay_together(recorder):
    fn, t = compile_moe_gemm2(**KW, doweight_stage2=False), torch.zeros(16)
    run(lambda i: fn._launch_quantising(t, t, t, t, t, t, t, t, 8, 2, None))
    assert recorder.overlaps == 0


def test_layer_launches_stay_together(recorder):
    layer = ExpertParallelMoe(model_dim=256, inter_dim=128, experts=4, topk=2, tile_m=16, rank=0, world=1)
    x = torch.zeros(8, 256)
    run(lambda i: layer._forward_native(x, x, x, x, 8, x.device))
    assert recorder.overlaps == 0


def test_a_copy_of_a_launcher_has_scratch_of_its_own(recorder):
    import copy
    import pickle

    fn, t = compile_moe_gemm2(**KW, doweight_stage2=False), torch.zeros(16)
    fn._launch(t, t, t, t, t, t, t, t, t, 8, 2, None)
    for other in (copy.deepcopy(fn), pickle.loads(pickle.dumps(fn))):
        assert other._scratch == {} and other.model_dim == fn.model_dim
        other._launch(t, t, t, t, t, t, t, t, t, 8, 2, None)
        assert other._scratch[(None, 0)][0].data_ptr() != fn._scratch[(None, 0)][0].data_ptr()


@pytest.mark.gpu
@pytest.mark.parametrize("out_dtype", ["bf16", "f32"])
def test_threads_on_one_stream(out_dtype):
    d, inter, experts, topk, tokens = 1024, 512, 8, 2, 48
    layer = ExpertParallelMoe(model_dim=d, inter_dim=inter, experts=experts, topk=topk, tile_m=16, out_dtype=out_dtype, rank=0, world=1)
    g = torch.Generator(device="cuda").manual_seed(5)
    qd = torch.float8_e4m3fn
    w1, s1 = pertoken_quant(torch.randn(experts, 2 * inter, d, generator=g, device="cuda"), quant_dtype=qd)
    w2, s2 = pertoken_quant(torch.randn(experts, d, inter, generator=g, device="cuda"), quant_dtype=qd)
    layer.load_expert_weights(w1, s1, w2, s2)
    calls, want = [], []
    for _ in range(4):
        x, sx = pertoken_quant(torch.randn(tokens, d, generator=g, device="cuda"), quant_dtype=qd)
        v, ids = torch.topk(torch.rand(tokens, experts, generator=g, device="cuda"), k=topk, dim=1)
        calls.append((x, sx, ids, torch.softmax(v, dim=1)))
        want.append(layer.forward_local(*calls[-1]))
    torch.cuda.synchronize()
    got = [[] for _ in calls]
    run(lambda i: got[i].extend(layer.forward_local(*calls[i]) for _ in range(50)))
    torch.cuda.synchronize()
    for i, ys in enumerate(got):
        for y in ys:  # two routes a token, added to zero: the same sum in either order
            assert torch.equal(y, want[i])
