"""Strips cut between CTAs: the counts that say who comes last lie in the caller's scratch (csrc/arrivals.cuh).  Whatever the scratch held, in
graphs replayed side by side and in streams hundreds of launches apart, the bits are those of a launch by itself.  Shapes: few strips
with many contributors, contributors that share two strips, ragged strips."""
import ctypes as C

import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def e():
    import custom_esimd_kernels_vllm as pkg
    yield pkg
    pkg.set_force_kernel(0)
    pkg.set_overlap_mode(1)


class Linear:
    """A cut linear through the C ABI, on scratch and output of its own."""

    def __init__(self, e, kind, M, N, K, seed):
        g = torch.Generator(device=DEV).manual_seed(seed)
        self.L, self.kind, self.M, self.N, self.K = e._lib, kind, M, N, K
        self.x = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
        if kind == "int4":
            self.w = torch.randint(-2 ** 31, 2 ** 31, (N, K // 8), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)
            self.s = ((0.5 + torch.rand(N, K // 128, generator=g, device=DEV)) * 0.01).to(torch.bfloat16)
            self.bytes = self.L.lib.b2q_linear_workspace_bytes(M, N, K)
        else:
            self.w = (torch.randn(N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(torch.float8_e4m3fn)
            self.s = torch.full((1,), 1 / 4096, device=DEV) if kind == "fp8" else (0.5 + torch.rand((N + 127) // 128, K // 128, generator=g, device=DEV)) / 4096
            self.bytes = self.L.lib.b2q_linear_fp8_workspace_bytes(M, N, K)
        self.ws = torch.zeros(self.bytes, dtype=torch.uint8, device=DEV)
        self.out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)

    def run(self, out=None):
        out = self.out if out is None else out
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        if self.kind == "int4":
            rc = self.L.lib.b2q_linear_int4(self.x.data_ptr(), self.L.dt(self.x), self.K, self.w.data_ptr(), self.L.W4_NMAJOR, self.s.data_ptr(), self.L.dt(self.s),
                                            self.K // 128, 1, out.data_ptr(), self.N, self.M, self.N, self.K, 128, self.ws.data_ptr(), self.bytes, st)
        else:
            mode = self.L.SCALE_TENSOR if self.kind == "fp8" else self.L.SCALE_BLOCK128
            rc = self.L.lib.b2q_linear_fp8(self.x.data_ptr(), self.L.dt(self.x), self.K, self.w.data_ptr(), self.L.fp8_fmt(self.w), self.s.data_ptr(), self.L.dt(self.s),
                                           mode, out.data_ptr(), self.N, self.M, self.N, self.K, self.ws.data_ptr(), self.bytes, st)
        assert rc == 0, self.L.lib.b2q_strerror(rc)
        return out


# kernel, force, kind, M, N, K; the scratch holds partial sums for each of them
CUT = [("w4_stream", 7, "int4", 1, 2048, 16384), ("w4_stream", 7, "int4", 8, 520, 8192), ("w4_stream", 7, "int4", 5, 57344, 512),
       ("umma_w4", 2, "int4", 16, 2048, 14336), ("umma_w4", 2, "int4", 40, 520, 14336), ("umma_w4", 2, "int4", 64, 40960, 4096), ("umma_w4", 2, "int4", 100, 8192, 28672),
       ("umma_w4", 2, "block", 27, 8192, 14336), ("umma_w4", 2, "block", 64, 1000, 14336),
       ("umma_w8_direct", 0, "fp8", 20, 5120, 13824), ("umma_w8_direct", 0, "fp8", 33, 520, 8192), ("umma_w8_direct", 0, "fp8", 64, 9400, 14336),
       ("umma_w4_i8", 5, "int4", 8, 2048, 14336), ("umma_w4_i8", 5, "int4", 16, 8200, 1024)]


@pytest.mark.parametrize("name,force,kind,M,N,K", CUT)
def test_any_scratch(e, name, force, kind, M, N, K):
    e.set_force_kernel(force)
    lin = Linear(e, kind, M, N, K, 1)
    ref = lin.run().clone()
    assert e.last_kernel() == name
    g = torch.Generator(device=DEV).manual_seed(2)
    for fill in range(12):
        if fill < 3:
            lin.ws.fill_((0xFF, 0x01, 0x7F)[fill])
        elif fill % 2:
            lin.ws.random_(generator=g)                      # else: as the launch before it left it
        lin.out.fill_(float("nan"))
        lin.run()
        assert torch.equal(lin.out, ref)
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("name,force,kind,M,N,K", CUT)
def test_replays_on_scratch_that_others_used(e, name, force, kind, M, N, K):
    """A captured launch keeps its tag: it must find no count of its own last replay, nor take another launch's for one."""
    e.set_force_kernel(force)
    lin = Linear(e, kind, M, N, K, 3)
    ref = lin.run().clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        lin.run()
    for i in range(8):
        lin.out.fill_(float("nan"))
        graph.replay()
        if i % 2:
            torch.cuda.synchronize()
            assert torch.equal(lin.out, ref)
        if i % 4 == 2:
            lin.ws.random_()
        if i % 4 == 3:
            lin.run()
    torch.cuda.synchronize()
    assert torch.equal(lin.out, ref) and e._lib.device_status() == 0


@pytest.mark.parametrize("name,force,kind,M,N,K", CUT)
def test_streams_and_graphs_side_by_side(e, name, force, kind, M, N, K):
    """Two streams with hundreds of launches queued on each, and two graphs of 64 launches replayed on a stream each."""
    e.set_force_kernel(force)
    lins = [Linear(e, kind, M, N, K, seed) for seed in (4, 5)]
    refs = [lin.run().clone() for lin in lins]
    streams = [torch.cuda.Stream() for _ in lins]
    outs = [torch.full((12, M, N), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in lins]
    graphs = []
    for lin in lins:
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            for _ in range(64):
                lin.run()
    torch.cuda.synchronize()
    for i, st in enumerate(streams):
        with torch.cuda.stream(st):
            for j in range(300):
                lins[i].run(outs[i][j % 12])
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(o, refs[i]) for o in outs[i])
    for _ in range(4):
        for lin in lins:
            lin.out.fill_(float("nan"))
        torch.cuda.synchronize()
        for graph, st in zip(graphs, streams):
            with torch.cuda.stream(st):
                graph.replay()
        torch.cuda.synchronize()
        for lin, ref in zip(lins, refs):
            assert torch.equal(lin.out, ref)
    assert e._lib.device_status() == 0


def test_reset_invalidates_counts_that_are_half_full(e):
    """What a launch leaves behind in which a wait ran out, and a replay of its graph finds: counts with its own tag and an arrival too many.
    After the reset they are nobody's.  (The tag is read off the counts of strips that one CTA has alone: opened, and never added to.)"""
    e.set_force_kernel(7)
    M, N, K = 5, 57344, 512
    lin = Linear(e, "int4", M, N, K, 6)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        lin.run()
    graph.replay()
    ref = lin.out.clone()
    grid = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    counts = lin.ws[2 * grid * 4096:2 * grid * 4096 + N // 128 * 4 * 8].view(torch.int64)
    tags = counts[counts != 0].unique()
    assert tags.numel() == 1 and int(tags[0]) & 1023 == 0
    counts.fill_(int(tags[0]) + 1)
    e._lib.device_status_reset()
    lin.out.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(lin.out, ref) and e._lib.device_status() == 0
