"""The tensor-core GEMM between the kernels of its stream, under programmatic dependent launch."""

import ctypes
import shutil
import subprocess

import pytest
import torch

from fdk import models, native

pytestmark = pytest.mark.gpu

# Lets the next kernel start, stays busy for a while (bounded by its clock and by a count), then writes x.
SLOW_PRODUCER = r"""
#include <cuda_runtime.h>
__global__ void slow_producer(const uint4* src, uint4* dst, int vectors, unsigned long long ns) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  unsigned long long t0, now;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (unsigned i = 0; i < 100000000u; ++i) {
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (now - t0 > ns) break;
    __nanosleep(1000);
  }
  for (int i = threadIdx.x; i < vectors; i += blockDim.x) dst[i] = src[i];
}
extern "C" int launch_slow_producer(const void* src, void* dst, int vectors, unsigned long long ns, void* stream) {
  slow_producer<<<1, 256, 0, (cudaStream_t)stream>>>((const uint4*)src, (uint4*)dst, vectors, ns);
  return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def slow_producer(tmp_path_factory):
    folder = tmp_path_factory.mktemp("slow_producer")
    source, library = folder / "slow_producer.cu", folder / "slow_producer.so"
    source.write_text(SLOW_PRODUCER)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC",
                    "-o", str(library), str(source)], check=True)
    fn = ctypes.CDLL(str(library)).launch_slow_producer
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_ulonglong, ctypes.c_void_p]
    return fn


@pytest.mark.parametrize("m,bits", [(32, 4), (200, 8), (32, 1), (100, 3)])
def test_bounded_waits_do_not_count_the_kernel_before(slow_producer, m, bits):
    """The kernel before takes longer than the two seconds after which a wait gives up, and hands over x only
    then: no wait runs out, and the result is that of a launch in plain order.  Every CTA's share is longer than its
    rings of code slots and stages, so that every role reaches its second uses."""
    n, k = 11264, 16384
    gen = torch.Generator(device="cuda").manual_seed(m + bits)
    w = (torch.randn((n, k), generator=gen, device="cuda") * k**-0.5).bfloat16()
    layer = models.QuantisedLinear.create(w, models.QuantisationConfig(bits, 64))
    source = torch.randn((m, k), generator=gen, device="cuda").bfloat16()
    args = (layer.tiled(), layer.lut)
    want = torch.empty((m, n), device="cuda", dtype=torch.bfloat16)
    native.linear_lut(source, *args, want, n, k, bits)
    x, got = torch.full_like(source, float("nan")), torch.empty_like(want)
    torch.cuda.synchronize()
    assert slow_producer(source.data_ptr(), x.data_ptr(), x.numel() // 8, 2_600_000_000, native._stream()) == 0
    native.linear_lut(x, *args, got, n, k, bits, pdl=True)
    torch.cuda.synchronize()
    assert native.device_status() == 0
    assert torch.equal(got, want)


class EdgeData(ctypes.Structure):
    """`cudaGraphEdgeData`; type 1 is a programmatic dependency, 0 a full one."""

    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte), ("reserved", ctypes.c_ubyte * 5)]


def graph_edges(graph: int) -> list[tuple[int, int, bool]]:
    """(node, its successor, whether the successor may start before the node has completed) of a captured graph."""
    get = ctypes.CDLL("libcudart.so.12").cudaGraphGetEdges_v2
    count = ctypes.c_size_t(0)
    assert get(ctypes.c_void_p(graph), None, None, None, ctypes.byref(count)) == 0
    sources, targets = ((ctypes.c_void_p * count.value)() for _ in range(2))
    data = (EdgeData * count.value)()
    assert get(ctypes.c_void_p(graph), sources, targets, data, ctypes.byref(count)) == 0
    return [(a, b, e.type == 1) for a, b, e in zip(sources, targets, data)]


@pytest.mark.parametrize("m", [1, 8, 32])
def test_no_launch_reads_a_tiled_buffer_early_that_the_kernel_before_wrote(m):
    """The first call of a layer repacks its weight and launches the projection, which reads codes before it waits
    for its predecessor.  Captured and not run: the repack's successor depends on it in full, and the
    projection's early start is on a kernel that wrote nothing."""
    layer = models.QuantisedLinear.create(torch.randn((256, 512), device="cuda").bfloat16(), models.QuantisationConfig(4, 64))
    x = torch.randn((m, 512), device="cuda").bfloat16()
    graph, stream = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        layer.tiled()
        stream.synchronize()
        layer(x)  # the stream's workspace and the host copy of the table
        stream.synchronize()
        layer._tiled_key = None  # as after a change of the weight
        with torch.cuda.graph(graph, stream=stream):
            layer(x)
    edges = graph_edges(graph.raw_cuda_graph())
    (repack,) = {a for a, _, _ in edges} - {b for _, b, _ in edges}  # the first kernel
    assert not any(programmatic for a, _, programmatic in edges if a == repack), edges
    assert any(programmatic for _, _, programmatic in edges), edges


@pytest.mark.parametrize("left", [1, 2])
def test_flags_of_an_earlier_launch_are_not_taken_for_this_ones(left):
    """What a launch whose wait ran out can leave behind: flags published late, sums that belong to nothing, a status
    word that is set.  Few tiles over long rows, so that nearly every CTA parks its sums; launches 1 and 2 on
    the workspace are over."""
    m, n, k = 40, 64, 64 * 150
    layer = models.QuantisedLinear.create(torch.randn((n, k), device="cuda").bfloat16(), models.QuantisationConfig(4, 64))
    x = torch.randn((m, k), device="cuda").bfloat16()
    want = [layer(x) for _ in range(3)][-1]
    workspace = native.workspace(x.device)
    flags, counted, status = 1327104, 160 * 48 * 4, 4095 * 4  # as laid out in lut_table.cuh
    assert bool((workspace[flags: flags + counted].view(torch.int32) != 0).any())
    workspace[flags: flags + counted].view(torch.int32).fill_(left)
    workspace[flags + counted + 256:].view(torch.float32).fill_(float("nan"))
    workspace[status: status + 4].view(torch.int32).fill_(1)
    try:
        for _ in range(3):
            assert torch.equal(layer(x), want)
        assert native.device_status() == 1  # set until the workspace is initialised again
    finally:
        native.check(native.lib().fdk_workspace_init(workspace.data_ptr(), workspace.numel(), native._stream()))
    assert torch.equal(layer(x), want) and native.device_status() == 0
