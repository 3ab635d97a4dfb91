"""b200_decoder_linears_only says how many kernels it launched (include/b200llm.h): counted in a captured graph for every weight format on both sides of the sizes at which
a norm leaves its linear and a linear goes in passes."""
import ctypes
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
m = importlib.import_module("llm-inference-engine_b200")
DEV = "cuda"


@pytest.mark.parametrize("batch", [1, 2, 4, 5, 16, 17, 40])
@pytest.mark.parametrize("fmt", ["f32", "dense", "fp8", "int4"])
def test_the_number_of_launches(fmt, batch):
    h, heads, inter, layers, d = 512, 4, 768, 2, 128
    dtype = torch.float32 if fmt == "f32" else torch.bfloat16
    gen = torch.Generator(device=DEV).manual_seed(batch)

    def weight(n, k):
        if fmt == "fp8":
            return torch.randn(n, k, generator=gen, device=DEV).to(torch.float8_e4m3fn).view(torch.uint8), torch.rand(n, generator=gen, device=DEV) / k ** 0.5, None
        if fmt == "int4":
            return (torch.randint(0, 256, (n, k // 2), generator=gen, device=DEV, dtype=torch.uint8), (torch.rand(n, k // 128, generator=gen, device=DEV) / k ** 0.5).to(dtype),
                    torch.full((n, k // 128), 8, device=DEV, dtype=torch.uint8))
        return (torch.randn(n, k, generator=gen, device=DEV) / k ** 0.5).to(dtype)

    ones = torch.ones(h, device=DEV, dtype=dtype)
    code, form = (m.F32 if fmt == "f32" else m.BF16), {"fp8": m.W_FP8, "int4": m.W_INT4}.get(fmt, m.W_DENSE)
    dec = m.Decoder(m.DecoderConfig(h, heads, heads, d, inter, layers, 64, batch, code, form, 128, 1e-6, d, 10000.0, 1, 0), DEV)
    for i in range(layers):
        dec.set_layer(i, {"g1": ones, "g2": ones, "qkv": weight(3 * heads * d, h), "o": weight(h, heads * d), "gate_up": weight(2 * inter, h), "down": weight(h, inter)})
    k, v = (torch.zeros(layers, batch, heads, 64, d, device=DEV, dtype=dtype) for _ in range(2))
    dec.step(torch.randn(batch, h, generator=gen, device=DEV).to(dtype), k, v, 1)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        said = dec.linears_only(batch)
    nodes = ctypes.c_size_t(0)  # (kernels are all that it launches)
    assert ctypes.CDLL("libcuda.so.1").cuGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None, ctypes.byref(nodes)) == 0
    assert said == nodes.value
