"""The shared memory that a kernel's launches may ask for is a property of the function in the whole process: only allow_smem (csrc/runtime.cu) raises it, once per
device, to the most that any launch asks for.  A launch that set its own size would lower it between another thread's set and launch."""
import glob
import importlib
import os
import re
import threading

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm-inference-engine_b200", "csrc")


def test_one_place_raises_the_limit():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        found += [os.path.basename(path)] * len(re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize", text))
    assert found == ["runtime.cu"], found


@pytest.mark.gpu
def test_decoded_tokens_of_two_threads():
    """Two engines whose decoded tokens ask for different shared memory (eight query heads of one key head of 128, a sixteenth of 6500 and of 8000 keys a CTA: 50 and
    53 KB), stepped by a thread each."""
    import torch
    import vasolix_oracle as ref

    config = ref.make_config([ref.attention_layer(heads=8, kv_heads=1, dim=128, size=8192, scale=128 ** -0.5) for _ in range(4)], width=64)
    _, packed = ref.make_weights(config, seed=5)
    cls = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel
    serving = importlib.import_module("llm-inference-engine_b200.serving")
    steps, contexts = 150, (6500, 8000)

    def run(n, out):
        with torch.cuda.stream(torch.cuda.Stream()):
            model = cls(config, packed, dtype="bfloat16", device="cuda:0", max_tokens=2048, max_seqs=1, max_pages_per_seq=128)
            sess = serving.Session(model, 8192, max_seqs=1, max_batch_tokens=2048, poison=True)
            toks = np.random.default_rng(n).integers(0, config["vocab"], n + steps).tolist()
            i = sess.open()
            for a in range(0, n, 2000):
                sess.feed([(i, toks[a:min(a + 2000, n)], [])])
            out[n] = torch.cat([sess.feed([(i, toks[n + k:n + k + 1], [0])]) for k in range(steps)])
            torch.cuda.synchronize()

    alone, together = {}, {}
    for n in contexts:
        run(n, alone)
    threads = [threading.Thread(target=run, args=(n, together)) for n in contexts]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for n in contexts:
        assert n in together, "a step failed"
        assert torch.equal(together[n], alone[n])
