"""The order in which a window of <= 16 rows is summed is part of its results: eight products an instruction, partial sums of 256 k (or
of the next cut that leaves at most eight), added ascending.  tests/golden/window_sums.json holds SHA-256 sums of layer outputs
recorded from the three-launch kernels that the streamed kernel replaced; the streamed kernel gives the same bytes."""
import hashlib
import json
import os

import numpy as np
import pytest

from conftest import ROOT

GOLDEN = os.path.join(ROOT, "tests", "golden", "window_sums.json")
# hidden, inter, experts, slots, rows: splits of 256 k, of 512 k, of 384 k (K = 2304), of 640 k (3840) and of 1024 k (8192); a single one;
# one member set and two, and members beyond the eighth
CASES = [(2048, 1536, 6, 3, 1), (2048, 1536, 6, 3, 8), (2048, 1536, 6, 3, 16), (4096, 512, 8, 5, 1), (4096, 512, 8, 5, 11), (2304, 768, 4, 3, 3),
         (512, 2304, 4, 3, 13), (3840, 256, 3, 2, 2), (8192, 256, 3, 2, 1), (256, 256, 2, 2, 9), (768, 1280, 12, 9, 5), (1280, 3072, 3, 2, 4)]


def layer_digest(pkg, synth, cuda, H, I, E, S, rows):
    import torch
    bank = synth.to_device(synth.expert_bank(61 + H + I, H, I, E, svh_scale=True), cuda)
    x, (picks, rw) = synth.activations_bf16(62 + rows, rows, H), synth.route(63 + rows, rows, E, S - 1, shared_bias=rows > 1)
    moe = pkg.Moe(pkg.make_config(H, I, E, S, max_rows=rows))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    moe.run(bank, t(x.view(np.int16)).view(torch.bfloat16), t(picks), t(rw), rows)
    torch.cuda.synchronize()
    assert int(moe.status.cpu()[0]) == 0
    return hashlib.sha256(moe.output[:rows].contiguous().cpu().numpy().tobytes()).hexdigest()


@pytest.mark.gpu
@pytest.mark.parametrize("H,I,E,S,rows", CASES)
def test_window_sums_keep_their_bytes(pkg, synth, cuda, H, I, E, S, rows):
    want = json.load(open(GOLDEN))
    assert layer_digest(pkg, synth, cuda, H, I, E, S, rows) == want[f"{H}x{I}x{E}x{S}x{rows}"]
