"""Order of the sums in the parameter gradients of the U-Net.  A gradient near
zero takes its sign from the rounding of its sum, and Adam turns that sign
into a whole step of the weight, so the sums keep their composition: chains
over all rows of a tile in order, the same tiles in one chain, the same pixels
in a chain of a bias or head sum, and meet in one order.  The recorded gradients
(golden/unet_grads.npz) are those of the kernels with one warp per tap and one
thread per chain; `python tests/test_gpu_unet_sums.py FILE` on a GPU writes
the present ones.

16 x 16, one image: at most two partial sums per weight, so any order of the
atomics gives the same bits (and for the biases of the 128- and 256-channel
layers, of one or two chains).  16 x 256 x 256: chains of 12 and 13 tiles in
the 256- and 384-channel layers, ten to thirteen partial sums per weight.
Each of the 12 additions, in both runs, rounds by at most 2^-24 of its result
(2^-24 / sqrt 3 RMS), so two orders differ by sqrt(24) 2^-24 / sqrt 3 = 1.7e-7
of the RMS.  The head's 33 sums of up to 2368 partial sums: sqrt(2 x 2368)
2^-24 / sqrt 3 = 2.4e-6."""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).resolve().parent / "golden" / "unet_grads.npz"
DEEP = (7, 8)  # layers 256 -> 256 and 384 -> 128
STRIDE = 61    # one weight of so many is recorded


def _gradients(sdp, n, size, seed):
    import torch
    import unet_ref as U
    rng = np.random.default_rng(seed)
    p = U.init_params(32, 3, rng)
    net = sdp.UNet(sdp.load(), 3, n, size, size)
    net.set_params(p)
    x = torch.from_numpy(rng.standard_normal((n, 3, size, size)).astype(np.float32)).cuda()
    go = torch.from_numpy((1e-3 * rng.standard_normal((n, size, size))).astype(np.float32)).cuda()
    out = torch.empty((n, size, size), device="cuda")
    net.forward(x, out)
    net.zero_grads()
    net.backward(go)
    g = net.get_grads()
    net.close()
    layers, head, _ = U.layer_table(32)
    return g, layers, head


def _record(sdp):
    g, layers, _ = _gradients(sdp, 1, 16, 21)
    d = {f"small_w{k}": g[wo:wo + 9 * ci * co:STRIDE].copy() for k, (ci, co, wo, bo) in enumerate(layers)}
    d.update({f"small_b{k}": g[bo:bo + co].copy() for k, (ci, co, wo, bo) in enumerate(layers) if co >= 128})
    g, layers, head = _gradients(sdp, 16, 256, 22)
    d.update({f"large_w{k}": g[layers[k][2]:layers[k][2] + 9 * layers[k][0] * layers[k][1]:STRIDE].copy() for k in DEEP})
    d["large_head"] = g[head[0]:].copy()
    return d


def test_sums_keep_their_composition(sdp, device):
    got, ref = _record(sdp), np.load(GOLDEN)
    assert set(got) == set(ref.files)
    for k in ref.files:
        if k.startswith("small"):
            np.testing.assert_array_equal(got[k], ref[k], err_msg=k)
        else:
            bound = 2.4e-6 if k == "large_head" else 1.7e-7
            d = got[k].astype(np.float64) - ref[k]
            rel = np.sqrt(np.mean(d ** 2) / np.mean(ref[k].astype(np.float64) ** 2))
            assert rel <= bound, (k, rel)


def test_steps_repeat_bit_for_bit(sdp, device):
    """Three training steps from one state, twice: no sum depends on the order
    in which CTAs finish."""
    import torch
    import unet_ref as U
    rng = np.random.default_rng(5)
    p = U.init_params(32, 3, rng)
    n, size = 4, 128
    x = torch.from_numpy(rng.standard_normal((n, 3, size, size)).astype(np.float32)).cuda()
    target = torch.from_numpy(rng.standard_normal((n, size, size)).astype(np.float32)).cuda()
    runs = []
    for _ in range(2):
        net = sdp.UNet(sdp.load(), 3, n, size, size)
        net.set_params(p)
        out, grad = torch.empty((n, size, size), device="cuda"), torch.empty((n, size, size), device="cuda")
        scratch, loss = torch.empty(2 * n * size * size, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
        seen = []
        for _ in range(3):
            net.forward(x, out)
            device.blur_mse(out, target, scratch, grad, loss)
            net.zero_grads()
            net.backward(grad)
            net.adam_step(1e-3)
            seen += [out.cpu().numpy(), net.get_grads(), net.get_params()]
        net.close()
        runs.append(seen)
    for a, b in zip(*runs):
        np.testing.assert_array_equal(a, b)


def test_gradients_accumulate(sdp, device):
    """A second backward pass adds to the gradients of the first."""
    import torch
    import unet_ref as U
    rng = np.random.default_rng(6)
    net = sdp.UNet(sdp.load(), 3, 2, 64, 64)
    net.set_params(U.init_params(32, 3, rng))
    x = torch.from_numpy(rng.standard_normal((2, 3, 64, 64)).astype(np.float32)).cuda()
    go = torch.from_numpy(rng.standard_normal((2, 64, 64)).astype(np.float32)).cuda()
    net.forward(x, torch.empty((2, 64, 64), device="cuda"))
    net.zero_grads()
    net.backward(go)
    once = net.get_grads()
    net.backward(go)
    twice = net.get_grads()
    net.close()
    np.testing.assert_allclose(twice, 2 * once, rtol=2.0 ** -22, atol=0)


if __name__ == "__main__":
    sys.path[:0] = [str(Path(__file__).resolve().parent.parent / "simsdp-generic-imaging-pipeline_b200"),
                    str(Path(__file__).resolve().parent.parent / "oracle")]
    import sdp_b200
    np.savez_compressed(sys.argv[1], **_record(sdp_b200))
