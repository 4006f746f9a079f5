"""The sizing network's fused training step against its gradients: a step
changes weights and biases by Adam of exactly the gradients that kc_mlp_gradients
reports, whatever the batch (tiles of 16 and 64 rows, remainders, one row) and
layer widths (multiples of 8, for the 16-byte copies, and not; contractions
short and long), over several steps whose inputs alternate buffers."""
import numpy as np
import pytest

from kmertreecounter_b200 import sizing

pytestmark = pytest.mark.gpu


def _bf16(a):
    u = np.ascontiguousarray(a, np.float32).view(np.uint32).astype(np.uint64)
    return (((u + 0x7FFF + ((u >> 16) & 1)) >> 16) << 16).astype(np.uint32).view(np.float32)


@pytest.mark.parametrize("dims", [(72, 48, 40), (2056, 136, 2304), (131, 77, 203), (4104, 512, 8192)])
@pytest.mark.parametrize("batch", [1, 15, 32, 64, 100])
def test_step_is_adam_of_the_gradients(dims, batch):
    if dims[0] > 4000 and batch not in (32, 100):
        pytest.skip("the full width at two batch sizes")
    rng = np.random.default_rng(batch + dims[0])
    m = sizing.MLP(*dims, max_batch=batch, seed=5)
    layers = [m.get_layer(l) for l in range(3)]
    mom = [[np.zeros_like(a, np.float64) for a in wb] for wb in layers]
    vel = [[np.zeros_like(a, np.float64) for a in wb] for wb in layers]
    lr = 1e-3
    for step in range(1, 4):
        x = rng.normal(size=(batch, dims[0])).astype(np.float32)
        t = rng.normal(size=(batch, dims[2])).astype(np.float32)
        grads = [m.gradients(x, t, l) for l in range(3)]
        # forward in 32 bits from the 16-bit operands: the loss both calls report
        h = _bf16(x)
        for l, (w, b) in enumerate(layers):
            z = h.astype(np.float64) @ _bf16(w).astype(np.float64) + b
            h = _bf16(np.maximum(z, 0.0)) if l < 2 else z
        want = float(np.mean((h - t) ** 2))
        loss = m.train_step(x, t, lr)
        assert loss == pytest.approx(grads[0][2], rel=1e-5)
        # a 32-bit sum that rounds the other way moves a 16-bit activation by 2^-8
        assert loss == pytest.approx(want, rel=2.0 ** -8)
        for l in range(3):
            new = m.get_layer(l)
            for p in range(2):
                g = grads[l][p].astype(np.float64)
                mom[l][p] = 0.9 * mom[l][p] + 0.1 * g
                vel[l][p] = 0.999 * vel[l][p] + 0.001 * g * g
                step_by = lr * (mom[l][p] / (1 - 0.9 ** step)) / (np.sqrt(vel[l][p] / (1 - 0.999 ** step)) + 1e-8)
                expect = layers[l][p].astype(np.float64) - step_by
                # 32-bit arithmetic: a few roundings of the step and one of the
                # weight; a gradient whose square underflows divides by eps
                normal = np.abs(g) > 1e-18
                err = np.abs(new[p].astype(np.float64) - expect)
                assert np.all(err[normal] <= 2e-5 * lr + 2.0 ** -22 * np.abs(expect[normal]))
            layers[l] = new
    m.close()
