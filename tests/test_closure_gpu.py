"""The closure network's tensor-core kernels (tcgen05 implicit GEMMs) against the CPU oracle: forward
outputs and parameter gradients on random inputs and weights. Both sides round to BF16 at the same
points; the remaining differences are FP32 summation order (which moves a value near a BF16 rounding
boundary to the neighbouring BF16 value, 2^-8 relative in that element) and BF16 rounding of the backward's
intermediate gradients. Measured on a B200: 3.6e-4..4.5e-4 relative L2 forward, 1.3e-3..4.6e-3 per gradient
block; the bounds are 2e-3 (forward) and 1.5e-2 (gradients)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rand_case(shape, seed):
    from kaiju_b200 import gamera as gm
    Nip, Njp, Nkp = shape
    c = gm.Closure(Nip, Njp, Nkp, seed=seed)
    rng = np.random.default_rng(seed)
    p = c.params()
    p *= 4.0   # larger weights than the initial scale: the output and gradients are far from zero
    c.set_params(p)
    x = rng.normal(size=(Nip + 8, Njp + 8, Nkp + 8, 8)).astype(np.float32)
    return c, p, x


@pytest.mark.parametrize("shape", [(16, 8, 8), (32, 16, 12), (128, 4, 4)])
def test_forward_matches_oracle(shape):
    from oracle import closure_oracle as co
    c, p, x = _rand_case(shape, 3)
    y = c.forward_host(x)
    ref = co.net_forward(p, x)
    rel = np.linalg.norm(y - ref) / np.linalg.norm(ref)
    assert rel < 2e-3, rel
    c.close()


@pytest.mark.parametrize("shape", [(16, 8, 8), (32, 16, 12)])
def test_gradients_match_oracle(shape):
    from kaiju_b200 import gamera as gm
    from oracle import closure_oracle as co
    c, p, x = _rand_case(shape, 5)
    rng = np.random.default_rng(7)
    gout = rng.normal(size=shape + (gm.CLOSURE_OUT,)).astype(np.float32)
    g = c.backward_host(x, gout)
    ref = co.net_grads(p, x, gout)
    o = 0
    for cin, cout in co.LAYERS:
        for n in (27 * cin * cout, cout):
            a, b = g[o:o + n], ref[o:o + n]
            rel = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)
            assert rel < 1.5e-2, (cin, cout, n, rel)
            o += n
    c.close()


def test_boxes_of_several_tiles_per_cta():
    """A box in which every CTA of the convolution (two per SM, 126 cells a tile) takes three tiles or more, so that both
    accumulators, the rows handed from warp to warp and the window ring come round again, and every CTA of the weight
    gradient (one per SM, 128 cells) seven or eight, several turns of its ring. Forward and gradients against the oracle,
    with the bounds of the small boxes."""
    from kaiju_b200 import gamera as gm
    from oracle import closure_oracle as co
    shape = (40, 40, 40)   # 56 x 49 x 49 cells in the device's layout
    c, p, x = _rand_case(shape, 13)
    gout = np.random.default_rng(17).normal(size=shape + (gm.CLOSURE_OUT,)).astype(np.float32)
    y, g = c.forward_host(x), c.backward_host(x, gout)
    c.close()
    ref = co.net_forward(p, x)
    assert np.linalg.norm(y - ref) < 2e-3 * np.linalg.norm(ref)
    # every cell by itself: one that took a wrong row for one of its 27 taps would be off by about 1 / sqrt(27) of the
    # outputs' size, and a value on the other side of a BF16 rounding boundary moves one of its 864 terms by 2^-8 of it
    assert np.abs(y - ref).max() < 0.05 * np.sqrt(np.mean(ref ** 2))
    ref, o = co.net_grads(p, x, gout), 0
    for cin, cout in co.LAYERS:
        for n in (27 * cin * cout, cout):
            rel = np.linalg.norm(g[o:o + n] - ref[o:o + n]) / np.linalg.norm(ref[o:o + n])
            assert rel < 1.5e-2, (cin, cout, n, rel)
            o += n


@pytest.mark.parametrize("shape", [(16, 16, 16), (32, 32, 32), (48, 40, 40)])
def test_output_layer_gradient_sums(shape):
    """The sums over cells of the output layer's weight and bias gradients, against double sums of the same values: with
    zero weights below it its activations are the same everywhere. The tensor core truncates each addition to an
    accumulator (half of 2^-23 on the mean); a chain of 8 positive terms of a size is off by the sum of k/8 * 2^-24
    over k = 1..8, 2.7e-7, and the rounding of the result adds 2^-24 at most, whatever the number of cells."""
    import torch
    from kaiju_b200 import gamera as gm
    from oracle import closure_oracle as co
    c = gm.Closure(*shape, seed=2)
    rng = np.random.default_rng(11)
    p = np.zeros_like(c.params())
    o = 0
    for cin, cout in co.LAYERS[:3]:
        o += 27 * cin * cout
        p[o:o + cout] = rng.uniform(0.5, 2.0, cout)
        o += cout
    c.set_params(p)
    x = np.zeros((shape[0] + 8, shape[1] + 8, shape[2] + 8, 8), np.float32)
    act = np.asarray(co.hidden_activations(p, x[:9, :9, :9]), np.float64)   # one value per channel
    # exact in BF16, over many exponents, so that no sum of the products is exact in 24 bits
    gout = co._bf16(torch.from_numpy(np.exp(2.0 * rng.normal(size=shape + (gm.CLOSURE_OUT,))).astype(np.float32))).numpy()
    g = c.backward_host(x, gout).astype(np.float64)[o:]
    c.close()
    s = gout.astype(np.float64).sum(axis=(0, 1, 2))
    cin, cout = co.LAYERS[3]
    for got, want in ((g[:27 * cin * cout], np.tile(np.outer(s, act).ravel(), 27)), (g[27 * cin * cout:], s)):
        rel = np.linalg.norm(got - want) / np.linalg.norm(want)
        assert rel <= 2.7e-7 + 2.0 ** -24, rel


def test_phase_times_count_the_network_with_the_deltas():
    """profile_phases times the network with Flux2Deltas, which takes its corrections: many times the predictor's work."""
    from kaiju_b200 import gamera as gm, turbulence as tu
    g = tu.turbulence_problem(32, seed=5)
    c = gm.Closure(32, 32, 32, seed=1)
    plain = g.profile_phases(4)
    g.set_closure(c)
    g.profile_phases(2)
    t = g.profile_phases(8)
    assert t["predictor"] < 2.0 * plain["predictor"] + 0.02 and t["deltas"] > 2.0 * t["predictor"], (plain, t)
    g.set_closure(None)
    g.close()
    c.close()
