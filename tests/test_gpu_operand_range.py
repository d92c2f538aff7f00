"""Accuracy of the expert term, token by token, for layers whose values are uneven inside the rows of an operand.

Most cases rescale an ordinary layer by powers of two that cancel: one neuron with large weights whose wo column makes up
for it, LayerNorm weights of many magnitudes, and so on.  The layer computes the same function, so its accuracy has to
be that of the ordinary one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Expert term of one token, 2-norm, relative: operands to 2^-22 and sums of truncating 256-value chunks, 2e-6 to 3e-6 on
# ordinary weights; the layer's stated limit.  The residual add rounds once more, 2^-24 of the output.
TOL = 1e-5


def _ordinary(rng, n, D, F):
    x = rng.standard_normal((n, D)).astype(np.float32)
    ln = (1 + 0.01 * rng.standard_normal(D)).astype(np.float32)
    wi0, wi1 = ((rng.standard_normal((F, D)) / np.sqrt(D)).astype(np.float32) for _ in range(2))
    wo = (rng.standard_normal((D, F)) / np.sqrt(F)).astype(np.float32)
    return x, ln, wi0, wi1, wo


def _powers(rng, n, most):
    return np.exp2(rng.integers(-most, most + 1, n)).astype(np.float32)


def _neuron(c, wo_factor):
    def scale(rng, x, ln, wi0, wi1, wo):
        f = wi0.shape[0] // 3
        wi0[f] *= np.float32(c)
        wi1[f] *= np.float32(c)
        wo[:, f] *= np.float32(wo_factor)
        return x, ln, wi0, wi1, wo
    return scale


def _gamma(most):
    def scale(rng, x, ln, wi0, wi1, wo):
        k = _powers(rng, ln.size, most)
        return x, ln * k, wi0 / k, wi1 / k, wo
    return scale


def _wi1_rows(most):
    def scale(rng, x, ln, wi0, wi1, wo):
        k = _powers(rng, wi1.shape[0], most)
        return x, ln, wi0, wi1 * k[:, None], wo / k
    return scale


def _features(most, into):
    def scale(rng, x, ln, wi0, wi1, wo):
        k = _powers(rng, ln.size, most)
        return (x * k, ln / k, wi0, wi1, wo) if into == "gamma" else (x * k, ln, wi0 / k, wi1 / k, wo)
    return scale


def _dead_feature(rng, x, ln, wi0, wi1, wo):
    """a feature that takes nearly all of LayerNorm's variance and that no neuron reads"""
    x[:, 3] = np.float32(2.0 ** 14)
    wi0[:, 3] = wi1[:, 3] = 0
    return x, ln * np.float32(2.0 ** 14 / np.sqrt(ln.size)), wi0, wi1, wo


def _heavy_column(rng, x, ln, wi0, wi1, wo):
    """a feature with large weights that half of the tokens do not have"""
    wi0[:, 3] *= np.float32(2.0 ** 12)
    wi1[:, 3] *= np.float32(2.0 ** 12)
    x[::2, 3] = x[::2].mean(axis=1)
    return x, ln, wi0, wi1, wo


def _far_magnitudes(rng, x, ln, wi0, wi1, wo):
    return x, ln * np.float32(2.0 ** -30), wi0 * np.float32(2.0 ** 10), wi1 * np.float32(2.0 ** 50), wo


CASES = {
    "ordinary": lambda rng, *w: w,
    "neuron_x100": _neuron(100.0, 1e-4),
    "neuron_x1000": _neuron(1000.0, 1e-6),
    "neuron_x1000_without_output": _neuron(1000.0, 0.0),
    "gamma_2^6": _gamma(6),
    "gamma_2^8": _gamma(8),
    "gamma_2^24": _gamma(24),
    "wi1_rows_2^8": _wi1_rows(8),
    "wi1_rows_2^24": _wi1_rows(24),
    "features_2^6_gamma_inverse": _features(6, "gamma"),
    "features_2^6_wi_inverse": _features(6, "wi"),
    "dead_feature": _dead_feature,
    "heavy_column": _heavy_column,
    "far_magnitudes": _far_magnitudes,
}


def _token_errors(got, x, want):
    """Error of each token beyond the residual add's rounding, relative to its expert term."""
    err = np.maximum(np.abs(got.astype(np.float64) - want) - 2.0 ** -24 * np.abs(want), 0.0)
    return np.linalg.norm(err, axis=1) / np.linalg.norm(want - x.astype(np.float64), axis=1)


# weights laid out in one launch and in three, one and two token tiles, one CTA and pairs (K >= 2048), K tails
@pytest.mark.parametrize("n,D,F", [(33, 200, 600), (40, 512, 1024), (150, 1000, 2724), (70, 2048, 516)])
@pytest.mark.parametrize("case", list(CASES))
def test_expert_term_of_every_token(oracle, case, n, D, F):
    from tests import gpu_util as g
    rng = np.random.default_rng(n + D + F)
    x, ln, wi0, wi1, wo = CASES[case](rng, *_ordinary(rng, n, D, F))
    got = g.t5ff_run(x, ln, wi0, wi1, wo)
    err = _token_errors(got, x, oracle.expert_ffn_f64(x, ln, wi0, wi1, wo))
    print(f"{case} {n} x {D} x {F}: worst token {err.max():.2e}")
    assert 1e-8 < err.max() <= TOL                   # and the expert term is what is looked at


@pytest.mark.parametrize("n,D,F", [(64, 1024, 2048), (100, 4096, 1024)])
@pytest.mark.parametrize("c", [64.0, 128.0, 1024.0, 4096.0])
def test_one_large_neuron_leaves_tokens_it_is_off_for_alone(oracle, c, n, D, F):
    """Nothing makes up for the large neuron here.  It decides the result of the tokens it is on for; those for which
    gelu switches it off have an ordinary result, to which its scale must not matter."""
    from tests import gpu_util as g
    rng = np.random.default_rng(int(c) + D)
    x, ln, wi0, wi1, wo = _neuron(c, 1.0)(rng, *_ordinary(rng, n, D, F))
    f = F // 3
    centred = x.astype(np.float64) - x.mean(axis=1, keepdims=True, dtype=np.float64)
    a = (ln * centred / np.sqrt((centred ** 2).mean(axis=1, keepdims=True) + 1e-6)) @ wi0[f].astype(np.float64)
    off = a < -20.0                                  # gelu(a) below 10^-80
    assert off.sum() >= 10
    got = g.t5ff_run(x, ln, wi0, wi1, wo)
    err = _token_errors(got, x, oracle.expert_ffn_f64(x, ln, wi0, wi1, wo))[off]
    print(f"neuron x {c:.0f}, {n} x {D} x {F}: worst of {off.sum()} tokens {err.max():.2e}")
    assert err.max() <= TOL


# smallest widths, both sides of the one-launch layout (131072 values a matrix), K and row tails of the layout's blocks of 128 and 32
@pytest.mark.parametrize("n,D,F", [(3, 8, 8), (17, 36, 12), (9, 2048, 64), (9, 2052, 64), (65, 132, 2044),
                                   (40, 2080, 388), (200, 640, 520)])
def test_powers_of_two_moved_between_gamma_and_wi_change_no_bit(n, D, F):
    """The layout moves the exponent of a column's largest weight into the LayerNorm weight, so a power of two moved from
    the one to the other is moved back, exactly."""
    from tests import gpu_util as g
    rng = np.random.default_rng(n * D + F)
    plain = _ordinary(rng, n, D, F)
    np.testing.assert_array_equal(g.t5ff_run(*_gamma(24)(rng, *plain)), g.t5ff_run(*plain))


def _layer(experts, centroids, D, F, host, cache):
    import torch
    from infmoe_b200 import MoELayer
    layer = MoELayer.create(len(experts), D, F, 2, centroids, None, "T5_FF", "base_layer", None)
    for e, ex in enumerate(experts):
        layer.set_expert(e, *(ex if host else [torch.from_numpy(a).cuda() for a in ex]))
    layer.set_residency(0 if host else 1)
    if cache:
        layer.set_expert_cache(cache)
    return layer


# few and many tokens take different scatter kernels, and so do the widths; the rows of a streamed expert are scattered once
# it has arrived on its first pass, with all others from then on
@pytest.mark.parametrize("T,D,F", [(1, 256, 512), (200, 256, 512), (1500, 256, 512), (1300, 4100, 64), (100, 6020, 64)])
def test_layer_resident_streamed_and_cached(oracle, T, D, F):
    import torch
    rng = np.random.default_rng(T + D)
    E = 4
    experts = []
    for e in range(E):
        w = _ordinary(rng, 1, D, F)
        w = _wi1_rows(8)(rng, *_gamma(3 + 7 * e)(rng, *w))
        experts.append([np.ascontiguousarray(a) for a in w[1:]])
    x = rng.standard_normal((T, D)).astype(np.float32)
    centroids = rng.standard_normal((E, D)).astype(np.float32) * np.float32(0.02)
    layer = _layer(experts, centroids, D, F, False, 0)
    out = layer.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    layer.sync_status()
    layer.terminate()
    ref = oracle.layer_forward_f32(x, "base_layer", centroids, None, experts)
    want = oracle.layer_forward_f64(x, "base_layer", ref["gate"], ref["score"], experts)
    assert _token_errors(out, x, want).max() <= TOL
    for cache in (0, 2, E):
        layer = _layer(experts, centroids, D, F, True, cache)
        for _ in range(2):                           # the second call finds the slots, or the cache, filled
            np.testing.assert_array_equal(layer.forward(torch.from_numpy(x).cuda()).cpu().numpy(), out)
        # other weights with another LayerNorm weight in the place of one expert's, and the next pass on another stream
        layer.set_expert(1, *experts[3])
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
            replaced = layer.forward(torch.from_numpy(x).cuda())
            torch.cuda.current_stream().synchronize()
        layer.terminate()
        same = [experts[0], experts[3], experts[2], experts[3]]
        layer = _layer(same, centroids, D, F, False, 0)
        np.testing.assert_array_equal(replaced.cpu().numpy(), layer.forward(torch.from_numpy(x).cuda()).cpu().numpy())
        layer.terminate()


def test_weights_at_unaligned_addresses(oracle):
    """Device matrices that start on a 4-byte boundary take scalar loads into the same layout."""
    import torch
    from infmoe_b200 import MoELayer
    rng = np.random.default_rng(5)
    D, F = 132, 260
    x, *expert = _gamma(8)(rng, *_ordinary(rng, 50, D, F))
    outs = []
    for shift in (0, 1, 3):
        layer = MoELayer.create(1, D, F, 2, np.ones((1, D), np.float32), None, "T5_FF", "default", None)
        held = []
        for a in expert:
            t = torch.empty(a.size + shift, device="cuda")
            t[shift:] = torch.from_numpy(np.ascontiguousarray(a)).cuda().ravel()
            held.append(t[shift:].view(a.shape))
        layer.set_expert(0, *held)
        outs.append(layer.forward(torch.from_numpy(x).cuda()).cpu().numpy())
        layer.terminate()
    assert _token_errors(outs[0], x, oracle.expert_ffn_f64(x, *expert)).max() <= TOL
    np.testing.assert_array_equal(outs[1], outs[0])
    np.testing.assert_array_equal(outs[2], outs[0])
