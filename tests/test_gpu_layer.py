"""GPU parity of the whole layer (MoELayerPlugin::enqueue) through the C ABI."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5   # relative L2 against the FP64-accumulated oracle


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available(), "these tests need a GPU"
    return torch


def _build(w, synth, tmp_path=None, residency=-1, from_npz=True, mc=None):
    from infmoe_b200 import MoELayer
    x, c, ln = synth.gen_inputs(w)
    experts = [synth.gen_expert_numpy(w, e) for e in range(w.expert_count)]
    path = synth.write_npz(w, str(tmp_path / f"{w.name}.npz")) if from_npz else None
    layer = MoELayer.create(w.expert_count, w.embedding_size, w.hidden_size, mc or w.max_concurrency, c, path, "T5_FF",
                            w.variant, ln)
    if from_npz:
        layer.initialize()
    else:
        for e, ex in enumerate(experts):
            layer.set_expert(e, *ex)
    layer.set_residency(residency)
    return layer, x, c, ln, experts


def _routing(layer, T, E, torch):
    from tests.gpu_util import read_device as rd
    gate, score, pos, count, offset = layer.last_routing()
    return (rd(gate, T, np.int32), rd(score, T, np.float32), rd(pos, T, np.int32), rd(count, E, np.int32),
            rd(offset, E + 1, np.int32))


def _check(layer, w, x, c, ln, experts, oracle, torch, tol=TOL):
    out = layer.forward_host(x)
    ref = oracle.layer_forward_f32(x, w.variant, c, ln, experts)
    gate, score, pos, count, offset = _routing(layer, w.tokens, w.expert_count, torch)
    np.testing.assert_array_equal(gate, ref["gate"])
    np.testing.assert_array_equal(score.view(np.uint32), ref["score"].view(np.uint32))
    np.testing.assert_array_equal(count, ref["count"])
    np.testing.assert_array_equal(offset, ref["offset"])
    np.testing.assert_array_equal(pos, ref["pos"])
    o64 = oracle.layer_forward_f64(x, w.variant, ref["gate"], ref["score"], experts)
    err = oracle.rel_l2(out, o64)
    assert err <= tol, err
    assert oracle.rel_l2(out - x, o64 - x) <= 10 * tol      # the expert contribution itself
    return out


@pytest.mark.parametrize("variant", ["default", "cpm_2", "base_layer"])
def test_tiny_layer_from_npz(torch_cuda, oracle, tmp_path, variant):
    from infmoe_b200 import synth
    w = synth.scaled(synth.WORKLOADS["tiny_default"], variant=variant)
    layer, x, c, ln, experts = _build(w, synth, tmp_path)
    out = _check(layer, w, x, c, ln, experts, oracle, torch_cuda)
    assert layer.kernel_launches > 0
    # determinism: a second call gives the same bits
    np.testing.assert_array_equal(layer.forward_host(x), out)
    layer.terminate()


def test_compressed_weight_file_loads_to_the_same_layer(torch_cuda, oracle, tmp_path):
    """initialize() reads the members of the npz with several threads into one page-locked arena; a deflated file
    (np.savez_compressed) and a stored one must give the same layer."""
    from infmoe_b200 import MoELayer, synth
    w = synth.scaled(synth.WORKLOADS["cpm2"], expert_count=12, embedding_size=128, hidden_size=384, batch=1, seq_len=200)
    x, c, ln = synth.gen_inputs(w)
    experts = [synth.gen_expert_numpy(w, e) for e in range(w.expert_count)]
    outs = []
    for compressed in (False, True):
        path = synth.write_npz(w, str(tmp_path / f"w{int(compressed)}.npz"), compressed=compressed)
        layer = MoELayer.create(w.expert_count, w.embedding_size, w.hidden_size, 2, c, path, "T5_FF", w.variant, ln)
        layer.initialize()
        outs.append(_check(layer, w, x, c, ln, experts, oracle, torch_cuda))
        layer.terminate()
    np.testing.assert_array_equal(outs[0], outs[1])


@pytest.mark.parametrize("name,kw", [
    ("cpm2", dict(expert_count=8, embedding_size=512, hidden_size=1024, batch=2, seq_len=300)),
    ("base_layer_zipf", dict(expert_count=16, embedding_size=256, hidden_size=512, batch=4, seq_len=256)),
    ("cpm2", dict(expert_count=40, embedding_size=128, hidden_size=256, batch=1, seq_len=64)),   # empty experts
    ("tiny_default", dict(expert_count=3, embedding_size=64, hidden_size=128, batch=1, seq_len=1)),   # one token
])
def test_scaled_workloads(torch_cuda, oracle, name, kw):
    from infmoe_b200 import synth
    w = synth.scaled(synth.WORKLOADS[name], **kw)
    layer, x, c, ln, experts = _build(w, synth, from_npz=False)
    _check(layer, w, x, c, ln, experts, oracle, torch_cuda)
    layer.terminate()


def test_all_tokens_to_one_expert(torch_cuda, oracle):
    from infmoe_b200 import synth
    w = synth.scaled(synth.WORKLOADS["tiny_default"], expert_count=5, embedding_size=128, hidden_size=256, batch=1,
                     seq_len=450)
    layer, x, c, ln, experts = _build(w, synth, from_npz=False)
    layer.terminate()
    from infmoe_b200 import MoELayer
    c = np.zeros_like(c)
    c[3] = 1.0
    x = np.abs(x)
    layer = MoELayer.create(5, 128, 256, 2, c, None, "T5_FF", "default", None)
    for e, ex in enumerate(experts):
        layer.set_expert(e, *ex)
    _check(layer, w, x, c, None, experts, oracle, torch_cuda)
    layer.terminate()


@pytest.mark.parametrize("mc", [1, 2, 3])
def test_streamed_experts_match_resident(torch_cuda, oracle, tmp_path, mc):
    """max_concurrency slots fed from pinned host memory give the same bits as resident weights
    (mc = 1 is broken in the reference, plugin/MoELayerPlugin.cc:375-393; here it is just serial)."""
    from infmoe_b200 import synth
    w = synth.scaled(synth.WORKLOADS["cpm2"], expert_count=6, embedding_size=128, hidden_size=256, batch=1, seq_len=90)
    res, x, c, ln, experts = _build(w, synth, tmp_path, residency=1)
    st, *_ = _build(w, synth, tmp_path, residency=0, mc=mc)
    a = _check(res, w, x, c, ln, experts, oracle, torch_cuda)
    b = _check(st, w, x, c, ln, experts, oracle, torch_cuda)
    np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(st.forward_host(x), b)     # slots are reusable across calls
    res.terminate()
    st.terminate()


@pytest.mark.parametrize("slots", [2, 3, 6])
def test_expert_cache_keeps_experts_across_calls(torch_cuda, oracle, tmp_path, slots):
    """Streamed mode with the layer's expert cache: same bits as resident weights whatever the cache size; with
    room for every expert the second call copies nothing; replaced weights are not served from the cache."""
    from infmoe_b200 import synth
    w = synth.scaled(synth.WORKLOADS["cpm2"], expert_count=6, embedding_size=128, hidden_size=256, batch=1, seq_len=90)
    res, x, c, ln, experts = _build(w, synth, tmp_path, residency=1)
    st, *_ = _build(w, synth, tmp_path, residency=0, mc=2)
    st.set_expert_cache(slots)
    want = _check(res, w, x, c, ln, experts, oracle, torch_cuda)
    per_expert = 3 * 4 * w.embedding_size * w.hidden_size
    got = st.forward_host(x)
    np.testing.assert_array_equal(got, want)
    first = st.weight_h2d_bytes()
    assert first == w.expert_count * per_expert            # every expert is routed to in this workload
    np.testing.assert_array_equal(st.forward_host(x), want)
    second = st.weight_h2d_bytes() - first
    if slots >= w.expert_count:
        assert second == 0
    else:
        assert 0 < second <= w.expert_count * per_expert
    # a permuted batch routes to the same experts: still nothing to copy when they all fit
    perm = np.random.default_rng(0).permutation(w.tokens)
    np.testing.assert_array_equal(st.forward_host(x[perm]), want[perm])
    if slots >= w.expert_count:
        assert st.weight_h2d_bytes() == first
    # new weights for expert 0 (those of expert 1): the cached copy must not be used
    st.set_expert(0, *experts[1])
    res.set_expert(0, *experts[1])
    before = st.weight_h2d_bytes()
    np.testing.assert_array_equal(st.forward_host(x), res.forward_host(x))
    assert st.weight_h2d_bytes() - before >= per_expert
    res.terminate()
    st.terminate()


@pytest.mark.parametrize("variant", ["cpm_2", "base_layer"])
def test_forward_host_into_page_locked_output(torch_cuda, oracle, variant):
    """A page-locked output buffer is written by the layer's last kernel directly; same bits as the copied path."""
    from infmoe_b200 import synth
    torch = torch_cuda
    w = synth.scaled(synth.WORKLOADS["cpm2"], variant=variant, expert_count=6, embedding_size=128, hidden_size=256,
                     batch=1, seq_len=200)
    layer, x, c, ln, experts = _build(w, synth, from_npz=False)
    want = _check(layer, w, x, c, ln, experts, oracle, torch)          # pageable numpy output
    hx = torch.from_numpy(x).pin_memory()
    hout = torch.full_like(hx, float("nan")).pin_memory()
    layer.forward_host_ptr(hx.data_ptr(), hout.data_ptr(), w.tokens)
    np.testing.assert_array_equal(hout.numpy(), want)
    layer.terminate()


@pytest.mark.parametrize("pinned,resident", [(True, True), (False, True), (True, False)])
def test_two_host_steps_in_flight_give_the_bits_of_the_blocking_call(torch_cuda, oracle, pinned, resident):
    """infmoe_layer_submit_host / _wait_host: step k brings the rows rolled by k, two steps in flight; page-locked
    buffers are written by the pass itself, pageable ones through a device buffer and a copy stream.  A NaN row is
    reported by the wait of its own step only."""
    from infmoe_b200 import capi, synth
    torch = torch_cuda
    w = synth.scaled(synth.WORKLOADS["cpm2"], variant="cpm_2", expert_count=6, embedding_size=128, hidden_size=256,
                     batch=1, seq_len=200)
    layer, x, c, ln, experts = _build(w, synth, from_npz=False)
    layer.set_residency(1 if resident else 0)          # streamed experts: every pass waits for its weight copies
    want = torch.from_numpy(_check(layer, w, x, c, ln, experts, oracle, torch))
    hx = torch.from_numpy(x)
    mem = (lambda t: t.pin_memory()) if pinned else (lambda t: t.clone())
    steps = 5
    ins = [mem(torch.roll(hx, k, 0).contiguous()) for k in range(steps)]
    if resident:    # (a streamed pass waits for its weight copies on the host and reports such a token from submit)
        ins[3][7, :] = float("nan")                               # step 3 has a token without an expert
    outs = [mem(torch.full_like(hx, float("nan"))) for _ in range(steps)]
    status = []
    for k in range(steps):
        layer.submit_host_ptr(ins[k].data_ptr(), outs[k].data_ptr(), w.tokens)
        if k >= 1:
            try:
                layer.wait_host()
                status.append(0)
            except capi.InfMoEError as e:
                status.append(e.status)
    with pytest.raises(capi.InfMoEError):                         # the blocking call is refused while a step is in flight
        layer.forward_host_ptr(ins[0].data_ptr(), outs[0].data_ptr(), w.tokens)
    layer.wait_host()
    status.append(0)
    with pytest.raises(capi.InfMoEError):                         # nothing left to wait for
        layer.wait_host()
    assert status == ([0, 0, 0, 3, 0] if resident else [0] * 5)
    for k in range(steps):
        got, exp = outs[k], torch.roll(want, k, 0)
        if k == 3 and resident:                                   # the NaN token's row is left alone
            keep = torch.ones(w.tokens, dtype=torch.bool)
            keep[7] = False
            got, exp = got[keep], exp[keep]
        assert torch.equal(got, exp), k
    layer.terminate()


def test_bounded_wait_runs_out_and_leaves_the_context_usable(torch_cuda, oracle, tmp_path):
    """The wait every role of the expert GEMM uses, pointed at a barrier nothing completes, with a 50 ms limit:
    it gives up, raises the status bit and returns; the next layer call on the same context works."""
    import ctypes

    from infmoe_b200 import capi, synth
    timed_out, waited = ctypes.c_int32(0), ctypes.c_float(0)
    capi.check(capi.lib().infmoe_wait_timeout_probe(50, ctypes.byref(timed_out), ctypes.byref(waited)))
    assert timed_out.value == 1
    assert 50.0 <= waited.value < 200.0
    w = synth.scaled(synth.WORKLOADS["tiny_default"], variant="cpm_2")
    layer, x, c, ln, experts = _build(w, synth, tmp_path)
    _check(layer, w, x, c, ln, experts, oracle, torch_cuda)
    layer.terminate()


@pytest.mark.parametrize("variant,path", [("cpm_2", ""), ("base_layer", ""), ("base_layer", "simt")])
def test_expert_forward_scatter_writes_rows_to_given_addresses(torch_cuda, oracle, monkeypatch, variant, path):
    """The expert-parallel building block: rows with known experts, each result written to its own address
    (here: a permutation of the rows of a local tensor), optionally with the base_layer mix."""
    from infmoe_b200 import synth
    torch = torch_cuda
    if path:
        monkeypatch.setenv("INFMOE_FFN", path)
    w = synth.scaled(synth.WORKLOADS["cpm2"], variant=variant, expert_count=6, embedding_size=128, hidden_size=256,
                     batch=1, seq_len=300)
    layer, x, c, ln, experts = _build(w, synth, from_npz=False)
    rng = np.random.default_rng(5)
    n, D = w.tokens, w.embedding_size
    expert_of_row = torch.from_numpy(rng.integers(0, w.expert_count, n).astype(np.int32)).cuda()
    rows = torch.from_numpy(x).cuda()
    want = layer.expert_forward(rows, expert_of_row)            # rows in, rows out, same order
    perm = torch.from_numpy(rng.permutation(n)).cuda()
    out = torch.full((n, D), float("nan"), device="cuda")
    dst = out.data_ptr() + perm.to(torch.int64) * (D * 4)
    score = None
    if variant == "base_layer":
        score = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
        alpha = torch.sigmoid(score.double())[:, None]
        want = (alpha * want.double() + (1 - alpha) * rows.double()).float()
    layer.expert_forward_scatter(rows, expert_of_row, dst.contiguous(), score)
    layer.sync_status()
    got = out[perm]
    if variant == "base_layer":
        torch.testing.assert_close(got, want, rtol=2e-6, atol=2e-6)
    else:
        assert torch.equal(got, want)
    layer.terminate()


def test_exact_path_matches_tensor_core_path(torch_cuda, oracle, monkeypatch):
    from infmoe_b200 import synth
    w = synth.scaled(synth.WORKLOADS["base_layer_zipf"], expert_count=8, embedding_size=128, hidden_size=256, batch=2,
                     seq_len=200)
    layer, x, c, ln, experts = _build(w, synth, from_npz=False)
    a = layer.forward_host(x)
    layer.terminate()
    monkeypatch.setenv("INFMOE_FFN", "simt")
    layer, *_ = _build(w, synth, from_npz=False)
    b = layer.forward_host(x)
    layer.terminate()
    assert oracle.rel_l2(a, b) < 2e-6


def test_identity_sublayer_returns_input(torch_cuda):
    from infmoe_b200 import MoELayer
    rng = np.random.default_rng(0)
    x = rng.standard_normal((70, 32)).astype(np.float32)
    c = rng.standard_normal((4, 32)).astype(np.float32)
    layer = MoELayer.create(4, 32, 64, 2, c, None, "Identity", "default", None)
    np.testing.assert_array_equal(layer.forward_host(x), x)
    layer.terminate()


@pytest.mark.parametrize("variant", ["default", "base_layer"])
def test_registered_sublayer_is_driven_like_the_built_in_ones(torch_cuda, oracle, variant):
    """A sublayer type registered through the C ABI (the reference's extension point is a class derived from
    MoESubLayer, plugin/sublayers/SubLayer.h:18-48): expert e scales its rows by a weight that the layer fetches
    into one of max_concurrency device slots before every run.  Routing, dispatch and combine are the layer's."""
    import ctypes
    from infmoe_b200 import MoELayer, capi
    torch = torch_cuda
    E, D, T, mc = 7, 96, 333, 2
    rng = np.random.default_rng(9)
    x = rng.standard_normal((T, D)).astype(np.float32)
    c = (rng.standard_normal((E, D)) * 0.1).astype(np.float32)
    scales = np.arange(E, dtype=np.float32) + 2.0
    # The fetch goes through the CUDA runtime directly: a torch copy from page-locked memory would make torch's host
    # allocator remember the layer's copy stream, which no longer exists when the test's tensors are freed.
    cudart = ctypes.CDLL("libcudart.so.12")
    cudart.cudaMemcpyAsync.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int, ctypes.c_void_p]
    calls = {"init": 0, "copy": [], "run": []}

    def tensor_at(ptr, n):
        class V:
            __cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (int(ptr), False), "version": 2}
        return torch.as_tensor(V(), device="cuda")

    def initialize(user, e, d, f, path):
        calls["init"] += 1
        return 0 if (e, d) == (E, D) else 1

    def copy_weights(user, dst, expert, stream):
        calls["copy"].append(int(expert))
        return cudart.cudaMemcpyAsync(dst, scales[expert:expert + 1].ctypes.data, 4, 1, stream)   # 1: host to device

    def run(user, expert, n, weights, src, dst, ws, stream):
        calls["run"].append((int(expert), int(n)))
        with torch.cuda.stream(torch.cuda.ExternalStream(int(stream or 0))):
            torch.mul(tensor_at(src, n * D), tensor_at(weights, 1), out=tensor_at(dst, n * D))
        return 0

    vt = capi.SublayerVtable(None, capi.SUB_INIT_FN(initialize), capi.SUB_WEIGHT_SIZE_FN(lambda user: 4),
                             capi.SUB_WS_SIZE_FN(lambda user, n: 0), capi.SUB_COPY_FN(copy_weights), capi.SUB_RUN_FN(run))
    capi.check(capi.lib().infmoe_register_sublayer(b"ScaleByExpert", ctypes.byref(vt)))
    layer = MoELayer.create(E, D, 4 * D, mc, c, None, "ScaleByExpert", variant, None)
    with pytest.raises(capi.InfMoEError):
        layer.forward_host(x)                       # not initialized yet
    layer.initialize()
    out = layer.forward_host(x)
    gate, score = oracle.route(x, c, None)
    want = x * (gate[:, None].astype(np.float32) + 2.0)
    if variant == "base_layer":
        alpha = (1.0 / (1.0 + np.exp(-score.astype(np.float64))))[:, None]
        want = alpha * want + (1 - alpha) * x
    np.testing.assert_allclose(out, want, rtol=2e-6, atol=1e-6)
    active = sorted(set(int(e) for e in gate))
    assert calls["init"] == 1 and calls["copy"] == active
    assert calls["run"] == [(e, int(np.count_nonzero(gate == e))) for e in active]
    layer.terminate()
    with pytest.raises(capi.InfMoEError):
        MoELayer.create(E, D, 4 * D, mc, c, None, "NoSuchSublayer", variant, None)


def test_nan_input_is_reported_not_trapped(torch_cuda):
    from infmoe_b200 import MoELayer, capi, synth
    w = synth.scaled(synth.WORKLOADS["tiny_default"])
    layer, x, c, ln, experts = _build(w, synth, from_npz=False)
    bad = x.copy()
    bad[3, :] = np.nan
    with pytest.raises(capi.InfMoEError) as e:
        layer.forward_host(bad)
    assert e.value.status == 3
    layer.forward_host(x)            # the context is still usable and the status was cleared
    layer.terminate()


@pytest.mark.parametrize("variant", ["cpm_2", "base_layer"])
def test_nan_tokens_touch_nothing_outside_their_own_rows(torch_cuda, oracle, variant):
    """A workspace is not zeroed between calls (TensorRT hands out the same block again and again).  With a few
    NaN rows in the input the call must report them, leave their output rows alone, and still give every other
    token its expert's result: no stage may index anything with what a previous call left in the workspace."""
    from infmoe_b200 import capi, synth
    torch = torch_cuda
    w = synth.scaled(synth.WORKLOADS["cpm2"], variant=variant, expert_count=6, embedding_size=128, hidden_size=256,
                     batch=1, seq_len=500)
    layer, x, c, ln, experts = _build(w, synth, from_npz=False)
    layer.set_residency(1)
    T, D = w.tokens, w.embedding_size
    need = layer.get_workspace_size(T)
    ws = torch.full((need,), 0x7f, dtype=torch.uint8, device="cuda")      # garbage indices everywhere
    bad_rows = np.array([0, 17, 255, 256, 499])
    bad = x.copy()
    bad[bad_rows, 5] = np.nan
    dx = torch.from_numpy(bad).cuda()
    out = torch.full((T, D), -7.0, device="cuda")
    layer.enqueue(dx.data_ptr(), out.data_ptr(), ws.data_ptr(), need, T, torch.cuda.current_stream().cuda_stream)
    with pytest.raises(capi.InfMoEError) as e:
        layer.sync_status(torch.cuda.current_stream().cuda_stream)
    assert e.value.status == 3
    got = out.cpu().numpy()
    assert np.all(got[bad_rows] == -7.0)                                  # untouched
    good = np.setdiff1d(np.arange(T), bad_rows)
    ref = oracle.layer_forward_f32(x[good], w.variant, c, ln, experts)
    o64 = oracle.layer_forward_f64(x[good], w.variant, ref["gate"], ref["score"], experts)
    assert oracle.rel_l2(got[good], o64) <= TOL
    gate, _, pos, count, offset = _routing(layer, T, w.expert_count, torch)
    assert np.all(gate[bad_rows] == -1) and offset[-1] == T - bad_rows.size
    np.testing.assert_array_equal(pos[offset[-1]:], bad_rows)
    layer.terminate()


@pytest.mark.parametrize("variant", ["cpm_2", "base_layer"])
def test_deserialised_layer_gives_the_same_bits(torch_cuda, oracle, tmp_path, variant):
    """serialize -> deserialize -> initialize -> enqueue (the deserialising constructor of the reference,
    plugin/MoELayerPlugin.cc:104-143, fed by serialize, :425-458) equals the layer the blob came from."""
    from infmoe_b200 import MoELayer, synth
    w = synth.scaled(synth.WORKLOADS["cpm2"], variant=variant, expert_count=6, embedding_size=128, hidden_size=256,
                     batch=2, seq_len=150)
    layer, x, c, ln, experts = _build(w, synth, tmp_path)
    want = _check(layer, w, x, c, ln, experts, oracle, torch_cuda)
    blob = layer.serialize()
    layer.terminate()
    twin = MoELayer.deserialize(blob)
    assert twin.moe_variant == variant and twin.expert_count == 6
    twin.initialize()                       # reads the weight file named in the blob
    got = _check(twin, w, x, c, ln, experts, oracle, torch_cuda)
    np.testing.assert_array_equal(got, want)
    clone = twin.clone()                    # TensorRT runs clones of the deserialised plugin
    np.testing.assert_array_equal(clone.forward_host(x), want)
    clone.terminate()
    twin.terminate()


def test_clones_on_two_streams_share_one_upload(torch_cuda, oracle, tmp_path):
    """Clones share the expert store; TensorRT gives each execution context its own clone and stream.  The first
    enqueue uploads the weights on its stream; a clone whose first enqueue overlaps it on another stream must
    wait for that upload instead of reading half-written planes."""
    from infmoe_b200 import synth
    torch = torch_cuda
    w = synth.scaled(synth.WORKLOADS["cpm2"], expert_count=8, embedding_size=512, hidden_size=2048, batch=1,
                     seq_len=400)
    layer, x, c, ln, experts = _build(w, synth, tmp_path, residency=1)
    clone = layer.clone()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    dx = torch.from_numpy(x).cuda()
    o1, o2 = torch.empty_like(dx), torch.empty_like(dx)
    torch.cuda.synchronize()
    layer.forward(dx, o1, stream=s1.cuda_stream)      # queues 8 x (3 copies + 2 retile kernels) and returns at once
    clone.forward(dx, o2, stream=s2.cuda_stream)      # sees the experts marked resident
    torch.cuda.synchronize()
    ref = oracle.layer_forward_f32(x, w.variant, c, ln, experts)
    o64 = oracle.layer_forward_f64(x, w.variant, ref["gate"], ref["score"], experts)
    assert oracle.rel_l2(o1.cpu().numpy(), o64) <= TOL
    assert torch.equal(o1, o2)
    clone.terminate()
    layer.terminate()


def test_enqueue_argument_checks(torch_cuda):
    from infmoe_b200 import MoELayer, capi, synth
    torch = torch_cuda
    w = synth.WORKLOADS["tiny_default"]
    layer, x, c, ln, experts = _build(w, synth, from_npz=False)
    dx = torch.from_numpy(x).cuda()
    ws = torch.empty(1024, dtype=torch.uint8, device="cuda")
    with pytest.raises(capi.InfMoEError) as e:
        layer.enqueue(dx.data_ptr(), dx.data_ptr(), ws.data_ptr(), 1024, w.tokens)
    assert "alias" in str(e.value)
    out = torch.empty_like(dx)
    with pytest.raises(capi.InfMoEError) as e:
        layer.enqueue(dx.data_ptr(), out.data_ptr(), ws.data_ptr(), 1024, w.tokens)
    assert "workspace" in str(e.value)
    y = layer.forward(dx)
    layer.sync_status()
    np.testing.assert_array_equal(y.cpu().numpy(), layer.forward_host(x))
    layer.terminate()
    empty = MoELayer.create(2, 8, 16, 2, np.zeros((2, 8), np.float32), None, "T5_FF", "default", None)
    with pytest.raises(capi.InfMoEError) as e:
        empty.forward_host(np.zeros((2, 8), np.float32))
    assert e.value.status == 8


# (tokens, d_model, d_ff) of one expert.  infmoe_t5ff_run never cuts a tile; the layer does when the last round of tiles
# leaves enough SMs idle: few long tiles (several CTAs to a tile), a K that ends inside a chunk of 256 and inside a block
# of 32, token tiles of 16, 64 and two of 112 columns, and a tail behind whole rounds.
@pytest.mark.parametrize("T,D,F", [(1, 4096, 512), (16, 2048, 4096), (5, 600, 2724), (64, 1032, 3000), (210, 1000, 2724),
                                   (300, 1024, 9600)])
def test_tiles_cut_along_k_have_the_bits_of_uncut_ones(oracle, T, D, F):
    import torch
    from infmoe_b200 import MoELayer
    from tests import gpu_util as g
    rng = np.random.default_rng(T + D + F)
    x = rng.standard_normal((T, D)).astype(np.float32)
    ln = (1 + 0.01 * rng.standard_normal(D)).astype(np.float32)
    wi0, wi1 = ((rng.standard_normal((F, D)) / np.sqrt(D)).astype(np.float32) for _ in range(2))
    wo = (rng.standard_normal((D, F)) / np.sqrt(F)).astype(np.float32)
    layer = MoELayer.create(1, D, F, 2, np.ones((1, D), np.float32), None, "T5_FF", "default", None)
    layer.set_expert(0, *(torch.from_numpy(a).cuda() for a in (ln, wi0, wi1, wo)))
    got = [layer.forward(torch.from_numpy(x).cuda()).cpu().numpy() for _ in range(3)]
    layer.sync_status()
    layer.terminate()
    want = g.t5ff_run(x, ln, wi0, wi1, wo)
    for out in got:                                # also again: the counters of the cut tiles are back at zero
        np.testing.assert_array_equal(out, want)
    assert oracle.rel_l2(want[:4], oracle.expert_ffn_f64(x[:4], ln, wi0, wi1, wo)) <= TOL


# CUDA-core GEMM: experts with 0, 1, 15 .. 17 and 63 .. 65 rows (its tiles are 16 rows high when the experts have at most
# 16 on average, else 64), widths inside, at and past a block of 32 and a 128-row weight block.
@pytest.mark.parametrize("counts", [(1, 0, 15, 16, 17), (63, 64, 65, 0, 1, 130)])
@pytest.mark.parametrize("D,F", [(510, 1022), (33, 63), (6, 5), (129, 257)])
def test_cuda_core_experts_against_oracle(oracle, counts, D, F):
    import torch
    from infmoe_b200 import MoELayer
    rng = np.random.default_rng(D + F + len(counts))
    E, n = len(counts), sum(counts)
    layer = MoELayer.create(E, D, F, 2, np.ones((E, D), np.float32), None, "T5_FF", "default", None)
    experts = []
    for e in range(E):
        experts.append([(1 + 0.01 * rng.standard_normal(D)).astype(np.float32)] +
                       [(rng.standard_normal((F, D)) / np.sqrt(D)).astype(np.float32) for _ in range(2)] +
                       [(rng.standard_normal((D, F)) / np.sqrt(F)).astype(np.float32)])
        layer.set_expert(e, *(torch.from_numpy(a).cuda() for a in experts[e]))
    gate = rng.permutation(np.repeat(np.arange(E, dtype=np.int32), counts))
    x = rng.standard_normal((n, D)).astype(np.float32)
    out = layer.expert_forward(torch.from_numpy(x).cuda(), torch.from_numpy(gate).cuda()).cpu().numpy()
    layer.sync_status()
    layer.terminate()
    for e in range(E):
        rows = gate == e
        if rows.any():
            want = oracle.expert_ffn_f64(x[rows], *experts[e])
            assert oracle.rel_l2(out[rows] - x[rows], want - x[rows]) <= 2e-6   # FP32 chains of up to 1022 adds


# A row's outputs are summed over one, two or four CTAs that share the k blocks, by K alone: the edges between them (96 | 97,
# 224 | 225 values), and the same rows in calls with 16-row and 64-row tiles have the same bits.
@pytest.mark.parametrize("D,F", [(95, 97), (225, 223), (97, 226), (450, 161)])
def test_cuda_core_experts_with_k_shared_by_a_cluster(oracle, D, F):
    import torch
    from infmoe_b200 import MoELayer
    rng = np.random.default_rng(D * F)
    layer = MoELayer.create(1, D, F, 2, np.ones((1, D), np.float32), None, "T5_FF", "default", None)
    expert = [(1 + 0.01 * rng.standard_normal(D)).astype(np.float32)] + \
             [(rng.standard_normal((F, D)) / np.sqrt(D)).astype(np.float32) for _ in range(2)] + \
             [(rng.standard_normal((D, F)) / np.sqrt(F)).astype(np.float32)]
    layer.set_expert(0, *(torch.from_numpy(a).cuda() for a in expert))
    x = rng.standard_normal((130, D)).astype(np.float32)
    run = lambda n: layer.expert_forward(torch.from_numpy(x[:n]).cuda(),
                                         torch.zeros(n, dtype=torch.int32, device="cuda")).cpu().numpy()
    out, few = run(130), run(16)
    layer.sync_status()
    layer.terminate()
    np.testing.assert_array_equal(few, out[:16])
    want = oracle.expert_ffn_f64(x, *expert)
    assert oracle.rel_l2(out - x, want - x) <= 2e-6     # FP32 chains of up to 450 adds


# Up to 1024 tokens one kernel computes the dispatch metadata and scatters, unless d_model > 6016; up to 4096 another one does for
# aligned rows of up to 2048 floats on the tensor-core path (more of its lines below); else two kernels do.
@pytest.mark.parametrize("T,D,E,variant", [(1, 64, 4, "default"), (33, 66, 3, "base_layer"), (1023, 36, 70, "cpm_2"),
                                           (1024, 40, 5, "base_layer"), (1025, 40, 5, "base_layer"),
                                           (7, 6016, 2, "default"), (7, 6020, 2, "default"), (129, 130, 33, "default")])
def test_few_and_many_tokens_dispatch_alike(oracle, T, D, E, variant):
    import torch
    from infmoe_b200 import MoELayer
    from infmoe_b200.devmem import read_device
    F = 40
    rng = np.random.default_rng(T + D + E)
    c = (rng.standard_normal((E, D)) * 0.02).astype(np.float32)
    ln = (1 + 0.01 * rng.standard_normal(D)).astype(np.float32) if variant == "cpm_2" else None
    experts = [[(1 + 0.01 * rng.standard_normal(D)).astype(np.float32)] +
               [(rng.standard_normal((F, D)) / np.sqrt(D)).astype(np.float32) for _ in range(2)] +
               [(rng.standard_normal((D, F)) / np.sqrt(F)).astype(np.float32)] for _ in range(E)]
    x = rng.standard_normal((T, D)).astype(np.float32)
    layer = MoELayer.create(E, D, F, 2, c, None, "T5_FF", variant, ln)
    for e, ex in enumerate(experts):
        layer.set_expert(e, *(torch.from_numpy(a).cuda() for a in ex))
    out = layer.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    layer.sync_status()
    gate_p, _, pos_p, count_p, offset_p = layer.last_routing()
    gate, score = oracle.route(x, c, ln)
    count, offset, pos = oracle.dispatch(gate, E)
    np.testing.assert_array_equal(read_device(gate_p, T, np.int32), gate)
    np.testing.assert_array_equal(read_device(pos_p, T, np.int32), pos)
    np.testing.assert_array_equal(read_device(count_p, E, np.int32), count)
    np.testing.assert_array_equal(read_device(offset_p, E + 1, np.int32), offset)
    assert oracle.rel_l2(out, oracle.layer_forward_f64(x, variant, gate, score, experts)) <= TOL
    # the experts alone, every seventh token without one: its row stays as it was
    bad = gate.copy()
    bad[::7] = -1
    keep = torch.full((T, D), -7.0, device="cuda")
    layer.expert_forward(torch.from_numpy(x).cuda(), torch.from_numpy(bad).cuda(), out=keep)
    with pytest.raises(Exception):
        layer.sync_status()
    keep = keep.cpu().numpy()
    assert np.all(keep[::7] == -7.0)
    good = bad >= 0
    if good.any() and variant != "base_layer":
        np.testing.assert_array_equal(keep[good], out[good])
    layer.terminate()


def test_pass_under_capture_between_other_kernels():
    """Kernels of a pass start before their predecessors have ended; their reads and writes still follow them: the
    input is filled by the kernel before the pass and the output overwritten by the one after it, eagerly and in a graph."""
    import torch
    from infmoe_b200 import MoELayer
    g = torch.Generator(device="cuda").manual_seed(3)
    E, D, F = 4, 256, 512
    layer = MoELayer.create(E, D, F, 2, torch.randn(E, D, generator=g, device="cuda").cpu().numpy(), None, "T5_FF",
                            "default", None)
    for e in range(E):
        layer.set_expert(e, torch.ones(D, device="cuda"), torch.randn(F, D, generator=g, device="cuda") / 16,
                         torch.randn(F, D, generator=g, device="cuda") / 16, torch.randn(D, F, generator=g, device="cuda") / 22)
    for T in (3, 1500):
        src = torch.randn(4, T, D, generator=g, device="cuda")
        want = [layer.forward(src[i].contiguous()).clone() for i in range(4)]
        torch.cuda.synchronize()
        x, out, acc = torch.zeros(T, D, device="cuda"), torch.zeros(T, D, device="cuda"), torch.zeros(T, D, device="cuda")
        side = torch.cuda.Stream()
        graph = torch.cuda.CUDAGraph()

        def step(i):
            x.copy_(src[i] * 1.0)
            layer.forward(x, out)
            acc.add_(out)
            out.fill_(-1.0)
            x.fill_(5.0)

        with torch.cuda.stream(side):
            for _ in range(3):
                acc.zero_()
                for i in range(4):
                    step(i)
        side.synchronize()
        ref = torch.zeros(T, D, device="cuda")
        for w in want:
            ref.add_(w)
        assert torch.equal(acc, ref)
        with torch.cuda.graph(graph, stream=side):
            acc.zero_()
            for i in range(4):
                step(i)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(acc, ref)
    layer.sync_status()
    layer.terminate()


# Second GEMM (K = d_ff >= 2048) and first GEMM (K = d_model >= 2048) on pairs of CTAs: an odd number of 128-row weight
# blocks (the pair's second CTA has nothing to write), token tiles of 32, 64 and 192 columns with remainders, experts
# without tokens, and the K just below the line.
@pytest.mark.parametrize("D,F", [(640, 2048), (2048, 192), (132, 2044), (2080, 2080)])
def test_paired_tiles_against_oracle(oracle, D, F):
    import torch
    from infmoe_b200 import MoELayer
    counts = (0, 1, 31, 33, 192, 193, 0, 70)
    rng = np.random.default_rng(D + F)
    E, n = len(counts), sum(counts)
    layer = MoELayer.create(E, D, F, 2, np.ones((E, D), np.float32), None, "T5_FF", "default", None)
    experts = []
    for e in range(E):
        experts.append([(1 + 0.01 * rng.standard_normal(D)).astype(np.float32)] +
                       [(rng.standard_normal((F, D)) / np.sqrt(D)).astype(np.float32) for _ in range(2)] +
                       [(rng.standard_normal((D, F)) / np.sqrt(F)).astype(np.float32)])
        layer.set_expert(e, *(torch.from_numpy(a).cuda() for a in experts[e]))
    gate = rng.permutation(np.repeat(np.arange(E, dtype=np.int32), counts))
    x = rng.standard_normal((n, D)).astype(np.float32)
    dx, dg = torch.from_numpy(x).cuda(), torch.from_numpy(gate).cuda()
    out = [layer.expert_forward(dx, dg).cpu().numpy() for _ in range(3)]
    layer.sync_status()
    # the same rows among fewer: one CTA per tile, 64 columns, with the same additions
    few = np.sort(rng.choice(n, 60, replace=False))
    alone = layer.expert_forward(dx[few].contiguous(), dg[few].contiguous()).cpu().numpy()
    layer.sync_status()
    layer.terminate()
    np.testing.assert_array_equal(out[1], out[0])
    np.testing.assert_array_equal(out[2], out[0])
    np.testing.assert_array_equal(alone, out[0][few])
    for e in range(E):
        rows = np.flatnonzero(gate == e)[:24]
        if rows.size:
            want = oracle.expert_ffn_f64(x[rows], *experts[e])
            assert oracle.rel_l2(out[0][rows], want) <= TOL


# From 1025 to 4096 tokens of aligned rows of up to 2048 floats one kernel computes the dispatch metadata and scatters, eight
# tokens to a block: its lines, a last block of one and of seven tokens, rows that end inside a register and one expert.
@pytest.mark.parametrize("T,D,E,variant", [(1025, 36, 1, "default"), (1031, 1024, 70, "cpm_2"), (2063, 1028, 9, "default"),
                                           (4095, 132, 33, "base_layer"), (4096, 2048, 5, "cpm_2"), (4097, 132, 5, "default"),
                                           (1100, 2052, 6, "default")])
def test_dispatch_of_a_few_thousand_tokens_alike(oracle, T, D, E, variant):
    test_few_and_many_tokens_dispatch_alike(oracle, T, D, E, variant)


# A tile's columns are shared out evenly over four warps per row quarter, 4 to 48 columns each: every width from 16 to 192,
# full and with one token less, tiles of one CTA (K < 2048) and of two.
@pytest.mark.parametrize("D,F", [(260, 516), (2052, 132)])
def test_token_tiles_of_every_width(oracle, D, F):
    import torch
    from infmoe_b200 import MoELayer
    counts = tuple(range(16, 193, 16)) + tuple(range(15, 192, 16))
    rng = np.random.default_rng(D)
    E, n = len(counts), sum(counts)
    layer = MoELayer.create(E, D, F, 2, np.ones((E, D), np.float32), None, "T5_FF", "default", None)
    expert = [(1 + 0.01 * rng.standard_normal(D)).astype(np.float32)] + \
             [(rng.standard_normal((F, D)) / np.sqrt(D)).astype(np.float32) for _ in range(2)] + \
             [(rng.standard_normal((D, F)) / np.sqrt(F)).astype(np.float32)]
    for e in range(E):
        layer.set_expert(e, *(torch.from_numpy(a).cuda() for a in expert))
    gate = torch.from_numpy(rng.permutation(np.repeat(np.arange(E, dtype=np.int32), counts))).cuda()
    x = rng.standard_normal((n, D)).astype(np.float32)
    dx = torch.from_numpy(x).cuda()
    out = layer.expert_forward(dx, gate).cpu().numpy()
    # the same rows, all experts being alike, in one expert's tiles of 192 columns
    same = layer.expert_forward(dx, torch.zeros_like(gate)).cpu().numpy()
    layer.sync_status()
    layer.terminate()
    np.testing.assert_array_equal(same, out)
    assert oracle.rel_l2(out[:64] - x[:64], oracle.expert_ffn_f64(x[:64], *expert) - x[:64]) <= TOL


# Odd widths take the CUDA-core path, where two kernels dispatch and scatter from 1025 tokens on.
def test_dispatch_of_a_few_thousand_tokens_of_odd_width_alike(oracle):
    test_few_and_many_tokens_dispatch_alike(oracle, 1025, 42, 5, "cpm_2")
    test_few_and_many_tokens_dispatch_alike(oracle, 1025, 41, 5, "base_layer")


# Tokens that start one float past an aligned address: no wide loads, and from 1025 on two kernels; the same additions either way.
@pytest.mark.parametrize("T", [33, 1024, 1025, 4097])
@pytest.mark.parametrize("variant", ["cpm_2", "base_layer"])
def test_unaligned_tokens_have_the_bits_of_aligned_ones(T, variant):
    import torch
    from infmoe_b200 import MoELayer
    E, D, F = 5, 40, 44
    g = torch.Generator(device="cuda").manual_seed(T)
    ln = np.linspace(0.9, 1.1, D, dtype=np.float32) if variant == "cpm_2" else None
    layer = MoELayer.create(E, D, F, 2, torch.randn(E, D, generator=g, device="cuda").cpu().numpy(), None, "T5_FF", variant, ln)
    for e in range(E):
        layer.set_expert(e, torch.ones(D, device="cuda"), torch.randn(F, D, generator=g, device="cuda") / 6,
                         torch.randn(F, D, generator=g, device="cuda") / 6, torch.randn(D, F, generator=g, device="cuda") / 6)
    x = torch.randn(T, D, generator=g, device="cuda")
    shifted = torch.empty(T * D + 1, device="cuda")[1:].view(T, D)
    shifted.copy_(x)
    assert x.data_ptr() % 16 == 0 and shifted.data_ptr() % 16 == 4
    want, got = layer.forward(x), layer.forward(shifted)
    layer.sync_status()
    assert torch.equal(got, want)
    layer.terminate()


# Passes behind and in front of other kernels, one form of a pass each: separate dispatch and scatter for many tokens and for long
# rows (pairs of CTAs), the CUDA-core path, LayerNorm weights and centroids that are read early, the mix.  Every step routes
# differently, so that counts, positions or gates that an earlier step left in the workspace would show.
@pytest.mark.parametrize("T,D,E,F,variant", [(4200, 256, 4, 512, "default"), (1500, 2052, 4, 132, "default"),
                                             (300, 254, 4, 510, "cpm_2"), (1100, 130, 4, 66, "base_layer"), (5, 4096, 20, 64, "cpm_2"),
                                             (600, 512, 6, 256, "cpm_2"), (2500, 256, 4, 512, "base_layer"), (16384, 64, 8, 64, "cpm_2")])
def test_steps_that_route_differently_between_other_kernels(T, D, E, F, variant):
    import torch
    from infmoe_b200 import MoELayer
    g = torch.Generator(device="cuda").manual_seed(T + D)
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    centroids = normal(E, D)
    layer = MoELayer.create(E, D, F, 2, centroids.cpu().numpy(), None, "T5_FF", variant,
                            np.linspace(0.9, 1.1, D, dtype=np.float32) if variant == "cpm_2" else None)
    for e in range(E):
        layer.set_expert(e, 1 + normal(D) / 100, normal(F, D) / D ** 0.5, normal(F, D) / D ** 0.5, normal(D, F) / F ** 0.5)
    # step i draws most of its tokens to expert i
    src = torch.stack([normal(T, D) + (torch.rand(T, 1, generator=g, device="cuda") < 0.2 + 0.2 * i) * centroids[i % E] for i in range(4)])
    want = []
    for i in range(4):
        want.append(layer.forward(src[i].contiguous()).clone())
        layer.sync_status()
    ref = torch.zeros(T, D, device="cuda")
    for w in want:
        ref.add_(w)
    torch.cuda.synchronize()
    x, out, acc = (torch.zeros(T, D, device="cuda") for _ in range(3))
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()

    def steps():
        acc.zero_()
        for i in range(4):
            x.copy_(src[i] * 1.0)
            layer.forward(x, out)
            acc.add_(out)
            out.fill_(-1.0)
            x.fill_(5.0)

    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        steps()
        steps()
    side.synchronize()
    assert torch.equal(acc, ref)
    with torch.cuda.graph(graph, stream=side):
        steps()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(acc, ref)
    layer.sync_status()
    layer.terminate()


# The GEMMs fetch weights before their wait.  Experts are replaced on the device between passes of another stream that are issued
# without a wait of the host: each pass has the results of a layer that only ever had its weights.
@pytest.mark.parametrize("T", [3, 700, 4200])
def test_experts_replaced_between_passes_of_another_stream(T):
    import torch
    from infmoe_b200 import MoELayer
    E, D, F = 3, 256, 512
    g = torch.Generator(device="cuda").manual_seed(T)
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    centroids = normal(E, D).cpu().numpy()
    sets = [[(1 + normal(D) / 100, normal(F, D) / 16, normal(F, D) / 16, normal(D, F) / 22) for _ in range(E)] for _ in range(4)]
    x = normal(T, D)

    def make(experts):
        layer = MoELayer.create(E, D, F, 2, centroids, None, "T5_FF", "default", None)
        for e in range(E):
            layer.set_expert(e, *experts[e])
        return layer

    want = []
    for experts in sets:
        layer = make(experts)
        want.append(layer.forward(x))
        layer.sync_status()
        layer.terminate()
    layer = make(sets[0])
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    outs = [torch.empty_like(x) for _ in sets]
    for i in range(len(sets)):
        with torch.cuda.stream(side):
            layer.forward(x, outs[i])
        torch.cuda.current_stream().wait_stream(side)      # the replacement runs on the default stream
        if i + 1 < len(sets):
            for e in range(E):
                layer.set_expert(e, *sets[i + 1][e])
    torch.cuda.synchronize()
    layer.sync_status()
    layer.terminate()
    for got, w in zip(outs, want):
        assert torch.equal(got, w)


# Many rows: one CTA per tile, which takes the parts of the k blocks one after the other, instead of a cluster that shares them out.
# Row counts on both sides of the lines (parts of up to three k blocks, longer ones, a single one; either GEMM), the last ones with
# 16-row tiles; the bits are those of the same rows in a call of 16.
@pytest.mark.parametrize("D,F,E,T", [(66, 34, 1, 700), (130, 258, 1, 1087), (130, 258, 1, 1088), (161, 450, 1, 15807), (161, 450, 1, 15808),
                                     (450, 161, 1, 7935), (450, 161, 1, 7936), (1030, 33, 1, 3200), (510, 1022, 6, 2500),
                                     (130, 320, 64, 1024), (322, 130, 64, 1024), (510, 70, 64, 1000)])
def test_cuda_core_experts_of_one_cta_per_tile(oracle, D, F, E, T):
    import torch
    from infmoe_b200 import MoELayer
    rng = np.random.default_rng(D * F + T)
    layer = MoELayer.create(E, D, F, 2, np.ones((E, D), np.float32), None, "T5_FF", "default", None)
    expert = [(1 + 0.01 * rng.standard_normal(D)).astype(np.float32)] + \
             [(rng.standard_normal((F, D)) / np.sqrt(D)).astype(np.float32) for _ in range(2)] + \
             [(rng.standard_normal((D, F)) / np.sqrt(F)).astype(np.float32)]
    for e in range(E):
        layer.set_expert(e, *(torch.from_numpy(a).cuda() for a in expert))
    x = torch.from_numpy(rng.standard_normal((T, D)).astype(np.float32)).cuda()
    gate = torch.from_numpy(rng.integers(0, E, T).astype(np.int32)).cuda()
    score = torch.from_numpy(rng.standard_normal(T).astype(np.float32)).cuda()
    out = layer.expert_forward(x, gate)
    # rows to addresses, in another order and mixed with their scores
    mixed, perm = torch.empty_like(x), torch.from_numpy(rng.permutation(T)).cuda()
    if F >= D:       # what the call asks for
        layer.expert_forward_scatter(x, gate, mixed.data_ptr() + 4 * D * perm, score)
    few = [layer.expert_forward(x[i:i + 16].contiguous(), gate[i:i + 16].contiguous()) for i in (0, (T - 16) // 2, T - 16)]
    layer.sync_status()
    layer.terminate()
    for i, rows in zip((0, (T - 16) // 2, T - 16), few):
        assert torch.equal(rows, out[i:i + 16])
    alpha = torch.sigmoid(score.double())[:, None]
    want = alpha * out.double() + (1 - alpha) * x.double()
    assert F < D or float((mixed[perm] - want).norm() / want.norm()) <= 5e-7     # eight roundings at most, the sigmoid included
    head = x[:64].cpu().numpy()
    want = oracle.expert_ffn_f64(head, *expert)
    assert oracle.rel_l2(out[:64].cpu().numpy() - head, want - head) <= 2e-6     # FP32 chains of up to 1030 adds
