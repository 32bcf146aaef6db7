"""GPU parity of the fused network path (inference, forward-with-stash, adjoint, weight/bias/grid gradients) against
the CPU oracle, called through the C ABI. Mirrors the structure of the reference's
tests_py/qmlp_tests/test_network_base.py:87-147 (fused vs simulated network: inference, forward, input gradients,
parameter gradients at several batch sizes) and tests_cpp/test_against_eigen2.cpp (uneven widths, all-gradient modes).
"""
import ctypes as C
import json

import numpy as np
import pytest

import helpers
import qmlp_oracle as oracle
import specs

pytestmark = pytest.mark.gpu

LEAKY = {"id": "leaky", "forward": "z = __hgt(x, hZERO()) ? x : __hmul(x, __float2half(0.125f))",
         "adjoint": "adjx = __hgt(x, hZERO()) ? adjz : __hmul(adjz, __float2half(0.125f))"}


def _leaky_oracle():
    acts = dict(oracle.ACTIVATIONS)
    acts["leaky"] = oracle.OracleActivation(lambda x: np.where(x > 0, x, 0.125 * x).astype(x.dtype),
                                            lambda x, g: np.where(x > 0, g, 0.125 * g).astype(g.dtype))
    return acts


def network_cases():
    """name -> (cfg, input range, parameter style)"""
    return {
        "config1": (specs.config1(), (0.0, 1.0), "reference"),
        "config2": (specs.config2(), (-1.0, 1.0), "xavier"),
        "ref_widths": (specs.identity_net(16, [32, 48, 16], ["celu", "identity", "celu"], bias=False), (-1.0, 1.0), "reference"),
        "uneven": (specs.identity_net(5, [20, 23, 7], ["sine", "relu", "identity"], bias=[True, False, True]), (-1.0, 1.0), "reference"),
        "custom_act": (specs.identity_net(4, [32, 32, 2], ["leaky", "sine", "leaky"], bias=True, extra_activations=[LEAKY]), (-1.0, 1.0), "reference"),
        # one activation per output channel (the reference parses such arrays and refuses them at code generation,
        # src_cpp/src/fused_network.cpp:106-125, 447): runs of built-ins, a user snippet, and a uniform array
        "per_channel": (specs.identity_net(4, [24, 20, 16, 3],
                                           [["relu"] * 8 + ["sine"] * 10 + ["celu"] * 6, ["identity"] * 5 + ["leaky"] * 15,
                                            ["celu"] * 16, "identity"], bias=True, extra_activations=[LEAKY]),
                        (-1.0, 1.0), "reference"),
        # rays (start, direction) integrated through a hash grid, plus the raw ray as identity features
        "line_net": ({"num_inputs": 6, "num_outputs": 3, "activation_specification": specs.BUILTIN,
                      "encodings": [{"id": "LineIntegration", "start_in": 0, "n_in": 3, "stepsize": 0.07, "blending": "average",
                                     "volume": specs.hashgrid(3, 4, 4, 10, 4, 32)},
                                    {"id": "Identity", "start_in": 0, "n_in": 6}],
                      "network": specs.mlp([32, 3], ["celu", "identity"], True)}, (-0.3, 1.3), "xavier"),
        "config3_small": (specs.config3(log2_hashmap_size=12), (0.0, 1.0), "xavier"),
        "config4_small": (specs.config4(log2_hashmap_size=10, dense_resolution=16), (0.0, 1.0), "xavier"),
        "config5_small": (specs.config5(log2_hashmap_size=12), (0.0, 1.0), "xavier"),
        "grid2d_add_plus_identity": (
            {"num_inputs": 4, "num_outputs": 3, "activation_specification": specs.BUILTIN,
             "encodings": [specs.hashgrid(2, 4, 4, 8, 4, 64, combination_mode="add", start_in=1, box_min=[-1, -1], box_size=[2, 2]),
                           {"id": "Identity", "start_in": 0, "n_in": 4}],
             "network": specs.mlp([32, 3], ["celu", "identity"], True)}, (-1.0, 1.0), "reference"),
    }


def _setup(name):
    import torch
    from qmlp import bindings
    cfg, rng, style = network_cases()[name]
    spec = oracle.parse_spec(cfg)
    net = bindings.Network(json.dumps(cfg))
    params = helpers.xavier_parameters(spec, cfg, bias_scale=0.1) if style == "xavier" else helpers.reference_style_parameters(spec)
    tables = helpers.grid_tables(spec, scale=1.0)
    acts = _leaky_oracle()
    dev = torch.device("cuda")
    t_params = torch.from_numpy(params).to(dev)
    t_tables = [torch.from_numpy(t).to(dev) if t is not None else None for t in tables]
    return cfg, rng, spec, net, params, tables, acts, t_params, t_tables


@pytest.mark.parametrize("name", list(network_cases().keys()))
def test_spec_layout_matches_oracle(name):
    cfg, rng, spec, net, *_ = _setup(name)
    assert net.num_network_parameters() == spec.num_parameters
    assert net.num_layers() == len(spec.layers)
    for i, l in enumerate(spec.layers):
        cin, cout, bias, ws, bs = net.layer_info(i)
        assert (cin, cout, bias, ws) == (l.channels_in, l.channels_out, l.use_bias, l.weights_start)
        if l.use_bias:
            assert bs == l.bias_start
    for i, e in enumerate(spec.encodings):
        enc = net.encoding(i)
        assert enc.num_output_channels() == e.num_outputs
        assert enc.parameter_count() == e.num_parameters
        assert enc.grid_levels() == [(lv.memory_offset, lv.resolution, lv.hash_grid_size, lv.hashed) for lv in e.levels]


@pytest.mark.parametrize("name", list(network_cases().keys()))
@pytest.mark.parametrize("n", [1, 33, 1000])
@pytest.mark.parametrize("path", [0, 3])
def test_inference(name, n, path):
    """path 0: the kernel the library picks for this batch (the mma.sync kernel at these sizes); path 3: the tcgen05
    kernel regardless of the batch size (falls back to mma.sync for specs wider than 128)."""
    import torch
    from qmlp import bindings
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    x = helpers.uniform(42, 1, (n, spec.num_inputs), *rng)
    try:
        bindings.QuickMLP.set_kernel_path(path)
        out = net.inference(torch.from_numpy(x).cuda(), t_params, t_tables).cpu().numpy()
    finally:
        bindings.QuickMLP.set_kernel_path(0)
    assert bindings.QuickMLP.device_status() == 0
    emu = oracle.network_forward(spec, params, x, tables, half=True, activations=acts)
    ref = oracle.network_forward(spec, params, x, tables, half=False, activations=acts)
    assert np.isfinite(out).all()
    helpers.assert_close(out, emu, f"{name} inference vs fp16-emulating oracle", max_violations=0.01)
    helpers.assert_close(out, ref, f"{name} inference vs fp32 oracle", max_violations=helpers.MAX_VIOLATIONS)


@pytest.mark.parametrize("name", ["config2", "uneven", "custom_act", "per_channel", "config4_small", "config5_small"])
@pytest.mark.parametrize("n", [127, 128, 5000, 40001, 200_000])
def test_tensor_core_paths_agree(name, n):
    """The tcgen05 inference kernel and the mma.sync kernel compute the same function (same rounding points: fp32
    accumulate, one rounding to half per layer), and no kernel reports a timed-out on-chip wait."""
    import torch
    from qmlp import bindings
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    x = torch.from_numpy(helpers.uniform(42, 7, (n, spec.num_inputs), *rng)).cuda()
    try:
        bindings.QuickMLP.set_kernel_path(3)
        out_best = net.inference(x, t_params, t_tables)
        bindings.QuickMLP.set_kernel_path(1)
        out_mma = net.inference(x, t_params, t_tables)
    finally:
        bindings.QuickMLP.set_kernel_path(0)
    assert bindings.QuickMLP.device_status() == 0
    emu = oracle.network_forward(spec, params, x.cpu().numpy(), tables, half=True, activations=acts)
    helpers.assert_close(out_best.cpu().numpy(), emu, f"{name} best path vs oracle", max_violations=0.01)
    # accumulation order differs (K in steps of 16 inside one instruction vs per-fragment), so allow a few half ulps
    helpers.assert_close(out_best.cpu().numpy(), out_mma.cpu().numpy(), f"{name} tcgen05 vs mma.sync", rtol=5e-3, atol=1e-3,
                         max_violations=0.005)


@pytest.mark.parametrize("name", ["config3_small", "config4_small", "config5_small", "grid2d_add_plus_identity"])
@pytest.mark.parametrize("half_tables", [False, True])
def test_level_major_encoding_pass(name, half_tables):
    """Inference through the level-major encoding pass (encodings of a chunk computed one grid level at a time into
    feature planes, then the layer chain on the planes) equals the fused gather, also across several chunks."""
    import torch
    from qmlp import bindings
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    n = (1 << 22) + 4321 if name == "config3_small" else 3000       # more than one chunk (2^22 points) for one case
    x = torch.from_numpy(helpers.uniform(42, 8, (n, spec.num_inputs), *rng)).cuda()
    tabs = [t.half() if (t is not None and half_tables) else t for t in t_tables]
    try:
        bindings.QuickMLP.set_kernel_path(2)
        out_planes = net.inference(x, t_params, tabs)
        bindings.QuickMLP.set_kernel_path(3)     # gather fused into the layer kernel (automatic choice may pick the pass)
        out_fused = net.inference(x, t_params, tabs)
    finally:
        bindings.QuickMLP.set_kernel_path(0)
    assert bindings.QuickMLP.device_status() == 0
    helpers.assert_close(out_planes.cpu().numpy(), out_fused.cpu().numpy(), f"{name} planes vs fused", rtol=5e-3, atol=1e-3,
                         max_violations=0.005)
    m = 2000
    tabs_np = [t.astype(np.float16).astype(np.float32) if (t is not None and half_tables) else t for t in tables]
    emu = oracle.network_forward(spec, params, x[-m:].cpu().numpy(), tabs_np, half=True, activations=acts)
    helpers.assert_close(out_planes[-m:].cpu().numpy(), emu, f"{name} planes vs oracle", max_violations=0.01)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257])
@pytest.mark.parametrize("name", ["config3_small", "config4_small", "config5_small", "grid2d_add_plus_identity"])
def test_lane_pairs_of_the_plane_kernels(name, n):
    """The plane kernels give a point to two neighbouring lanes: batches that end inside a pair, a warp or a CTA, for both
    pairing dimensions (hashed and dense levels), concatenating and adding grids. Features through the inference output,
    table gradients against the scatter inside the backward kernel."""
    import torch
    from qmlp import _capi, bindings
    from qmlp._capi import check, lib, wrap
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    x = helpers.uniform(43, 1, (n, spec.num_inputs), *rng)
    tx = torch.from_numpy(x).cuda()
    tadj = torch.from_numpy(helpers.uniform(43, 2, (n, spec.num_outputs), -1.0, 1.0)).cuda()
    out = torch.empty((n, spec.num_outputs), device="cuda")
    fwd = torch.empty((net.forward_memory(n),), dtype=torch.uint8, device="cuda")
    bwd = torch.empty((net.adjoint_memory(n, 6),), dtype=torch.uint8, device="cuda")
    expected = oracle.network_forward(spec, params, x, tables, half=True, activations=acts)
    results = []
    try:
        bindings.QuickMLP.set_kernel_path(2)
        helpers.assert_close(net.inference(tx, t_params, t_tables).cpu().numpy(), expected, f"{name} n={n}", max_violations=0.01)
        bindings.QuickMLP.set_tuning("split_scatter", 1)
        for path in (2, 1):
            bindings.QuickMLP.set_kernel_path(path)
            grads = [torch.zeros_like(t) if t is not None else None for t in t_tables]
            net._bind(t_params, t_tables)
            for i, g in enumerate(grads):
                if g is not None:
                    net.encoding(i).set_parameter(g, _capi.QMLP_GRADIENTS)
            check(lib().qmlp_network_forward(net._h, wrap(tx), wrap(out), fwd.data_ptr(), None))
            check(lib().qmlp_network_adjoint(net._h, wrap(tx), wrap(tadj), 4, None, fwd.data_ptr(), bwd.data_ptr(), None))
            torch.cuda.synchronize()
            results.append(grads)
    finally:
        bindings.QuickMLP.set_kernel_path(0)
        bindings.QuickMLP.set_tuning("split_scatter", -1)
    for a, b in zip(*results):
        if a is not None:
            # the same fp32 terms in another order: at most a few dozen per row
            helpers.assert_close(a.cpu().numpy(), b.cpu().numpy(), f"{name} n={n} table gradient", rtol=1e-4,
                                 atol=1e-5 * float(b.abs().max()))


@pytest.mark.parametrize("n", [1, 2, 31, 33, 257])
@pytest.mark.parametrize("half_tables", [False, True])
@pytest.mark.parametrize("name", ["config3_small", "config4_small", "config5_small", "grid2d_add_plus_identity"])
def test_features_of_a_pass_with_gradients(name, half_tables, n):
    """The forward pass that a backward pass follows exchanges the rows of a lane pair instead of half sums: its encoded input
    (the first rows of the stash) against the oracle. One fp16 rounding; a coordinate rounded differently by half an ulp
    moves the fraction of a cell by resolution * 2^-24 per dimension, between rows that are at most 2 apart."""
    import torch
    from qmlp._capi import check, lib, wrap
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    x = helpers.uniform(43, 3, (n, spec.num_inputs), *rng)
    tx = torch.from_numpy(x).cuda()
    out = torch.empty((n, spec.num_outputs), device="cuda")
    fwd = torch.empty((net.forward_memory(n),), dtype=torch.uint8, device="cuda")
    net._bind(t_params, [t.half() if (t is not None and half_tables) else t for t in t_tables])
    check(lib().qmlp_network_forward(net._h, wrap(tx), wrap(out), fwd.data_ptr(), None))
    torch.cuda.synchronize()
    tabs = [t.astype(np.float16).astype(np.float32) if (t is not None and half_tables) else t for t in tables]
    expected = oracle.encode(spec, x, tabs)
    width = spec.layers[0].channels_in
    got = fwd.view(torch.float16)[:n * width].view(n, width).float().cpu().numpy()
    grids = [e for e in spec.encodings if e.levels]
    atol = max(2 * len(e.levels) * 4 * max(lv.resolution for lv in e.levels) for e in grids) * 2.0 ** -24
    helpers.assert_close(got, expected, f"{name} n={n}", rtol=2.0 ** -10, atol=atol)


@pytest.mark.parametrize("name,n,chunk", [("config2", 100_003, 0), ("config2", 5000, 1024), ("config3_small", 70_001, 4096),
                                          ("config1", 17, 0), ("config1", 0, 0)])
def test_inference_from_host_memory(name, n, chunk):
    """The chunk-pipelined host-memory entry point returns exactly what the device-tensor call returns, for ragged
    last chunks, batches smaller than a chunk, an empty batch, and when called twice in a row on the same buffers."""
    import torch
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    x = torch.from_numpy(helpers.uniform(42, 9, (n, spec.num_inputs), *rng))
    hx = x.pin_memory()
    ref = net.inference(x.cuda(), t_params, t_tables).cpu()
    out = net.inference_host(hx, t_params, t_tables, chunk_points=chunk)
    torch.cuda.current_stream().synchronize()
    assert out.shape == ref.shape
    assert torch.equal(out, ref)
    out.zero_()
    out2 = net.inference_host(hx, t_params, t_tables, output=out, chunk_points=chunk)
    torch.cuda.current_stream().synchronize()
    assert out2 is out and torch.equal(out, ref)
    assert bindings_status() == 0


def bindings_status():
    from qmlp import bindings
    return bindings.QuickMLP.device_status()


def test_inference_half_tables_and_strided_io():
    """fp16 gather table (extension) and non-contiguous input/output views."""
    import torch
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup("config3_small")
    n = 777
    x = helpers.uniform(42, 2, (n, spec.num_inputs), *rng)
    wide = torch.zeros((n, 8), device="cuda")
    wide[:, 2:5] = torch.from_numpy(x).cuda()
    half_tables = [t.half() if t is not None else None for t in t_tables]
    out = net.inference(wide[:, 2:5], t_params, half_tables).cpu().numpy()
    tables16 = [t.astype(np.float16).astype(np.float32) if t is not None else None for t in tables]
    emu = oracle.network_forward(spec, params, x, tables16, half=True)
    helpers.assert_close(out, emu, "fp16 table inference", max_violations=0.01)


def _read_stash(spec, fwd_tmp, n):
    """Forward stash layout: [encoded input (N32, Cin0) | pre-activation of layer 0 (N32, Cout0) | layer 1 ...],
    fp16, N32 = N rounded up to 32; the encoded input row-major, the pre-activations in 8 x 8 blocks
    (helpers.stash_rows). Rows >= N are never written."""
    n32 = (n + 31) // 32 * 32
    halfs = fwd_tmp.view(dtype=np.float16)
    out, off = [], 0
    for i, width in enumerate([spec.layers[0].channels_in] + [l.channels_out for l in spec.layers]):
        seg = halfs[off:off + n32 * width]
        rows = seg.reshape(n32, width) if i == 0 else helpers.stash_rows(seg, n32, width)
        out.append(rows[:n].astype(np.float32))
        off += n32 * width
    return out


@pytest.mark.parametrize("name", list(network_cases().keys()))
@pytest.mark.parametrize("n", [32, 513, 4100])
def test_forward_and_adjoint(name, n):
    """forward with stash, then the adjoint with every gradient enabled, through the C ABI.

    The forward stash (encoded input and pre-activations) is compared with the oracle's forward pass. The adjoint is
    then compared with the oracle adjoint evaluated AT THE STASHED STATE, as the reference's backward kernels do:
    with relu/celu a pre-activation within one fp16 ulp of zero flips a derivative and changes that point's whole
    upstream gradient, which says nothing about the adjoint arithmetic under test."""
    import torch
    from qmlp import _capi
    from qmlp._capi import check, lib, wrap
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    x = helpers.uniform(42, 3, (n, spec.num_inputs), *rng)
    adj = helpers.uniform(42, 4, (n, spec.num_outputs), -1.0, 1.0)
    tx, tadj = torch.from_numpy(x).cuda(), torch.from_numpy(adj).cuda()
    out = torch.empty((n, spec.num_outputs), device="cuda")
    fwd = torch.full((net.forward_memory(n),), 0x7e, dtype=torch.uint8, device="cuda")     # poison: fp16 NaN pattern
    bwd = torch.full((net.adjoint_memory(n),), 0x7e, dtype=torch.uint8, device="cuda")
    grads = torch.zeros((spec.num_parameters,), device="cuda")
    adj_in = torch.zeros_like(tx)
    grid_grads = [torch.zeros_like(t) if t is not None else None for t in t_tables]
    check(lib().qmlp_network_set_parameter(net._h, wrap(t_params), _capi.QMLP_INFERENCE))
    check(lib().qmlp_network_set_parameter(net._h, wrap(grads), _capi.QMLP_GRADIENTS))
    for i, t in enumerate(t_tables):
        if t is not None:
            net.encoding(i).set_parameter(t, _capi.QMLP_INFERENCE)
            net.encoding(i).set_parameter(grid_grads[i], _capi.QMLP_GRADIENTS)
    check(lib().qmlp_network_forward(net._h, wrap(tx), wrap(out), fwd.data_ptr(), None))
    ai = wrap(adj_in)
    check(lib().qmlp_network_adjoint(net._h, wrap(tx), wrap(tadj), 7, C.byref(ai), fwd.data_ptr(), bwd.data_ptr(), None))
    torch.cuda.synchronize()

    # forward: output and stash against the oracle's own forward pass
    feat = oracle.encode(spec, x, tables)
    o_out, o_pres, _ = oracle.mlp_forward(spec, params, feat, True, acts)
    helpers.assert_close(out.cpu().numpy(), o_out[:, :spec.num_outputs], f"{name} forward output", max_violations=0.01)
    stash = _read_stash(spec, fwd.cpu().numpy(), n)
    helpers.assert_close(stash[0], feat.astype(np.float16).astype(np.float32), f"{name} stashed encoding", rtol=2e-3, atol=1e-3)
    for i, p in enumerate(o_pres):
        helpers.assert_close(stash[1 + i], p, f"{name} stashed pre-activation {i}", max_violations=0.01)

    # adjoint at the stashed state
    g = oracle.network_backward(spec, params, x, adj, tables, half=True, activations=acts, stash=stash)
    in_scale = max(1.0, float(np.abs(g.adj_input).max()))
    helpers.assert_close(adj_in.cpu().numpy(), g.adj_input, f"{name} input gradient", atol=1e-3 * in_scale, max_violations=0.01)
    scale = max(1.0, float(np.abs(g.grad_params).max()))
    helpers.assert_close(grads.cpu().numpy(), g.grad_params, f"{name} weight+bias gradient", atol=1e-3 * scale, max_violations=0.01)
    for i, e in enumerate(spec.encodings):
        if e.num_parameters:
            gs = max(1.0, float(np.abs(g.grad_encodings[i]).max()))
            helpers.assert_close(grid_grads[i].cpu().numpy(), g.grad_encodings[i], f"{name} grid gradient", atol=1e-3 * gs,
                                 max_violations=0.01)

    # fully independent fp32 oracle (its own forward pass): norm-wise agreement
    g32 = oracle.network_backward(spec, params, x, adj, tables, half=False, activations=acts)

    def rel(a, b):
        return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-12))
    assert rel(grads.cpu().numpy(), g32.grad_params) < 0.15, f"{name} weight gradient vs fp32 oracle"
    assert rel(adj_in.cpu().numpy(), g32.adj_input) < 0.15, f"{name} input gradient vs fp32 oracle"


@pytest.mark.parametrize("name", ["config2", "uneven", "config3_small", "grid2d_add_plus_identity"])
def test_autograd_binding(name):
    """The autograd path of the Python binding (role of NetworkBindings::forward, bind_network.cpp:120-321) returns the
    same gradients as direct C-ABI calls, for every flag subset a user can trigger with requires_grad."""
    import torch
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    n = 300
    x = helpers.uniform(42, 5, (n, spec.num_inputs), *rng)
    adj = torch.from_numpy(helpers.uniform(42, 6, (n, spec.num_outputs), -1.0, 1.0)).cuda()

    def run(want_x, want_w, want_t):
        tx = torch.from_numpy(x).cuda().requires_grad_(want_x)
        tp = t_params.float().requires_grad_(want_w)      # fp32 master, cast to half per call like the reference binding
        tt = [t.clone().requires_grad_(want_t) if t is not None else None for t in t_tables]
        out = net.forward(tx, tp, tt)
        out.backward(adj)
        torch.cuda.synchronize()
        return out.detach(), tx.grad, tp.grad, [t.grad if t is not None else None for t in tt]

    o_all, gx, gw, gt = run(True, True, True)
    o_inf = net.inference(torch.from_numpy(x).cuda(), t_params, t_tables)
    # forward-with-stash rounds every pre-activation to half before the activation (it is what backward reads);
    # the inference kernel may apply the activation to the fp32 accumulator: same function, a few half ulps apart
    helpers.assert_close(o_all.cpu().numpy(), o_inf.cpu().numpy(), "forward vs inference", rtol=5e-3, atol=1e-3, max_violations=0.005)
    assert gw.dtype == torch.float32 and gw.shape == t_params.shape
    _, gx1, gw1, _ = run(True, False, False)
    assert gw1 is None
    helpers.assert_close(gx1.cpu().numpy(), gx.cpu().numpy(), "input-only flags", rtol=1e-3, atol=1e-4 * max(1.0, float(gx.abs().max())))
    _, gx2, gw2, _ = run(False, True, False)
    assert gx2 is None
    helpers.assert_close(gw2.cpu().numpy(), gw.cpu().numpy(), "weights-only flags", rtol=1e-3, atol=1e-4 * max(1.0, float(gw.abs().max())))
    if any(t is not None for t in t_tables):
        _, _, _, gt3 = run(False, False, True)
        for a, b in zip(gt3, gt):
            if a is not None:
                helpers.assert_close(a.cpu().numpy(), b.cpu().numpy(), "encoding-only flags", rtol=1e-3,
                                     atol=1e-4 * max(1.0, float(b.abs().max())))


@pytest.mark.parametrize("name", ["config3_small", "config4_small", "config5_small", "grid2d_add_plus_identity"])
def test_table_gradient_scatter_paths_agree(name):
    """Weight + table gradients without input gradients: the level-major scatter kernel (adjoint feature planes, merged
    corner pairs) and the scatter inside the backward kernel produce the same sums."""
    import torch
    from qmlp import _capi, bindings
    from qmlp._capi import check, lib, wrap
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    n = 20_011
    tx = torch.from_numpy(helpers.uniform(42, 11, (n, spec.num_inputs), *rng)).cuda()
    tadj = torch.from_numpy(helpers.uniform(42, 12, (n, spec.num_outputs), -1.0, 1.0)).cuda()
    out = torch.empty((n, spec.num_outputs), device="cuda")
    fwd = torch.empty((net.forward_memory(n),), dtype=torch.uint8, device="cuda")
    assert net.adjoint_memory(n, 6) > net.adjoint_memory(n, 2) > 0
    bwd = torch.full((net.adjoint_memory(n, 6),), 0x7e, dtype=torch.uint8, device="cuda")
    results = []
    try:
        for path in (0, 1):
            bindings.QuickMLP.set_kernel_path(path)
            grads = torch.zeros((spec.num_parameters,), device="cuda")
            grid_grads = [torch.zeros_like(t) if t is not None else None for t in t_tables]
            check(lib().qmlp_network_set_parameter(net._h, wrap(t_params), _capi.QMLP_INFERENCE))
            check(lib().qmlp_network_set_parameter(net._h, wrap(grads), _capi.QMLP_GRADIENTS))
            for i, t in enumerate(t_tables):
                if t is not None:
                    net.encoding(i).set_parameter(t, _capi.QMLP_INFERENCE)
                    net.encoding(i).set_parameter(grid_grads[i], _capi.QMLP_GRADIENTS)
            launches = net.launch_count()
            check(lib().qmlp_network_forward(net._h, wrap(tx), wrap(out), fwd.data_ptr(), None))
            check(lib().qmlp_network_adjoint(net._h, wrap(tx), wrap(tadj), 6, None, fwd.data_ptr(), bwd.data_ptr(), None))
            torch.cuda.synchronize()
            results.append((grads, grid_grads, net.launch_count() - launches))
    finally:
        bindings.QuickMLP.set_kernel_path(0)
    assert bindings.QuickMLP.device_status() == 0
    (w0, g0, l0), (w1, g1, l1) = results
    # the separate scatter kernel is used when every grid has two features (only then can corner pairs be merged)
    split = all(e.n_features == 2 for e in spec.encodings if e.num_parameters)
    assert l0 == l1 + (1 if split else 0)
    helpers.assert_close(w0.cpu().numpy(), w1.cpu().numpy(), f"{name} weight gradient, both paths", rtol=1e-4,
                         atol=1e-5 * max(1.0, float(w1.abs().max())))
    for a, b in zip(g0, g1):
        if a is not None:
            assert float(b.abs().max()) > 0
            helpers.assert_close(a.cpu().numpy(), b.cpu().numpy(), f"{name} table gradient, both paths", rtol=1e-3,
                                 atol=1e-5 * max(1.0, float(b.abs().max())))


def test_gradients_accumulate():
    """adjoint adds to the bound gradient tensors (reference: outAdjWeights[i] += ..., callers zero them)."""
    import torch
    from qmlp import _capi
    from qmlp._capi import check, lib, wrap
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup("config1")
    n = 200
    x = torch.from_numpy(helpers.uniform(1, 5, (n, 3))).cuda()
    adj = torch.from_numpy(helpers.uniform(1, 6, (n, 1), -1, 1)).cuda()
    out = torch.empty((n, 1), device="cuda")
    grads = torch.zeros((spec.num_parameters,), device="cuda")
    adj_in = torch.zeros_like(x)
    fwd = torch.empty((net.forward_memory(n),), dtype=torch.uint8, device="cuda")
    bwd = torch.empty((net.adjoint_memory(n),), dtype=torch.uint8, device="cuda")
    check(lib().qmlp_network_set_parameter(net._h, wrap(t_params), _capi.QMLP_INFERENCE))
    check(lib().qmlp_network_set_parameter(net._h, wrap(grads), _capi.QMLP_GRADIENTS))
    check(lib().qmlp_network_forward(net._h, wrap(x), wrap(out), fwd.data_ptr(), None))
    ai = wrap(adj_in)
    for _ in range(2):
        check(lib().qmlp_network_adjoint(net._h, wrap(x), wrap(adj), 7, C.byref(ai), fwd.data_ptr(), bwd.data_ptr(), None))
    torch.cuda.synchronize()
    stash = _read_stash(spec, fwd.cpu().numpy(), n)
    once = oracle.network_backward(spec, params, x.cpu().numpy(), adj.cpu().numpy(), half=True, stash=stash)
    scale = max(1.0, float(np.abs(once.grad_params).max()))
    helpers.assert_close(grads.cpu().numpy(), 2 * once.grad_params, "accumulated weight gradient", atol=1e-3 * scale, max_violations=0.01)
    helpers.assert_close(adj_in.cpu().numpy(), 2 * once.adj_input, "accumulated input gradient", max_violations=0.01)
    check(lib().qmlp_network_zero_gradients(net._h, None))
    torch.cuda.synchronize()
    assert float(grads.abs().max()) == 0.0


def test_argument_errors():
    """Same failures as the reference's CHECK_* macros (src_cpp/src/fused_network.cpp:257-278, 509-516)."""
    import torch
    from qmlp._capi import QmlpError, ConfigurationError
    from qmlp import bindings
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup("config1")
    with pytest.raises(QmlpError):
        net.inference(torch.zeros((4, 2), device="cuda"), t_params)            # wrong channel count
    with pytest.raises(QmlpError):
        net.inference(torch.zeros((4, 3), device="cuda"), t_params[:-1].contiguous())   # wrong parameter count
    with pytest.raises(ConfigurationError):
        bindings.Network(json.dumps(dict(specs.config1(), num_outputs=2)))        # last layer != num_outputs
    with pytest.raises(ConfigurationError):
        bad = specs.config1(); bad["encodings"][0]["id"] = "identity"              # factory key is "Identity"
        bindings.Network(json.dumps(bad))
    with pytest.raises(ConfigurationError):
        bad = specs.config1(); bad["network"][0]["activation"] = "nope"
        bindings.Network(json.dumps(bad))
    out = net.inference(torch.zeros((0, 3), device="cuda"), t_params)             # empty batch is a no-op
    assert out.shape == (0, 1)


def wide_grid_config():
    """A grid in front of hidden layers that are all wider than 64 channels: activations in tensor memory, two tiles in flight"""
    return specs.grid_net(3, [specs.hashgrid(3, 8, 4, 10, 4, 48)], [128, 96, 128, 4], ["relu", "celu", "relu", "identity"])


# Path 3 runs the kernel on identity inputs at any number of points. From feature planes (path 2) it runs from two tiles per SM
# on (fewer points of a chunk go to the mma.sync kernel): 37 888 on 148 SMs. 16 tiles per SM give each of eight slots
# its second tile.
@pytest.mark.parametrize("name,path,n", [(name, 3, n) for name in ("config1", "config2", "uneven", "per_channel")
                                         for n in (1, 127, 128, 129, 148 * 128 + 1, 148 * 128 * 6 + 33, 148 * 128 * 16 + 33)] +
                                        [(name, 2, n) for name in ("config3_small", "config5_small", "wide_grid")
                                         for n in (148 * 256 - 1, 148 * 256, 148 * 256 + 1, 148 * 256 + 127, 148 * 256 + 128, 148 * 256 + 129,
                                                   148 * 128 * 16 + 33)])
def test_activations_in_tensor_memory(name, path, n):
    """The kernel that keeps the activations in tensor memory (identity inputs, and feature planes): batches that end inside a
    tile, fill one, and give a slot its second and third; 16 to 128 channels, with and without bias. Against the mma.sync
    kernel: both round every layer to fp16 once (2^-11), the fp32 sums differ in order."""
    import torch
    from qmlp import bindings
    if name == "wide_grid":
        cfg, rng = wide_grid_config(), (0.0, 1.0)
        spec, net = oracle.parse_spec(cfg), bindings.Network(json.dumps(cfg))
        t_params = torch.from_numpy(helpers.xavier_parameters(spec, cfg, bias_scale=0.1)).cuda()
        t_tables = [torch.from_numpy(t).cuda() for t in helpers.grid_tables(spec)]
    else:
        cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    x = torch.from_numpy(helpers.uniform(46, 1, (n, spec.num_inputs), *rng)).cuda()
    out = []
    try:
        for p in (path, 1):
            bindings.QuickMLP.set_kernel_path(p)
            out.append(net.inference(x, t_params, t_tables).cpu().numpy())
    finally:
        bindings.QuickMLP.set_kernel_path(0)
    helpers.assert_close(out[0], out[1], f"{name} n={n}", rtol=5e-3, atol=2e-3, max_violations=0.005)


def _rounded_chain(spec, params, feat, acts, roundings):
    """Layer chain in 64 bits with fp16 inputs: one rounding per layer (bias and activation before it), or two (the
    accumulator, then the sum with the bias, and the activation of that)."""
    def half(a):
        return a.astype(np.float16).astype(np.float64)
    w = params.astype(np.float64)
    h = half(feat)
    for i, l in enumerate(spec.layers):
        pre = h @ oracle.weight_view(spec, w, i).T
        b = oracle.bias_view(spec, w, i)
        bias = 0.0 if b is None else b[None, :]
        pre = half(half(pre) + bias) if roundings == 2 else pre + bias
        h = half(oracle._act_forward(acts, l.activation, pre))
    return h[:, :spec.num_outputs]


@pytest.mark.parametrize("name,path", [("config2", 1), ("config2", 3), ("uneven", 1), ("uneven", 3), ("config3_small", 1), ("config3_small", 2),
                                       ("config5_small", 2)])
def test_inference_rounds_a_layer_once(name, path):
    """Every inference kernel (mma.sync: path 1, and on a few points from the planes: path 2; tcgen05: path 3) adds the
    bias and applies the activation in fp32. Against the chain in 64 bits with one rounding per layer; how far the chain
    with two roundings is from that is the scale (fp32 sums and the special-function unit flip a rounding now and then)."""
    import torch
    from qmlp import bindings
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    params = helpers.xavier_parameters(spec, cfg, bias_scale=0.5)
    x = helpers.uniform(61, 1, (3000, spec.num_inputs), *rng)
    feat = oracle.encode(spec, x, tables)
    once, twice = (_rounded_chain(spec, params, feat, acts, r) for r in (1, 2))
    try:
        bindings.QuickMLP.set_kernel_path(path)
        out = net.inference(torch.from_numpy(x).cuda(), torch.from_numpy(params).cuda(), t_tables).cpu().numpy().astype(np.float64)
    finally:
        bindings.QuickMLP.set_kernel_path(0)
    assert np.linalg.norm(out - once) < 0.5 * np.linalg.norm(twice - once)


@pytest.mark.parametrize("path", [0, 1])
def test_relu_of_nan(path):
    """"z = __hgt(x, hZERO()) ? x : hZERO()" is 0 for NaN in the mma.sync kernel: a NaN coordinate ends in the first layer's
    relu and the outputs are those of zero activations behind it; other rows of its tile are not touched."""
    import torch
    from qmlp import bindings
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup("config2")
    x = helpers.uniform(61, 1, (300, spec.num_inputs), *rng)
    x[5, 1] = np.nan
    ref = oracle.network_forward(spec, params, x, tables, half=True)
    assert np.isfinite(ref).all()
    try:
        bindings.QuickMLP.set_kernel_path(path)
        out = net.inference(torch.from_numpy(x).cuda(), t_params).cpu().numpy()
    finally:
        bindings.QuickMLP.set_kernel_path(0)
    helpers.assert_close(out, ref, f"path {path}", max_violations=0.01)
    helpers.assert_close(out[5], ref[5], f"path {path}, row with a NaN")


@pytest.mark.parametrize("n,chunk", [(1, 0), (129, 0), (5000, 1024), ((1 << 18) + 33, 0)])
@pytest.mark.parametrize("pinned", [True, False], ids=["pinned", "pageable"])
def test_inference_from_host_memory_in_place(n, chunk, pinned):
    """One output channel: a page-locked result is written by the kernels, a pageable one goes through the download slots; one
    chunk, several chunks, a ragged last one, a result that starts inside its allocation, and calls on two streams in turn.
    Each chunk runs the kernel that its own size picks: compared chunk by chunk with the device call."""
    import torch
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup("config2")
    x = torch.from_numpy(helpers.uniform(45, 1, (n, spec.num_inputs), *rng))
    step = chunk if chunk else ((1 << 18) if pinned else (1 << 16))
    ref = torch.cat([net.inference(x[i:i + step].cuda(), t_params, t_tables).cpu() for i in range(0, n, step)])
    hx = x.pin_memory()
    buf = torch.full((n + 2, 1), 7.0, pin_memory=pinned)
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            out = net.inference_host(hx, t_params, t_tables, output=buf[1:n + 1], chunk_points=chunk)
        stream.synchronize()
        assert torch.equal(out, ref) and float(buf[0]) == 7.0 and float(buf[n + 1]) == 7.0
        out.zero_()


@pytest.mark.parametrize("name", ["config2", "uneven"])
def test_inference_from_host_memory_on_two_streams(name):
    """Calls on two streams with nothing between them: chunks of 2^15 points, one chunk of 300 001, and a pageable result
    after a page-locked one. Each call cuts the staging memory its own way, so a slot of one covers several of another."""
    import torch
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    jobs = []
    for i, (n, chunk, pinned) in enumerate([(1 << 20, 1 << 15, True), (300_001, 300_001, True), (1 << 19, 1 << 14, False),
                                            (300_001, 300_001, True), (1 << 20, 1 << 15, True), (100_003, 0, False)]):
        x = torch.from_numpy(helpers.uniform(62, i, (n, spec.num_inputs), *rng)).pin_memory()
        out = torch.empty((n, spec.num_outputs), pin_memory=pinned)
        ref = net.inference_host(x, t_params, t_tables, output=torch.empty_like(out, pin_memory=pinned), chunk_points=chunk)
        torch.cuda.synchronize()
        jobs.append((x, out, ref, chunk))
    for _ in range(5):
        for i, (x, out, ref, chunk) in enumerate(jobs):
            out.zero_()
        for i, (x, out, ref, chunk) in enumerate(jobs):
            with torch.cuda.stream(streams[i & 1]):
                net.inference_host(x, t_params, t_tables, output=out, chunk_points=chunk)
        torch.cuda.synchronize()
        for i, (x, out, ref, chunk) in enumerate(jobs):
            assert torch.equal(out, ref), i


@pytest.mark.parametrize("chunk", [0, 1024])
@pytest.mark.parametrize("name", ["config2", "uneven"])
def test_inference_from_host_memory_under_capture(name, chunk):
    """A call that is captured after one that was not, its replay, and a call that is not captured after it."""
    import torch
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    n = 5000
    x = torch.from_numpy(helpers.uniform(45, 1, (n, spec.num_inputs), *rng)).pin_memory()
    out = torch.zeros((n, spec.num_outputs), pin_memory=True)
    stream = torch.cuda.Stream()

    def call():
        net.inference_host(x, t_params, t_tables, output=out, chunk_points=chunk)

    def result():
        torch.cuda.synchronize()
        r = out.clone()
        out.zero_()
        return r
    with torch.cuda.stream(stream):
        call()
    ref = result()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    graph.replay()
    assert torch.equal(result(), ref)
    with torch.cuda.stream(stream):
        call()
    assert torch.equal(result(), ref)


@pytest.mark.parametrize("fresh", [False, True], ids=["main", "fresh_thread"])
def test_inference_from_host_memory_takes_the_result_in_place(fresh):
    """A page-locked result of one channel: chunks of 2^18 points (2^16 with a download), so two launches for 2^18 + 33 points;
    the same from a thread that has made no CUDA call before."""
    import threading
    import torch
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup("config2")
    n = (1 << 18) + 33
    x = torch.from_numpy(helpers.uniform(67, 1, (n, spec.num_inputs), *rng)).pin_memory()
    out = torch.empty((n, 1), pin_memory=True)
    before = net.launch_count()

    def call():
        net.inference_host(x, t_params, output=out)
    if fresh:
        thread = threading.Thread(target=call)
        thread.start()
        thread.join()
    else:
        call()
    torch.cuda.synchronize()
    assert net.launch_count() - before == 2
    ref = net.inference(x.cuda(), t_params).cpu()
    assert float((out - ref).norm()) <= 5e-3 * float(ref.norm())


@pytest.mark.parametrize("registered", [0, 4096, 8192, 16384])
def test_inference_from_host_memory_with_a_result_registered_in_part(registered):
    """A result buffer whose first pages only are page-locked: nothing is written through the mapping. The copy either refuses it
    or brings the whole result; a buffer registered to its end gets it in any case."""
    import torch
    from qmlp._capi import QmlpError
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup("config2")
    n = 4096
    x = torch.from_numpy(helpers.uniform(65, 1, (n, spec.num_inputs), *rng)).pin_memory()
    ref = net.inference(x.cuda(), t_params).cpu()
    raw = np.zeros(n + 1024, dtype=np.float32)
    first = (-raw.ctypes.data) % 4096 // 4                   # a page boundary
    out = torch.from_numpy(raw[first:first + n]).view(n, 1)
    out.fill_(7.0)
    rt = torch.cuda.cudart()
    if registered:
        assert int(rt.cudaHostRegister(out.data_ptr(), registered, 0)) == 0
    try:
        net.inference_host(x, t_params, output=out)
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
    except QmlpError:
        assert registered in (4096, 8192)
        assert torch.equal(net.inference(x.cuda(), t_params).cpu(), ref)     # an error is reported once
    finally:
        torch.cuda.synchronize()
        if registered:
            assert int(rt.cudaHostUnregister(out.data_ptr())) == 0


@pytest.mark.parametrize("n,offset", [(1, 0), (3, 0), (4, 0), (1024, 0), (1023, 0), (1024, 1), (4097, 2)])
def test_convert_half(n, offset):
    """fp32 -> fp16 copy of a parameter vector: vector and scalar kernels, lengths and alignments either side of the rule."""
    import torch
    from qmlp._capi import check, lib
    src = torch.from_numpy(helpers.uniform(44, 1, (n + offset,), -3.0, 3.0)).cuda()[offset:]
    dst = torch.zeros((n + offset + 1,), dtype=torch.float16, device="cuda")
    check(lib().qmlp_convert_half(src.data_ptr(), dst[offset:].data_ptr(), n, None))
    torch.cuda.synchronize()
    assert torch.equal(dst[offset:offset + n], src.half()) and float(dst[offset + n]) == 0.0


@pytest.mark.parametrize("n", [1, 128, 129, 40_001])
@pytest.mark.parametrize("name", ["config1", "config2", "ref_widths", "uneven", "per_channel", "config3_small", "config4_small", "config5_small",
                                  "grid2d_add_plus_identity", "line_net"])
def test_recomputing_backward_pass(name, n):
    """Autograd through the pair that keeps the encoded features only and computes the layers a second time, against the pair that
    stashes the pre-activations (kernel path 1): output, weight gradient, table gradients, and the input gradient where no
    grid asks for its own. Batches that end inside a tile, fill one, and give a CTA three. Both round the same values to
    fp16; fp32 sums in another order move a rounding by 2^-11 now and then, and a pre-activation within that of zero may
    flip a relu: 1e-2 of each gradient's norm. (line_net has no such pair: the call falls back.)"""
    import torch
    from qmlp import bindings
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    grid = any(e.num_parameters for e in spec.encodings)
    x0 = torch.from_numpy(helpers.uniform(47, 1, (n, spec.num_inputs), *rng)).cuda()
    adj = torch.from_numpy(helpers.uniform(47, 2, (n, spec.num_outputs), -1.0, 1.0)).cuda()
    results = []
    try:
        for path in (0, 1):
            bindings.QuickMLP.set_kernel_path(path)
            x = x0.clone().requires_grad_(not grid)
            w = t_params.float().requires_grad_(True)
            tabs = [t.clone().requires_grad_(True) if t is not None else None for t in t_tables]
            before = net.launch_count()
            out = net.forward(x, w, tabs)
            out.backward(adj)
            torch.cuda.synchronize()
            results.append(([out.detach(), w.grad] + [t.grad for t in tabs if t is not None] + ([x.grad] if not grid else []), net.launch_count() - before))
    finally:
        bindings.QuickMLP.set_kernel_path(0)
    (a, launches), (b, launches_stash) = results
    if not grid:
        assert launches < launches_stash     # no weight-gradient kernel of its own
    for i, (ga, gb) in enumerate(zip(a, b)):
        norm = float(gb.norm())
        assert norm > 0 or n == 1     # (a single point may sit where a relu output is zero)
        assert float((ga - gb).norm()) <= 1e-2 * norm, f"{name} n={n} result {i}: {float((ga - gb).norm())} of {norm}"


@pytest.mark.parametrize("switch", ["kernel_path", "split_scatter"])
def test_backward_after_a_switch(switch):
    """The backward pass of a forward call that keeps the encoded features only does not depend on the switches that forward
    calls choose by."""
    import torch
    from qmlp import bindings
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup("config3_small")
    x = torch.from_numpy(helpers.uniform(63, 1, (3000, 3), *rng)).cuda()
    adj = torch.from_numpy(helpers.uniform(63, 2, (3000, 1), -1.0, 1.0)).cuda()
    grads = []
    for switched in (False, True):
        w, tb = t_params.float().requires_grad_(True), t_tables[0].clone().requires_grad_(True)
        out = net.forward(x, w, [tb])
        try:
            if switched and switch == "kernel_path":
                bindings.QuickMLP.set_kernel_path(1)
            elif switched:
                bindings.QuickMLP.set_tuning(switch, 0)
            out.backward(adj)
        finally:
            bindings.QuickMLP.set_kernel_path(0)
            bindings.QuickMLP.set_tuning("split_scatter", -1)
        grads.append((w.grad, tb.grad))
    for a, b in zip(*grads):   # the same kernels: fp32 sums in another order
        assert float((a - b).norm()) <= 1e-5 * float(a.norm()) > 0


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("name", ["config2", "config4_small"])
def test_recomputing_pair_with_a_gradient_vector_at_any_offset(name, offset):
    """A caller of the C entry points may bind a gradient vector that starts at any element (16-byte reductions where they are
    aligned, scalar ones elsewhere), with weight gradients taken as delta^T * input and as input^T * delta."""
    import torch
    from qmlp import _capi
    from qmlp._capi import check, lib, wrap
    cfg, rng, spec, net, params, tables, acts, t_params, t_tables = _setup(name)
    n = 3000
    x = torch.from_numpy(helpers.uniform(64, 1, (n, spec.num_inputs), *rng)).cuda()
    adj = torch.from_numpy(helpers.uniform(64, 2, (n, spec.num_outputs), -1.0, 1.0)).cuda()
    out = torch.empty_like(adj)
    check(lib().qmlp_network_set_parameter(net._h, wrap(t_params), _capi.QMLP_INFERENCE))
    for i, t in enumerate(t_tables):
        if t is not None:
            net.encoding(i).set_parameter(t, _capi.QMLP_INFERENCE)
    forward, adjoint = C.c_size_t(), C.c_size_t()
    check(lib().qmlp_network_recompute_memory(net._h, n, 2, C.byref(forward), C.byref(adjoint)))
    assert forward.value > 0
    tmp = torch.empty((forward.value + 16,), dtype=torch.uint8, device="cuda")
    check(lib().qmlp_network_forward_recompute(net._h, wrap(x), wrap(out), tmp.data_ptr(), None))
    grads = []
    for off in (0, offset):
        buf = torch.zeros((spec.num_parameters + 4,), device="cuda")
        g = buf[off:off + spec.num_parameters]
        check(lib().qmlp_network_set_parameter(net._h, wrap(g), _capi.QMLP_GRADIENTS))
        check(lib().qmlp_network_adjoint_recompute(net._h, wrap(x), wrap(adj), 2, None, tmp.data_ptr(), None, None))
        torch.cuda.synchronize()
        assert float(buf[:off].abs().sum()) == 0.0 and float(buf[off + spec.num_parameters:].abs().sum()) == 0.0
        grads.append(g.clone())
    assert float((grads[0] - grads[1]).norm()) <= 1e-5 * float(grads[0].norm()) > 0      # fp32 sums in another order
    with pytest.raises(_capi.QmlpError):
        check(lib().qmlp_network_adjoint_recompute(net._h, wrap(x), wrap(adj), 2, None, tmp.data_ptr() + 2, None, None))


def one_layer_configs():
    """name -> network of one layer: few inputs and many outputs (three slots by tensor memory, two by threads), and the other way
    round, with and without a grid and a bias"""
    return {"16_to_128": specs.identity_net(16, [128], ["relu"]),
            "40_to_100": specs.identity_net(40, [100], ["celu"], bias=False),
            "100_to_7": specs.identity_net(100, [7], ["sine"]),
            "grid_to_72": specs.grid_net(3, [specs.hashgrid(3, 4, 2, 10, 4, 48)], [72], ["identity"])}


@pytest.mark.parametrize("n", [1, 129, 148 * 256 + 1])
@pytest.mark.parametrize("name", ["16_to_128", "40_to_100", "100_to_7", "grid_to_72"])
def test_one_layer(name, n):
    """Networks of a single layer through the kernels picked for them and through the mma.sync ones (kernel path 1): inference,
    the recomputing pair, and the kernel of a training step. Roundings to fp16 (2^-11) in the same places."""
    import torch
    from qmlp import bindings
    from qmlp.trainer import FusedTrainer
    cfg = one_layer_configs()[name]
    spec, net = oracle.parse_spec(cfg), bindings.Network(json.dumps(cfg))
    params = torch.from_numpy(helpers.xavier_parameters(spec, cfg, bias_scale=0.2)).cuda()
    tables = [torch.from_numpy(t).cuda() if t is not None else None for t in helpers.grid_tables(spec, scale=0.7)]
    grid = any(t is not None for t in tables)
    x = torch.from_numpy(helpers.uniform(66, 1, (n, spec.num_inputs))).cuda()
    adj = torch.from_numpy(helpers.uniform(66, 2, (n, spec.num_outputs), -1.0, 1.0)).cuda()
    results = []
    try:
        for path in (1, 0, 2, 3):
            bindings.QuickMLP.set_kernel_path(path)
            r = [net.inference(x, params, tables)]
            xx, w = x.clone().requires_grad_(not grid), params.float().requires_grad_(True)
            tt = [t.clone().requires_grad_(True) if t is not None else None for t in tables]
            net.forward(xx, w, tt).backward(adj)
            r += [w.grad] + [t.grad for t in tt if t is not None] + ([] if grid else [xx.grad])
            tr = FusedTrainer(net, grid_half_copy=False)
            tr.set_parameters(params, tables)
            tr.backend.gradients(x, adj, n, tr.loss_sum)
            results.append(r + [tr.gradient, tr.loss_sum])
            torch.cuda.synchronize()
    finally:
        bindings.QuickMLP.set_kernel_path(0)
    for r in results[1:]:
        for a, b in zip(r, results[0]):
            assert float((a - b).norm()) <= 5e-3 * float(b.norm())
