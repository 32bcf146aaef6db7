"""GPU parity of the stand-alone encoding and activation entry points, through the C ABI.
Follows the reference's tests_py/qmlp_tests/test_encoding.py:10-188 (identity, dense grid 1-D / 2-D against
torch grid_sample, output + input gradient + parameter gradient) and test_activations.py:8-66 (relu, sine against
torch, forward + gradient), and adds what the reference never pins: hashed levels, 3-D / 4-D grids."""
import json

import numpy as np
import pytest

import helpers
import qmlp_oracle as oracle
import specs

pytestmark = pytest.mark.gpu


def encoding_cases():
    return {
        "identity": {"id": "Identity", "start_in": 1, "n_in": 5},
        "dense1d": specs.hashgrid(1, 1, 4, -1, 2, 16, combination_mode="add", box_min=[-1], box_size=[2]),
        "dense2d": specs.hashgrid(2, 1, 4, -1, 2, 16, combination_mode="add", box_min=[-1, -1], box_size=[2, 2]),
        "dense2d_multires": specs.hashgrid(2, 5, 4, -1, 16, 256, combination_mode="concat"),
        "hash3d_f2": specs.hashgrid(3, 8, 2, 10, 4, 512, per_level_scale=2.0),
        "hash4d_f4": specs.hashgrid(4, 6, 4, 12, 4, 64),
        "hash3d_f3_add": specs.hashgrid(3, 4, 3, 9, 8, 128, combination_mode="add", start_in=2, box_min=[-2, -2, -2], box_size=[4, 4, 4]),
        "hash2d_f8": specs.hashgrid(2, 4, 8, 8, 8, 256),
        "dense6d": specs.hashgrid(6, 2, 1, -1, 2, 3),
        # ray start + direction in, the grid integrated along the ray out (src_cpp/src/encoding_line_integration.cpp)
        "line_average": {"id": "LineIntegration", "start_in": 1, "n_in": 3, "stepsize": 0.05, "blending": "average",
                         "volume": specs.hashgrid(3, 4, 2, 10, 4, 32)},
        "line_additive_add": {"id": "LineIntegration", "start_in": 0, "n_in": 3, "stepsize": 0.11, "blending": "additive",
                              "volume": specs.hashgrid(3, 3, 4, 9, 4, 24, combination_mode="add", box_min=[-1, -1, -1],
                                                       box_size=[2, 2, 2])},
    }


def _enc(name):
    from qmlp import bindings
    cfg = encoding_cases()[name]
    e = bindings.Encoding(json.dumps(cfg))
    oe = oracle.parse_encoding(cfg)
    return cfg, e, oe


@pytest.mark.parametrize("name", ["line_average", "line_additive_add"])
def test_line_integration(name):
    """Rays that start in and around the volume's bounding box, with arbitrary directions (some miss the box): output,
    table gradient and ray gradients against the oracle's restatement of encoding_line_integration.cuh:61-165."""
    import torch
    cfg, e, oe = _enc(name)
    n = 301
    bmin, bsize = float(cfg["volume"]["bounding_box_min"][0]), float(cfg["volume"]["bounding_box_size"][0])
    x = helpers.uniform(7, 1, (n, oe.start_in + 7), bmin - 0.4 * bsize, bmin + 1.4 * bsize)
    x[:, oe.start_in + 3:oe.start_in + 6] = helpers.uniform(7, 2, (n, 3), -1.0, 1.0)
    adj = helpers.uniform(7, 3, (n, oe.num_outputs), -1, 1)
    assert e.num_output_channels() == oe.num_outputs and e.max_input_channel() == oe.start_in + 5
    assert e.parameter_count() == oe.num_parameters and json.loads(e.to_json())["id"] == "LineIntegration"
    table = helpers.uniform(7, 4, (oe.num_parameters,), -1, 1)
    tx = torch.from_numpy(x).cuda().requires_grad_(True)
    tp = torch.from_numpy(table).cuda().requires_grad_(True)
    out = e.forward_with_parameter(tx, tp)
    expect = oracle.grid_forward(oe, x, table)
    assert float(np.abs(expect).sum(axis=1).min()) == 0.0 and float(np.abs(expect).max()) > 0.1   # misses and hits
    scale = float(np.abs(expect).max())
    helpers.assert_close(out.detach().cpu().numpy(), expect, f"{name} forward", rtol=1e-3, atol=1e-4 * scale, max_violations=0.01)
    out.backward(torch.from_numpy(adj).cuda())
    g, ai = oracle.grid_adjoint(oe, x, table, adj, True, True)
    helpers.assert_close(tp.grad.cpu().numpy(), g, f"{name} table gradient", rtol=1e-3, atol=1e-4 * float(np.abs(g).max()),
                         max_violations=0.01)
    helpers.assert_close(tx.grad.cpu().numpy(), ai, f"{name} ray gradient", rtol=2e-3, atol=1e-3 * float(np.abs(ai).max()),
                         max_violations=0.01)


@pytest.mark.parametrize("name", [k for k in encoding_cases() if not k.startswith("line_")])
def test_encoding_forward_and_adjoint(name):
    import torch
    cfg, e, oe = _enc(name)
    n = 257
    n_in = oe.start_in + oe.n_in + 1
    # 1 % beyond the bounding box on both sides: exercises the clamped cells without the ill-conditioned
    # extrapolation weights (|f| >> 1) that far-away points produce
    if oe.id == "Identity":
        lo, hi = -1.0, 1.0
    else:
        bmin, bsize = float(cfg["bounding_box_min"][0]), float(cfg["bounding_box_size"][0])
        lo, hi = bmin - 0.01 * bsize, bmin + 1.01 * bsize
    x = helpers.uniform(3, 1, (n, n_in), lo, hi)
    adj = helpers.uniform(3, 2, (n, oe.num_outputs), -1, 1)
    assert e.num_output_channels() == oe.num_outputs and e.max_input_channel() == oe.start_in + oe.n_in - 1
    tx = torch.from_numpy(x).cuda().requires_grad_(True)
    if oe.id == "Identity":
        out = e.forward(tx)
        assert torch.equal(out.detach().cpu(), torch.from_numpy(x[:, oe.start_in:oe.start_in + oe.n_in]))
        out.backward(torch.from_numpy(adj).cuda())
        expect = np.zeros_like(x); expect[:, oe.start_in:oe.start_in + oe.n_in] = adj
        assert np.array_equal(tx.grad.cpu().numpy(), expect)
        return
    assert e.parameter_count() == oe.num_parameters
    table = helpers.uniform(3, 3, (oe.num_parameters,), -1, 1)
    tp = torch.from_numpy(table).cuda().requires_grad_(True)
    out = e.forward_with_parameter(tx, tp)
    expect = oracle.grid_forward(oe, x, table)
    # fp32 blend on both sides: only summation order and fma contraction differ
    helpers.assert_close(out.detach().cpu().numpy(), expect, f"{name} forward", rtol=1e-4, atol=1e-4)
    out.backward(torch.from_numpy(adj).cuda())
    g, ai = oracle.grid_adjoint(oe, x, table, adj, True, True)
    helpers.assert_close(tp.grad.cpu().numpy(), g, f"{name} parameter gradient", rtol=1e-4, atol=1e-4)
    helpers.assert_close(tx.grad.cpu().numpy(), ai, f"{name} input gradient", rtol=1e-3, atol=1e-3)


def test_grid_indices_bit_exact():
    """One-hot tables turn the gather into an index probe: with table[i] = i (exactly representable) and points on
    cell corners, the output IS the row index, so dense and hashed indices can be compared for equality."""
    import torch
    from qmlp import bindings
    for cfg in (specs.hashgrid(3, 6, 1, 14, 8, 300), specs.hashgrid(4, 4, 1, 16, 8, 64), specs.hashgrid(2, 5, 1, -1, 4, 64)):
        e = bindings.Encoding(json.dumps(cfg))
        oe = oracle.parse_encoding(cfg)
        n = 500
        for li, lv in enumerate(oe.levels):
            # integer cell coordinates in [0, res-2] -> positions exactly on the low corner: weight 1 on one corner
            cells = (helpers.uniform(9, 10 + li, (n, oe.n_in)) * (lv.resolution - 1)).astype(np.int64)
            x = (cells.astype(np.float64) / (lv.resolution - 1)).astype(np.float32)
            iL, iH, f = oracle.grid_cell(oe, lv, x)
            rows = oracle.grid_index(oe, lv, iL)          # element index of the low corner
            level_size = (lv.hash_grid_size if lv.hashed else lv.resolution ** oe.n_in)
            table = np.zeros(oe.num_parameters, dtype=np.float32)
            table[lv.memory_offset:lv.memory_offset + level_size] = np.arange(level_size, dtype=np.float32)
            out = e.inference_with_parameter(torch.from_numpy(x).cuda(), torch.from_numpy(table).cuda()).cpu().numpy()
            exact = f.max(axis=1) == 0                     # points whose fraction is exactly zero
            assert exact.sum() > n // 4
            got = out[exact, li]
            want = (rows[exact] - lv.memory_offset).astype(np.float32)
            assert np.array_equal(got, want), f"level {li}: index mismatch"


def test_dense_grid_matches_grid_sample():
    """The reference's own check (tests_py/qmlp_tests/test_encoding.py:143-188): a dense level equals
    grid_sample(align_corners=True, padding_mode='border')."""
    import torch
    cfg, e, oe = _enc("dense2d")
    r, c, n = 2, 4, 64
    x = torch.from_numpy(helpers.uniform(5, 1, (n, 2), -1, 1)).cuda()
    p = torch.from_numpy(helpers.uniform(5, 2, (r * r * c,), -1, 1)).cuda()
    out = e.inference_with_parameter(x, p)
    inp = p.reshape(1, r, r, c).permute((0, 3, 2, 1))
    ref = torch.nn.functional.grid_sample(inp, x.reshape(1, -1, 1, 2), mode="bilinear", align_corners=True,
                                          padding_mode="border")[0, :, :, 0].t()
    assert torch.allclose(out, ref, atol=1e-6)


@pytest.mark.parametrize("name", ["relu", "celu", "sine", "identity", "leaky"])
def test_activation(name):
    import torch
    from qmlp import bindings
    leaky = {"id": "leaky", "forward": "z = __hgt(x, hZERO()) ? x : __hmul(x, __float2half(0.125f))",
             "adjoint": "adjx = __hgt(x, hZERO()) ? adjz : __hmul(adjz, __float2half(0.125f))"}
    act = bindings.Activation(json.dumps(leaky) if name == "leaky" else name)
    assert act.id() == name
    fn = {"relu": torch.relu, "celu": torch.nn.functional.celu, "sine": torch.sin, "identity": lambda t: t,
          "leaky": lambda t: torch.nn.functional.leaky_relu(t, 0.125)}[name]
    for shape, strided in (((8, 6), False), ((37, 5), False), ((16, 8), True)):
        x = torch.from_numpy(helpers.uniform(1, 1, shape, -3, 3)).cuda().half()
        g = torch.from_numpy(helpers.uniform(1, 2, shape, -1, 1)).cuda().half()
        if strided:
            x = x.t().contiguous().t()
        xa = x.clone().requires_grad_(True)
        out = act.forward(xa)
        out.backward(g)
        xr = x.float().clone().requires_grad_(True)
        ref = fn(xr)
        ref.backward(g.float())
        assert torch.allclose(out.float(), ref, rtol=2e-3, atol=2e-3)
        assert torch.allclose(xa.grad.float(), xr.grad, rtol=2e-3, atol=2e-3)


def test_encoding_errors():
    import torch
    from qmlp import bindings
    from qmlp._capi import QmlpError
    with pytest.raises(QmlpError):
        bindings.Encoding(json.dumps({"id": "Nope", "start_in": 0, "n_in": 1}))
    with pytest.raises(QmlpError):
        bindings.Encoding(json.dumps(specs.hashgrid(7, 1, 1, -1, 2, 2)))      # dimension must be in [1, 6]
    cfg, e, oe = _enc("dense2d")
    with pytest.raises(QmlpError):
        e.inference_with_parameter(torch.zeros((4, 2), device="cuda"), torch.zeros((3,), device="cuda"))  # wrong size


@pytest.mark.parametrize("name,n", [("dense2d_multires", 32769), ("dense2d_multires", 70001), ("hash3d_f2", 30000), ("hash3d_f2", 65),
                                    ("hash2d_f8", 20001), ("hash3d_f3_add", 30001)])
def test_adjoint_with_gradient_copies(name, n):
    """Table and input gradients with scratch memory for copies of the small levels (lengths at which no, some and all levels
    have copies, odd numbers of points) against the same call without scratch. Both add the same fp32 terms in different
    orders: a row of k terms of one sign may differ by k * 2^-24 relative, here k <= 2^15 on a level of a few hundred rows."""
    import ctypes as C
    import torch
    from qmlp._capi import check, lib, wrap
    cfg, e, oe = _enc(name)
    lo = float(oe.box_min.min())
    hi = lo + float((1.0 / oe.box_inv_size).max())
    x = torch.from_numpy(helpers.uniform(9, 1, (n, oe.start_in + oe.n_in), lo, hi)).cuda()
    adj = torch.from_numpy(helpers.uniform(9, 2, (n, oe.num_outputs), 0.0, 1.0)).cuda()
    table = torch.from_numpy(helpers.uniform(9, 3, (oe.num_parameters,), -1.0, 1.0)).cuda()
    need = C.c_size_t()
    check(lib().qmlp_encoding_adjoint_memory(e._h, n, 3, C.byref(need)))
    assert (need.value > 0) == (n != 65)
    results = []
    for tmp in (None, torch.full((max(need.value, 16),), 0x7e, dtype=torch.uint8, device="cuda")):
        gx, gt = torch.zeros_like(x), torch.zeros_like(table)
        p, g, ai = wrap(table), wrap(gt), wrap(gx)
        check(lib().qmlp_encoding_adjoint_with_memory(e._h, wrap(x), wrap(adj), ai, None, C.byref(p), C.byref(g), 3,
                                                      tmp.data_ptr() if tmp is not None else None, need.value if tmp is not None else 0))
        torch.cuda.synchronize()
        results.append((gx, gt))
    (gx0, gt0), (gx1, gt1) = results
    assert torch.equal(gx0, gx1)
    helpers.assert_close(gt1.cpu().numpy(), gt0.cpu().numpy(), f"{name} n={n}", rtol=2.0 ** -9, atol=1e-5 * float(gt0.abs().max()))


@pytest.mark.parametrize("name,n", [("dense2d_multires", 131073), ("hash3d_f2", 262147), ("hash4d_f4", 265001), ("hash2d_f8", 530001)])
def test_adjoint_added_up_by_cell(name, n):
    """Batches that are large enough for the gradient of the small levels to be added up by cell first, against the same call without
    scratch: points below the box (other corners than a cell's), above it and on its borders. Tolerance as above; no row
    gets more than 2^18 terms of a few times the largest adjoint, most of them of one sign."""
    import ctypes as C
    import torch
    from qmlp._capi import check, lib, wrap
    cfg, e, oe = _enc(name)
    x = helpers.uniform(10, 1, (n, oe.n_in), -0.02, 1.02)
    x[::97] = np.round(x[::97])
    x = torch.from_numpy(x).cuda()
    adj = torch.from_numpy(helpers.uniform(10, 2, (n, oe.num_outputs), 0.0, 1.0)).cuda()
    table = torch.from_numpy(helpers.uniform(10, 3, (oe.num_parameters,), -1.0, 1.0)).cuda()
    for mode in (2, 3):
        need = C.c_size_t()
        check(lib().qmlp_encoding_adjoint_memory(e._h, n, mode, C.byref(need)))
        assert need.value > 0
        results = []
        for tmp in (None, torch.full((need.value,), 0x7e, dtype=torch.uint8, device="cuda")):
            gx, gt = torch.zeros_like(x), torch.zeros_like(table)
            p, g, ai = wrap(table), wrap(gt), wrap(gx)
            check(lib().qmlp_encoding_adjoint_with_memory(e._h, wrap(x), wrap(adj), ai, None, C.byref(p), C.byref(g), mode,
                                                          tmp.data_ptr() if tmp is not None else None, need.value if tmp is not None else 0))
            torch.cuda.synchronize()
            results.append((gx, gt))
        (gx0, gt0), (gx1, gt1) = results
        assert torch.equal(gx0, gx1)
        helpers.assert_close(gt1.cpu().numpy(), gt0.cpu().numpy(), f"{name} n={n}", rtol=2.0 ** -9, atol=1e-5 * float(gt0.abs().max()))


@pytest.mark.parametrize("name,half", [("dense2d_multires", False), ("hash4d_f4", True), ("hash4d_f4", False), ("hash2d_f8", False), ("hash2d_f8", True)])
def test_forward_from_copies_by_cell(name, half):
    """Batches that are large enough for copies of the small levels by cell against the same call without scratch: points below the box (a warp
    that holds one reads the table), above it and on its borders; a table at an odd offset. The terms are the same; a compiler that
    forms the cell fraction with one rounding in one place and two in another moves it by R * 2^-24, R up to 256 here, and with it a feature
    by that times the largest slope of a cell, 2, in each dimension; points outside extrapolate, and so does the rounding."""
    import ctypes as C
    import torch
    from qmlp._capi import check, lib, wrap
    cfg, e, oe = _enc(name)
    n = (3 << 18) + 77
    x = helpers.uniform(11, 1, (n, oe.n_in), 0.0, 1.0)
    x[::1013] -= 0.5
    x[::1009] += 0.5
    x[::97] = np.round(x[::97])
    x = torch.from_numpy(x).cuda()
    for shift in (0, 1):
        data = torch.from_numpy(helpers.uniform(11, 3, (oe.num_parameters + 1,), -1.0, 1.0)).cuda()
        table = (data.half() if half else data)[shift:shift + oe.num_parameters]
        need = C.c_size_t()
        p = wrap(table)
        check(lib().qmlp_encoding_forward_memory(e._h, n, C.byref(p), C.byref(need)))
        assert need.value > 0
        check(lib().qmlp_encoding_forward_memory(e._h, 1000, C.byref(p), C.byref(C.c_size_t())))
        results = []
        for tmp in (None, torch.full((need.value,), 0x7e, dtype=torch.uint8, device="cuda")):
            out = torch.zeros((n, oe.num_outputs), device="cuda")
            check(lib().qmlp_encoding_forward_with_memory(e._h, wrap(x), wrap(out), None, C.byref(p), tmp.data_ptr() if tmp is not None else None,
                                                          need.value if tmp is not None else 0))
            torch.cuda.synchronize()
            results.append(out)
        inside = ((x >= 0) & (x <= 1)).all(dim=1)
        a, b = results[0][inside], results[1][inside]
        assert float((a - b).abs().max()) <= 256 * 2.0 ** -24 * 2 * oe.n_in
        a, b = results[0][~inside].double(), results[1][~inside].double()
        assert float((a - b).abs().max()) <= 1e-4 * float(a.abs().max())


def test_network_inference_from_copies_by_cell():
    """The level-major pass with and without copies by cell (memory for the planes alone): the same features up to the rounding of a cell
    fraction (above), which an fp16 rounding of a feature shows as 2^-11 now and then, and four layers pass on."""
    import ctypes as C
    import torch
    from qmlp import bindings
    from qmlp._capi import check, lib, wrap
    from test_gpu_network import network_cases
    cfg, rng, _ = network_cases()["config5_small"]
    spec = oracle.parse_spec(cfg)
    net = bindings.Network(json.dumps(cfg))
    n = (3 << 18) + 5
    x = torch.from_numpy(helpers.uniform(12, 1, (n, spec.num_inputs), -0.001, 1.0)).cuda()
    w = torch.from_numpy(helpers.xavier_parameters(spec, cfg, bias_scale=0.1)).cuda().half()
    t = torch.from_numpy(helpers.grid_tables(spec, scale=1.0)[0]).cuda().half()
    net.inference(x[:64], w, [t])   # binds the parameters
    try:
        bindings.QuickMLP.set_kernel_path(2)
        need = C.c_size_t()
        check(lib().qmlp_network_inference_memory(net._h, n, C.byref(need)))
        planes = (n + 65535) // 65536 * 65536 * sum(net.encoding(i).num_output_channels() for i in range(net.num_encodings())) * 2
        assert need.value > planes
        results = []
        for size in (planes, need.value):
            tmp = torch.full((size,), 0x7e, dtype=torch.uint8, device="cuda")
            out = torch.zeros((n, spec.num_outputs), device="cuda")
            o = wrap(out)
            check(lib().qmlp_network_inference_with_memory(net._h, wrap(x), C.byref(o), None, tmp.data_ptr(), size))
            torch.cuda.synchronize()
            results.append(out)
        assert float((results[0] - results[1]).norm()) <= 1e-4 * float(results[0].norm()) > 0
    finally:
        bindings.QuickMLP.set_kernel_path(0)


def test_two_chunks_of_an_inference_from_copies_by_cell():
    """Copies that the first chunk of an inference fills serve the second. Tolerance as above."""
    import ctypes as C
    import torch
    from qmlp import bindings
    from qmlp._capi import check, lib, wrap
    from test_gpu_network import network_cases
    cfg, rng, _ = network_cases()["config5_small"]
    spec = oracle.parse_spec(cfg)
    net = bindings.Network(json.dumps(cfg))
    n, chunk = (1 << 22) + 4099, 1 << 22
    x = torch.rand((n, spec.num_inputs), device="cuda", generator=torch.Generator(device="cuda").manual_seed(13))
    w = torch.from_numpy(helpers.xavier_parameters(spec, cfg, bias_scale=0.1)).cuda().half()
    t = torch.from_numpy(helpers.grid_tables(spec, scale=1.0)[0]).cuda().half()
    net.inference(x[:64], w, [t])   # binds the parameters
    try:
        bindings.QuickMLP.set_kernel_path(2)
        need = C.c_size_t()
        check(lib().qmlp_network_inference_memory(net._h, n, C.byref(need)))
        planes = chunk * sum(net.encoding(i).num_output_channels() for i in range(net.num_encodings())) * 2
        assert need.value > planes
        results = []
        for size in (planes, need.value):
            tmp = torch.full((size,), 0x7e, dtype=torch.uint8, device="cuda")
            out = torch.zeros((n, spec.num_outputs), device="cuda")
            o = wrap(out)
            check(lib().qmlp_network_inference_with_memory(net._h, wrap(x), C.byref(o), None, tmp.data_ptr(), size))
            torch.cuda.synchronize()
            results.append(out)
        for part in (slice(0, chunk), slice(chunk, n)):
            assert float((results[0][part] - results[1][part]).norm()) <= 1e-4 * float(results[0][part].norm()) > 0
    finally:
        bindings.QuickMLP.set_kernel_path(0)


@pytest.mark.parametrize("name", ["dense2d_multires", "hash2d_f8"])
def test_points_and_adjoints_that_are_not_finite(name):
    """NaN and infinite coordinates and adjoints with copies and records by cell: the same entries as without scratch are not finite, the others
    agree (tolerances as above)."""
    import ctypes as C
    import torch
    from qmlp._capi import check, lib, wrap
    cfg, e, oe = _enc(name)
    n = (3 << 18) + 77
    x = helpers.uniform(14, 1, (n, oe.n_in), 0.0, 1.0)
    adj = helpers.uniform(14, 2, (n, oe.num_outputs), 0.1, 1.0)
    for k, v in enumerate((np.nan, np.inf, -np.inf)):
        x[1000 + k, 0] = v
        x[2000 + k, -1] = v
        adj[200001 + 31 * k, k] = v
    x, adj = torch.from_numpy(x).cuda(), torch.from_numpy(adj).cuda()
    table = torch.from_numpy(helpers.uniform(14, 3, (oe.num_parameters,), -1.0, 1.0)).cuda()
    p, forward, adjoint = wrap(table), C.c_size_t(), C.c_size_t()
    check(lib().qmlp_encoding_forward_memory(e._h, n, C.byref(p), C.byref(forward)))
    check(lib().qmlp_encoding_adjoint_memory(e._h, n, 2, C.byref(adjoint)))
    assert forward.value > 0 and adjoint.value > 0
    results = []
    for scratch in (False, True):
        out, gt = torch.zeros((n, oe.num_outputs), device="cuda"), torch.zeros_like(table)
        g = wrap(gt)
        tmp = torch.full((max(forward.value, adjoint.value),), 0x7e, dtype=torch.uint8, device="cuda")
        at = tmp.data_ptr() if scratch else None
        check(lib().qmlp_encoding_forward_with_memory(e._h, wrap(x), wrap(out), None, C.byref(p), at, forward.value if scratch else 0))
        check(lib().qmlp_encoding_adjoint_with_memory(e._h, wrap(x), wrap(adj), None, None, C.byref(p), C.byref(g), 2, at, adjoint.value if scratch else 0))
        torch.cuda.synchronize()
        results.append((out, gt))
    for (a, b), rtol in zip(zip(*results), (0.0, 2.0 ** -9)):
        finite = torch.isfinite(a)
        assert torch.equal(finite, torch.isfinite(b)) and 0 < int((~finite).sum()) < a.numel() // 2
        a, b = a[finite], b[finite]
        atol = 256 * 2.0 ** -24 * 2 * oe.n_in if rtol == 0 else 1e-5 * float(a.abs().max())
        assert bool(((a - b).abs() <= rtol * a.abs() + atol).all())
