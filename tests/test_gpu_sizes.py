"""Sizes at which the kernels change their split of the work: tiles of the sort, blocks of the bottom-up pass, rays per warp of the
logged backward, the number of forwards whose logs are kept, upstream gradients that are not given."""
import numpy as np
import pytest
import torch

import helpers as hp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    from diff_surfel_tracing import _C
    assert torch.cuda.is_available()
    _C.lib()
    return _C


def _state(C, wc, wave=None):
    st = C.OptiXStateWrapper("")
    if wave is not None:
        st.set_wavefront_min_rays(0 if wave else 1 << 40)
    C.build_acceleration_structure(st, wc["v"], wc["f"], 1)
    return st


@pytest.mark.parametrize("P", [1, 2, 3, 5, 255, 256, 257, 4095, 4096, 4097, 8193])
def test_forward_at_block_and_tile_edges_of_the_build(C, oracle_mod, P):
    """Build and refit, rounds and per-ray kernel, against the oracle bit for bit; a ragged grid."""
    w = hp.workloads.make_workload(1, P=P, H=37, W=45)
    w["scales"] = w["scales"] * 3.0
    w["v"], w["f"] = hp.workloads.get_triangles(w["means3D"], w["scales"], w["rotations"])
    wc = hp.to_cuda(w)
    want = oracle_mod.Oracle(oracle_mod.Scene(w["v"]), impl="restatement", portable_exp=True).forward(w, training=True)
    for wave in (False, True):
        st = _state(C, wc, wave)
        for rebuild in (1, 0):
            C.build_acceleration_structure(st, wc["v"], wc["f"], rebuild)
            got = hp.cuda_forward(C, st, wc)
            torch.cuda.synchronize()
            assert st.status() == 0
            for k in ("rgb", "dpt", "acc", "norm", "mid"):
                assert np.array_equal(got[k].cpu().numpy().reshape(want[k].shape).view(np.uint32), want[k].view(np.uint32)), (wave, rebuild, k)


@pytest.mark.parametrize("H,W", [(17, 9), (64, 64), (129, 130), (190, 200), (460, 470)])
def test_logged_backward_at_every_split(C, H, W):
    """8, 16 and 32 rays per warp and the build for large calls: the gradients of the re-tracing backward."""
    w = hp.workloads.make_workload(3, P=30_000, H=H, W=W)
    wc = hp.to_cuda(w)
    st = _state(C, wc)
    f = hp.cuda_forward(C, st, wc)
    up = {k: torch.randn(f[k].shape, device="cuda") for k in ("rgb", "dpt", "norm", "aux")}
    logged = hp.cuda_backward(C, st, wc, f, up, serial=st.last_forward_serial)
    traced = hp.cuda_backward(C, st, wc, f, up, serial=0)
    torch.cuda.synchronize()
    assert st.status() == 0
    for k in hp.GRAD_KEYS:
        a, b = logged[k].cpu().numpy(), traced[k].cpu().numpy()
        m = np.isfinite(b)
        assert hp.rel_l2(a[m], b[m]) < 1e-4, k


@pytest.mark.parametrize("views", [2, 4, 5])
def test_logs_of_several_forwards(C, views):
    """Views traced one after the other, then their backwards: over the kept logs from the second step on, the first of more views than
    logs are kept by re-tracing; the gradients of a state that keeps one log."""
    w = hp.workloads.make_workload(3, P=20_000, H=48, W=64)
    wc = hp.to_cuda(w)
    ref, st = _state(C, wc), _state(C, wc)
    st.set_kept_logs(4)
    rays = [hp.workloads.pinhole_rays(48, 64, 50.0, (np.sin(a) * 4, -np.cos(a) * 4, 0.0)) for a in range(views)]
    cs = [dict(wc, ray_o=o.cuda(), ray_d=d.cuda()) for o, d in rays]
    for step in range(3):
        fs = []
        for c in cs:
            f = hp.cuda_forward(C, st, c)
            torch.cuda.synchronize()
            fs.append((f, st.last_forward_serial))
        walked = []
        for c, (f, serial) in zip(cs, fs):
            dg, up = {}, dict(rgb=torch.ones_like(f["rgb"]))
            g = hp.cuda_backward(C, st, c, f, up, diag=dg, serial=serial)
            r = hp.cuda_backward(C, ref, c, f, up, serial=0)
            torch.cuda.synchronize()
            walked.append(int(dg["counters"][2]) > 0)
            for k in ("means3D", "shs", "opacities", "scales", "rotations", "ray_o"):
                assert hp.rel_l2(g[k].cpu().numpy(), r[k].cpu().numpy()) < 1e-4, (step, k)
        assert st.status() == 0
    assert sum(walked) == (0 if views <= 4 else 4)        # a fifth forward finds the logs full and starts anew


def test_missing_upstream_gradients_are_zeros_and_the_arena_stays_clean(C):
    """None for an upstream gradient equals a tensor of zeros; a call's rows do not leak into the next one's, also across surfel counts."""
    st = C.OptiXStateWrapper("")
    e = torch.empty((0,), device="cuda")
    for P in (9_000, 4_000, 9_000):
        wc = hp.to_cuda(hp.workloads.make_workload(3, P=P, H=40, W=56))
        C.build_acceleration_structure(st, wc["v"], wc["f"], 1)
        f = hp.cuda_forward(C, st, wc)
        full = hp.cuda_backward(C, st, wc, f, dict(dpt=torch.ones_like(f["dpt"])), serial=st.last_forward_serial)
        part = C.trace_surfels_backward(st, True, wc["ray_o"], wc["ray_d"], wc["v"], wc["bg"], wc["means3D"], wc["shs"], wc["sh_degree"], e,
                                        wc["others_precomp"], wc["opacities"], wc["scales"], 1.0, wc["rotations"], e, e, e, e, False, False,
                                        wc["max_trace_depth"], wc["specular_threshold"], *(f[k] for k in ("rgb", "dpt", "acc", "norm", "dist", "aux", "mid")),
                                        None, torch.ones_like(f["dpt"]), None, None, None, None, _forward_serial=st.last_forward_serial)
        torch.cuda.synchronize()
        assert st.status() == 0
        for k, i in (("ray_o", 0), ("means3D", 2), ("shs", 5), ("opacities", 8), ("scales", 9), ("rotations", 10)):
            a, b = part[i].cpu().numpy(), full[k].cpu().numpy()
            assert np.array_equal(np.isfinite(a), np.isfinite(b)), k
            m = np.isfinite(b)
            assert hp.rel_l2(a[m], b[m]) < 1e-5, (P, k)


@pytest.mark.parametrize("missing", ["rgb", "dpt", "acc", "norm", "aux"])
def test_absent_upstream_gradients_are_an_error_unless_asked_for(C, missing):
    """A library caller that forgets a pointer is told; the module switches the meaning to zeros for its own calls."""
    wc = hp.to_cuda(hp.workloads.make_workload(1, P=2_000, H=32, W=32))
    st = _state(C, wc)
    f = hp.cuda_forward(C, st, wc)
    up = {k: torch.ones((*f["rgb"].shape[:2], 2 if k == "aux" else f[k].shape[-1]), device="cuda") for k in ("rgb", "dpt", "acc", "norm", "aux")}
    up[missing] = None
    hp.cuda_backward(C, st, wc, f, up)
    st.set_absent_gradients(False)
    with pytest.raises(RuntimeError, match="upstream gradient pointer is null"):
        hp.cuda_backward(C, st, wc, f, up)
    up[missing] = torch.ones((*f["rgb"].shape[:2], 2 if missing == "aux" else f[missing].shape[-1]), device="cuda")
    hp.cuda_backward(C, st, wc, f, dict(up, dist=None))
    torch.cuda.synchronize()
    assert st.status() == 0


@pytest.mark.parametrize("shift", [0.0, 300.0, 2e4])
@pytest.mark.parametrize("config,size", [(1, 4.0), (3, 2.0)])
def test_hulls_of_later_enumerations(C, config, size, shift):
    """The rounds walk for hulls of the rays from the least advanced one's distance on (or of the points they have reached), the per-ray kernel for one
    ray from its moved origin: the same bits, also where moving the origin rounds coarsely (a scene far from the world's origin), from the
    kernels with and without counters; the re-tracing backward composites the hits the forward logged."""
    w = hp.workloads.make_workload(config, P=150_000, H=256, W=320)
    w["scales"] = w["scales"] * size
    t = torch.tensor([shift, -0.5 * shift, shift])
    w["means3D"], w["ray_o"] = w["means3D"] + t, w["ray_o"] + t
    w["v"], w["f"] = hp.workloads.get_triangles(w["means3D"], w["scales"], w["rotations"])
    wc = hp.to_cuda(w)
    st, ray = _state(C, wc, True), _state(C, wc, False)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        f = hp.cuda_forward(C, st, wc)
        serial = st.last_forward_serial
        torch.cuda.synchronize()
    # what this is about did run: later enumerations of most rays in the rounds, and batches walked in groups (an idle launch takes 2 us)
    assert st.round_counts()[3] > 256 * 320 // 2
    assert sum("k_enum_group" in e.name and e.device_time > 30 for e in prof.events()) > 3
    up = dict(rgb=torch.randn(f["rgb"].shape, device="cuda"))
    logged, traced = {}, {}
    g = hp.cuda_backward(C, st, wc, f, up, diag=logged, serial=serial)
    counted = hp.cuda_forward(C, st, wc, diag={})
    r = hp.cuda_backward(C, st, wc, f, up, diag=traced, serial=0)
    rounds = st.round_counts()
    plain = hp.cuda_backward(C, st, wc, f, up, serial=0)
    want = hp.cuda_forward(C, ray, wc)
    torch.cuda.synchronize()
    assert st.status() == 0 and ray.status() == 0
    for k in ("rgb", "dpt", "acc", "norm", "aux", "mid"):
        bits = want[k].cpu().numpy().view(np.uint32)
        assert np.array_equal(f[k].cpu().numpy().view(np.uint32), bits), k
        assert np.array_equal(counted[k].cpu().numpy().view(np.uint32), bits), k
    assert rounds[2] > 256 * 320 // 2 and int(traced["counters"][2]) > 0 and int(logged["counters"][2]) == 0
    assert int(traced["counters"][5]) == int(logged["counters"][5])
    for k in hp.GRAD_KEYS:
        for got in (r, plain):
            a, b = got[k].cpu().numpy(), g[k].cpu().numpy()
            assert np.array_equal(np.isfinite(a), np.isfinite(b)), k
            m = np.isfinite(b)
            assert hp.rel_l2(a[m], b[m]) < 1e-4, k


@pytest.mark.parametrize("rays,limit", [("starts", 4.9), ("lengths", 3.4)])
def test_hulls_of_rays_that_start_or_step_differently(C, rays, limit):
    """Rays that start at distances of their own towards one surface, or whose directions differ in length, are walked from the points they have
    reached, whose box is narrower than that of their lines: nodes per walk against those of the plain view (lines only: 6.1 to 7 and 4.2
    times as many, the narrower of both: 3.9 and 2.8; the limits lie between), and the bits of the per-ray kernel."""
    w = hp.workloads.make_workload(2, P=300_000, H=300, W=400)
    r = torch.rand((300, 400, 1), generator=torch.Generator().manual_seed(1))
    nodes = []
    for o, d in ((w["ray_o"], w["ray_d"]), (w["ray_o"] + 2.5 * r * w["ray_d"], w["ray_d"]) if rays == "starts" else (w["ray_o"], w["ray_d"] * (0.8 + 0.2 * r))):
        wc = hp.to_cuda(dict(w, ray_o=o.contiguous(), ray_d=d.contiguous()))
        got = []
        for wave in (True, False):
            st, dg = _state(C, wc, wave), {}
            f = hp.cuda_forward(C, st, wc)
            hp.cuda_forward(C, st, wc, diag=dg)
            torch.cuda.synchronize()
            assert st.status() == 0
            got.append(f)
            if wave:
                nodes.append(int(dg["counters"][2]) / int(dg["counters"][1]))
    for k in ("rgb", "dpt", "acc", "norm", "mid"):
        assert np.array_equal(got[0][k].cpu().numpy().view(np.uint32), got[1][k].cpu().numpy().view(np.uint32)), k
    assert nodes[1] < limit * nodes[0], nodes


def _slots(H, W):
    """List slots of an image: whole blocks of 64 x 32 pixels."""
    return -(-W // 64) * -(-H // 32) * 2048


@pytest.mark.parametrize("coeffs,degree", [(16, 3), (16, 1), (9, 2), (4, 1)])
def test_composite_build_for_large_calls(C, coeffs, degree):
    """The composite kernel runs another build from 921,600 list slots on: each row of rays comes out as in a call below that, for SH rows of
    every alignment."""
    w = hp.workloads.make_workload(3, P=20_000, H=960, W=960)
    assert _slots(960, 960) >= 900 << 10 > _slots(928, 960)
    wc = hp.to_cuda(w)
    wc["shs"], wc["sh_degree"] = wc["shs"][:, :coeffs].contiguous(), degree
    st = _state(C, wc)
    large = hp.cuda_forward(C, st, wc, training=False)
    part = dict(wc, ray_o=wc["ray_o"][:928].contiguous(), ray_d=wc["ray_d"][:928].contiguous())
    small = hp.cuda_forward(C, st, part, training=False)
    torch.cuda.synchronize()
    assert st.status() == 0 and float(large["acc"].max()) > 0.5
    for k in ("rgb", "dpt", "acc", "norm", "mid"):
        assert torch.equal(large[k][:928], small[k]), k


def test_weight_sums_of_large_calls_against_64_bits(C):
    """The per-surfel weights of a call in fixed point against sums in 64 bits of what calls of four rows each give. Bounds: a contribution is
    at least 1e-4 / 255 and rounded to 2^-41 (1.2e-6 of it), the result and the parts to 2^-24; sums of 216,200 rays in float are off by
    9e-7 in the 2-norm here."""
    wc = hp.to_cuda(hp.workloads.make_workload(3, P=30_000, H=460, W=470))
    st = _state(C, wc)
    wet = hp.cuda_forward(C, st, wc)["wet"].double()
    parts = _state(C, wc, wave=False)
    want = torch.zeros_like(wet)
    for r in range(0, 460, 4):
        part = dict(wc, ray_o=wc["ray_o"][r:r + 4].contiguous(), ray_d=wc["ray_d"][r:r + 4].contiguous())
        want += hp.cuda_forward(C, parts, part)["wet"].double()
    torch.cuda.synchronize()
    assert st.status() == 0 and int((want > 0).sum()) > 10_000
    assert float((wet - want).norm() / want.norm()) < 3e-7
    assert float(((wet - want).abs() - 2e-6 * want).max()) <= 0.0


def test_logged_hits_that_no_longer_contribute(C):
    """Two views traced, then surfels made transparent in place, then the backwards. The first view's records are rebuilt from what the
    tensors hold by then: its logged hits on those surfels are passed over, as a re-trace passes them over."""
    wc = hp.to_cuda(hp.workloads.make_workload(3, P=20_000, H=48, W=64))
    st = _state(C, wc)
    st.set_kept_logs(4)
    for step in range(2):       # the second step's logs both fit
        fs = []
        for _ in range(2):
            f = hp.cuda_forward(C, st, wc)
            torch.cuda.synchronize()
            fs.append((f, st.last_forward_serial))
        if step == 0:
            for f, serial in fs[::-1]:
                hp.cuda_backward(C, st, wc, f, dict(rgb=torch.ones_like(f["rgb"])), serial=serial)
    gone = torch.rand(20_000, device="cuda") < 0.5
    kept = wc["opacities"].clone()
    wc["opacities"][gone] = 0.0
    f, serial = fs[0]
    dg = {}
    g = hp.cuda_backward(C, st, wc, f, {k: torch.ones_like(f[k]) for k in ("rgb", "dpt", "norm")}, diag=dg, serial=serial)
    torch.cuda.synchronize()
    wc["opacities"].copy_(kept)
    assert st.status() == 0 and int(dg["counters"][2]) == 0       # from the log
    for k in ("means3D", "opacities", "scales", "rotations"):
        assert float(g[k][gone].abs().max()) == 0.0 and float(g[k][~gone].abs().max()) > 0.0, k


def test_column_of_rays_whose_padded_tiles_exceed_a_list_word(C):
    """2^24 rays as one column: padded to whole blocks of tiles they would be 2^30 list slots, so they are walked linearly. The outputs and
    gradients of the same rays as 64 rows."""
    wc = hp.to_cuda(hp.workloads.make_workload(1, P=2_000, H=128, W=128))
    n = 1 << 24
    o, d = (wc[k].reshape(-1, 3).repeat(n // 128**2, 1) for k in ("ray_o", "ray_d"))
    got = []
    for shape in ((n, 1, 3), (64, n // 64, 3)):
        st = _state(C, wc)
        c = dict(wc, ray_o=o.view(shape), ray_d=d.view(shape))
        f = hp.cuda_forward(C, st, c, training=False)
        g = hp.cuda_backward(C, st, c, f, dict(rgb=torch.ones_like(f["rgb"])))
        torch.cuda.synchronize()
        assert st.status() == 0 and float(f["acc"].max()) > 0.5
        got.append((f["rgb"].view(n, 3), f["dpt"].view(n), f["mid"].view(n, -1)[:, :16].clone(), g["ray_o"].view(n, 3), g["opacities"]))
        del st, f, g, c
    for a, b in zip(got[0][:3], got[1][:3]):
        assert torch.equal(a, b)
    for a, b in zip(got[0][3:], got[1][3:]):       # (sums of 32-bit terms in another order)
        assert float((a - b).double().norm() / b.double().norm()) < 1e-4


def _dense(H, W):
    """Rays with 256 contributions each: 16 records, more than the 12 a log is first sized for."""
    w = hp.workloads.make_workload(3, P=20_000, H=H, W=W)
    w["scales"], w["opacities"], w["max_trace_depth"] = 10.0 * w["scales"], torch.full_like(w["opacities"], 0.05), 0
    w["v"], w["f"] = hp.workloads.get_triangles(w["means3D"], w["scales"], w["rotations"])
    return hp.to_cuda(w)


def test_no_memory_for_the_log_is_no_error(C):
    """Where several views' logs do not fit the device there is one view's, where that does not either there is none: the backward
    re-traces, with the gradients of a state that has its log."""
    wc = _dense(48, 64)
    ref = _state(C, wc)
    keys = ("means3D", "shs", "opacities", "scales", "rotations", "ray_o")

    def step(st, views):
        fs = []
        for _ in range(views):
            f = hp.cuda_forward(C, st, wc)
            torch.cuda.synchronize()
            fs.append((f, st.last_forward_serial))
        for f, serial in fs:
            g = hp.cuda_backward(C, st, wc, f, dict(rgb=torch.ones_like(f["rgb"])), serial=serial)
            r = hp.cuda_backward(C, ref, wc, f, dict(rgb=torch.ones_like(f["rgb"])), serial=0)
            torch.cuda.synchronize()
            for k in keys:
                assert hp.rel_l2(g[k].cpu().numpy(), r[k].cpu().numpy()) < 1e-4, k
        assert st.status() == 0
        return [serial for _, serial in fs], st.chunk_log()["records_held"]

    st = _state(C, wc)
    st.set_kept_logs(4)
    for _ in range(10):       # (what a forward wants is read back now and then)
        _, one = step(st, 1)
    st.set_log_alloc_limit(one * 132)
    for _ in range(3):       # from the second step on room for four is asked for
        serials, held = step(st, 4)
        assert all(serials) and held <= one
    st.set_log_alloc_limit(0)
    for _ in range(2):
        _, held = step(st, 4)
    assert held > one
    for limit in (1, 48 * 64 * 12 * 8):       # no records; records, but no room for their index or the other way round
        st = _state(C, wc)
        st.set_log_alloc_limit(limit)
        serials, held = step(st, 1)
        assert serials == [0] and held == 0
        st.set_log_alloc_limit(0)
        serials, held = step(st, 1)
        assert serials[0] > 0 and held > 0


def test_room_for_several_logs_is_asked_for_only_while_they_are_used(C):
    """Four views per step grow the log to four; after steps of one view a larger call's log is sized for one."""
    wc, big = _dense(48, 64), _dense(96, 128)
    held = {}
    for views in (1, 4):
        st = _state(C, wc)
        st.set_kept_logs(4)
        for c, n in (*[(wc, 1)] * 10, *[(wc, views)] * 3, (wc, 1), (wc, 1), (big, 1)):
            fs = [(hp.cuda_forward(C, st, c), st.last_forward_serial) for _ in range(n)]
            for f, serial in fs:
                hp.cuda_backward(C, st, c, f, dict(rgb=torch.ones_like(f["rgb"])), serial=serial)
            torch.cuda.synchronize()
            held.setdefault(views, []).append(st.chunk_log()["records_held"])
    assert held[4][-2] > held[1][-2] and held[4][-1] == max(held[4][-2], held[1][-1]) and held[1][-1] > held[1][-2]


@pytest.mark.parametrize("limit", [1, 31, 33, 1000])
def test_log_holds_no_more_records_than_its_limit(C, limit):
    """Limits that are no multiple of the 32 records that are interleaved: the rays that fit are taken from the log, the others re-traced."""
    wc = hp.to_cuda(hp.workloads.make_workload(3, P=20_000, H=48, W=64))
    st = _state(C, wc)
    st.set_chunk_log_max_records(limit)
    f = hp.cuda_forward(C, st, wc)
    up, dg = dict(rgb=torch.ones_like(f["rgb"])), {}
    logged = hp.cuda_backward(C, st, wc, f, up, diag=dg, serial=st.last_forward_serial)
    traced = hp.cuda_backward(C, st, wc, f, up, serial=0)
    torch.cuda.synchronize()
    assert st.status() == 0 and st.chunk_log()["records_held"] == limit and int(dg["counters"][2]) > 0
    for k in ("means3D", "shs", "opacities", "scales", "rotations", "ray_o"):
        assert hp.rel_l2(logged[k].cpu().numpy(), traced[k].cpu().numpy()) < 1e-4, k


def test_training_forwards_without_a_backward_keep_no_log(C):
    """Weights gathered under no_grad, or with nothing that takes a gradient: such calls leave no log behind, and the log of the forward
    whose backward is still to come stays."""
    from diff_surfel_tracing import SurfelTracer, SurfelTracingSettings
    w = hp.workloads.make_workload(3, P=20_000, H=48, W=64)
    wc = hp.to_cuda(w)
    tracer = SurfelTracer()
    tracer.build_acceleration_structure(wc["v"], wc["f"], rebuild=True)
    e = torch.zeros(1, device="cuda")
    settings = SurfelTracingSettings(48, 64, 1.0, 1.0, wc["bg"], 1.0, e, e, w["sh_degree"], e, False, False, w["max_trace_depth"], w["specular_threshold"])
    names = ("shs", "others_precomp", "opacities", "scales", "rotations")

    def trace(leaf):
        p = {k: wc[k].clone().requires_grad_(leaf) for k in names}
        return tracer(wc["ray_o"], wc["ray_d"], wc["v"], wc["means3D"], torch.zeros_like(wc["means3D"]), tracer_settings=settings, **p)

    first = trace(True)
    serial = tracer.optix_context.last_forward_serial
    assert serial > 0
    for k in range(6):
        if k % 2:
            out = trace(False)
        else:
            with torch.no_grad():
                out = trace(True)
        assert tracer.optix_context.last_forward_serial == 0
        assert torch.equal(out[0], first[0]) and torch.allclose(out[7], first[7], rtol=1e-5)
    diag = {}
    hp.cuda_backward(C, tracer.optix_context, wc, dict(zip(hp.FWD_KEYS, (t.detach() for t in first))), dict(rgb=torch.ones_like(first[0])),
                     diag=diag, serial=serial)
    torch.cuda.synchronize()
    assert tracer.optix_context.status() == 0 and int(diag["counters"][2]) == 0       # nothing was walked again


def test_round_counts_hold_list_lengths_only(C):
    """A caller's array longer than the list lengths is filled up with zeros, not with the counters that lie behind them."""
    import ctypes
    wc = hp.to_cuda(hp.workloads.make_workload(3, P=20_000, H=96, W=128))
    st = _state(C, wc, wave=True)
    hp.cuda_forward(C, st, wc)
    buf = (ctypes.c_int32 * 300)(*[-1] * 300)
    assert C.lib().dst_debug_round_counts(st.handle, buf, 300, None) == 0
    short = st.round_counts()
    assert len(short) > 1 and short == sorted(short, reverse=True)
    assert list(buf) == short + [0] * (300 - len(short))


def test_first_steps_of_a_small_state_map_memory_once(C):
    """Build, forward and backward of a new state with 10,000 surfels and 128 x 128 rays: one device allocation. Buffers that grow from call to
    call move to other places of it and then out of it; the results are a fresh state's."""
    w = hp.workloads.make_workload(1)
    wc = hp.to_cuda(w)
    st = _state(C, wc)
    f = hp.cuda_forward(C, st, wc)
    hp.cuda_backward(C, st, wc, f, dict(rgb=torch.ones_like(f["rgb"])), serial=st.last_forward_serial)
    assert st.device_allocations() == 1
    torch.cuda.synchronize()
    st = C.OptiXStateWrapper("")
    for P, side in ((500, 32), (2_000, 48), (5_000, 130), (20_000, 260), (45_000, 300), (120_000, 64), (1_000, 40)):
        wc = hp.to_cuda(hp.workloads.make_workload(3, P=P, H=side, W=side))
        C.build_acceleration_structure(st, wc["v"], wc["f"], 1)
        fresh = _state(C, wc)
        got = []
        for s in (st, fresh):
            f = hp.cuda_forward(C, s, wc)
            g = hp.cuda_backward(C, s, wc, f, dict(rgb=torch.ones_like(f["rgb"])), serial=s.last_forward_serial)
            got.append((f, g))
        torch.cuda.synchronize()
        assert st.status() == 0
        for k in ("rgb", "dpt", "acc", "norm", "mid"):
            assert torch.equal(got[0][0][k], got[1][0][k]), (P, k)
        for k in ("means3D", "shs", "opacities", "scales", "rotations", "ray_o"):
            assert hp.rel_l2(got[0][1][k].cpu().numpy(), got[1][1][k].cpu().numpy()) < 1e-5, (P, k)
    assert st.device_allocations() > 1
