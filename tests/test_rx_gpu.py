"""Rows c-e on the GPU (pilot fit, soft demap, block stage, LDPC, CRC) through the C ABI: held bit for bit to the
reference's own outputs (tests/golden/rx_ref.npz) and to the oracle on synthetic frames of every picture size."""
import os

import numpy as np
import pytest

import lizard_gb300 as lz
import oracle
from lizard_gb300_testing import synth

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")


def check(out, want, frame=0):
    assert np.array_equal(out["align"][frame][:2], want["align"])
    assert np.array_equal(out["llrf"][frame], want["llrf"])
    assert np.array_equal(out["sub_rms"][frame], want["sub_rms"])
    np.testing.assert_allclose(out["sub_est"][frame], want["sub_est"], rtol=1e-13)
    assert np.array_equal(out["its"][frame], want["its"].astype(np.int32))
    assert np.array_equal(out["ok"][frame], want["ok"])
    np.testing.assert_allclose(out["est"][frame], want["est"], rtol=1e-6)
    assert np.array_equal(out["pilot"][frame], want["pilot"], equal_nan=True)


@pytest.mark.parametrize("tag", ["a", "b"])
def test_finish_coef_matches_reference_golden(tag):
    g = np.load(os.path.join(GOLD, "rx_ref.npz"))
    n, subch, span = (int(x) for x in g[tag + "_fmt"])
    rx = lz.Receiver(n, subch, span, max_frames=1)
    out = rx.finish_coef(g[tag + "_coef"][None])
    check(out, {k: g[tag + "_" + k] for k in ("align", "llrf", "sub_rms", "sub_est", "its", "ok", "est", "pilot")})
    ok = out["ok"][0].astype(bool)
    assert ok.all()
    assert np.array_equal(out["blocks"][0], g[tag + "_blocks"])


def oracle_frames(fmt, frames, seed, shift=None, sigma=3.0):
    o = oracle.Fmt(fmt.n, fmt.subch, fmt.span)
    grids, blocks = synth.grids(fmt, frames, seed=seed, sigma=sigma, shift=shift)
    res = [o.receive(grids[f]) for f in range(frames)]
    return grids, blocks, res


@pytest.mark.parametrize("n,subch,frames,shift,sigma", [(384, 64, 3, None, 3.0), (512, 256, 2, (0.2, 0.1), 3.0),
                                                        (768, 320, 2, None, 12.0), (1024, 1024, 1, (-0.15, 0.3), 3.0),
                                                        (1152, 720, 1, None, 3.0), (1280, 880, 1, None, 3.0),
                                                        (1536, 1024, 2, (0.3, -0.25), 3.0)])
def test_finish_coef_matches_oracle(n, subch, frames, shift, sigma):
    fmt = lz.Format(n, subch, 128)
    _, blocks, res = oracle_frames(fmt, frames, seed=n + frames, shift=shift, sigma=sigma)
    rx = lz.Receiver(n, subch, 128, max_frames=frames)
    out = rx.finish_coef(np.stack([r["coef"] for r in res]))
    for f in range(frames):
        check(out, {"align": res[f]["align"], "llrf": res[f]["llrf"], "sub_rms": res[f]["sub_rms"], "sub_est": res[f]["sub_est"],
                    "its": res[f]["its"], "ok": res[f]["ok"], "est": res[f]["est"], "pilot": res[f]["pilot"]}, f)
        ok = out["ok"][f].astype(bool)
        assert np.array_equal(out["blocks"][f][ok], blocks[f][ok])
    assert rx.launches == 3 + fmt.tiers


@pytest.mark.parametrize("n,subch,frames,sigma", [(384, 64, 3, 3.0), (768, 320, 4, 60.0), (1536, 1024, 2, 3.0)])
def test_mixed_decode_matches_per_tier(n, subch, frames, sigma):
    """The decode stage in one persistent launch across the tiers (lizg_rx_set_ldpc_mixed) against a launch a tier:
    the same blocks, verdicts and iterations (declined, stalled and capped blocks included at the noisy size)."""
    fmt = lz.Format(n, subch, 128)
    grids, _ = synth.grids(fmt, frames, seed=n + 7, sigma=sigma)
    rx = lz.Receiver(n, subch, 128, max_frames=frames)
    assert rx.set_ldpc_mixed(0) == 0
    a = rx.finish_grid(grids)
    assert rx.launches == 4 + 3 + fmt.tiers
    assert rx.set_ldpc_mixed(1) == 0
    b = rx.finish_grid(grids)
    assert rx.launches == 4 + 3 + 1
    for k in ("blocks", "ok", "its", "llrf", "est"):
        assert np.array_equal(a[k], b[k]), k
    if sigma > 10:
        assert (a["its"] < 0).any() and (a["ok"] == 1).any()


def test_receiver_refuses_bad_calls():
    """Every receiver entry point checks its arguments before it queues anything: a zero or oversized batch, a frame
    under 2 x 2 or a pitch or frame stride too short for it, a NULL frame, registration or output, an unknown read,
    decode stage or tier; each is refused with LIZG_E_ARG and the handle stays usable."""
    import ctypes
    import torch
    n, subch, span, W, H = 384, 64, 128, 1280, 720
    fmt = lz.Format(n, subch, span)
    grey = synth.picture(fmt, synth.random_blocks(fmt.blocks, 5))
    luma, reg = synth.capture(fmt, grey, W, H, sigma=2.0, rng=np.random.default_rng(5))
    rx = lz.Receiver(n, subch, span, max_frames=2)
    o, s = lz.rx_outputs(rx.fmt, 2)
    d = torch.zeros((2, H, W), dtype=torch.uint8, device="cuda")
    r = torch.zeros((2, reg.size), dtype=torch.float32, device="cuda")
    L, P = lz.lib(), ctypes.c_void_p

    def call(luma=d.data_ptr(), w=W, h=H, pitch=W, stride=W * H, reg=r.data_ptr(), frames=1, out=s):
        return L.lizg_rx_finish_luma_dev(rx._h, P(luma), w, h, pitch, stride, P(reg), frames, ctypes.byref(out) if out else None,
                                         None, None, None)

    for kw in ({"frames": 0}, {"frames": 3}, {"w": 1}, {"pitch": W - 1}, {"stride": W * H - 1}, {"luma": 0}, {"reg": 0}, {"out": None}):
        assert call(**kw) == -1, kw
    assert call(out=lz.RxOut(None, s.ok, s.its, None, None, None, None, None, None)) == -1
    assert L.lizg_rx_set_read(rx._h, 7) == -1 and L.lizg_rx_set_ldpc_mixed(rx._h, 3) == -1 and L.lizg_rx_variant(rx._h, 9) == -1
    assert L.lizg_rx_finish_coef_dev(rx._h, None, 1, ctypes.byref(s), None) == -1
    # still usable: the clean frame decodes every block
    out = rx.finish_luma(luma[None], reg[None], grid=False)
    assert out["ok"].all()


@pytest.mark.parametrize("n,subch", [(384, 64), (768, 320), (1536, 1024)])
def test_pilot_fit_is_the_ordered_sums(n, subch):
    """The pilots' shift, its worth and its rounding as the reference's ordered double sums give them, over shifts about
    the threshold of turning back, and where the sums say little (no noise, an empty spectrum, scales at float's ends)."""
    fmt = lz.Format(n, subch, 128)
    o = oracle.Fmt(n, subch, 128)
    rng = np.random.default_rng(n)
    u, v = fmt.uv[0::2].astype(np.float64), fmt.uv[1::2].astype(np.float64)
    sym = (1.0 - 2.0 * fmt.white[0::2]) + 1j * (1.0 - 2.0 * fmt.white[1::2])
    cases = [(rng.normal(0, s, 2), noise, scale) for s in (0.0, 3e-4, 1e-3, 3e-3, 1e-2, 0.1) for noise in (0.0, 0.1, 0.7) for scale in (1.0, 400.0)]
    cases += [((0.01, -0.02), 0.3, 0.0), ((0.01, -0.02), 0.3, 1e-18), ((0.01, -0.02), 0.3, 1e14), ((0.3, 0.2), 0.0, 1e-9)]
    coef = np.empty((len(cases), u.size), np.complex64)
    for i, (d, noise, scale) in enumerate(cases):
        z = sym * np.exp(-2j * np.pi * (u * d[0] + v * d[1]) / n)
        coef[i] = scale * (z + noise * (rng.standard_normal(u.size) + 1j * rng.standard_normal(u.size)))
    rx = lz.Receiver(n, subch, 128, max_frames=len(cases))
    got = rx.finish_coef(coef)["align"]
    turned = 0
    for i in range(len(cases)):
        want, _ = o.pilot_align(coef[i].view(np.float32))
        assert np.array_equal(got[i, :2], want), (i, cases[i], got[i], want)
        assert got[i, 2] == float(np.any(want != 0))
        turned += int(np.any(want != 0))
    assert 0 < turned < len(cases)


@pytest.mark.parametrize("turn", [False, True])
def test_finish_coef_from_and_to_unaligned_buffers(turn):
    """Spectra 8 bytes past a 16-byte boundary, soft values and blocks at odd addresses: the values of the aligned call."""
    import ctypes
    import torch
    fmt = lz.Format(512, 128, 128)
    _, _, res = oracle_frames(fmt, 2, seed=11, shift=(0.2, 0.1) if turn else None)
    rx = lz.Receiver(512, 128, 128, max_frames=2)
    coef = np.ascontiguousarray(np.stack([r["coef"] for r in res]), np.float32).reshape(2, -1)
    want = rx.finish_coef(coef)
    assert bool(want["align"][:, 2].all()) == turn
    o, s = lz.rx_outputs(fmt, 2, keep=True)
    d = torch.zeros(coef.size + 8, dtype=torch.float32, device="cuda")
    d[2:2 + coef.size] = torch.from_numpy(coef.ravel()).cuda()
    soft = torch.zeros(o["llrf"].numel() + 16, dtype=torch.int8, device="cuda")
    blocks = torch.zeros(o["blocks"].numel() + 16, dtype=torch.uint8, device="cuda")
    s.llrf, s.blocks = soft.data_ptr() + 2, blocks.data_ptr() + 1
    lz._check(lz.lib().lizg_rx_finish_coef_dev(rx._h, ctypes.c_void_p(d.data_ptr() + 8), 2, ctypes.byref(s),
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "finish_coef")
    torch.cuda.synchronize()
    assert np.array_equal(soft[2:2 + o["llrf"].numel()].cpu().numpy(), want["llrf"].ravel())
    assert np.array_equal(blocks[1:1 + o["blocks"].numel()].cpu().numpy(), want["blocks"].ravel())
    for k in ("its", "ok", "est", "pilot", "sub_est", "sub_rms"):
        assert np.array_equal(o[k].cpu().numpy(), want[k], equal_nan=k == "pilot"), k


@pytest.mark.parametrize("frames", [10, 24, 36, 60])
def test_decode_of_many_frames_matches_oracle(frames):
    """Tiers on both sides of one and of two codewords a CTA (152 SMs hold 608, 456, 456 and 304 CTAs of the four codes; the
    tiers are of 57, 33, 17 and 17 blocks a frame): 10 frames keep every codeword alone, 60 take items of every code from
    the counter. Frames of six noise levels in shuffled order, so that a half takes its next block through the bit map and
    the whitening while its partner runs on, past declined blocks, among blocks that converge, stall and run to the cap."""
    fmt = lz.Format(1024, 1024, 128)
    o = oracle.Fmt(1024, 1024, 128)
    res = [o.receive(synth.grids(fmt, 1, seed=int(s), sigma=s)[0][0]) for s in (3.0, 38.0, 45.0, 60.0, 75.0, 120.0)]
    for kind in (-1, -2, -3):
        assert any((r["its"] == kind).any() for r in res), kind
    order = np.random.default_rng(frames).integers(0, len(res), frames)
    rx = lz.Receiver(1024, 1024, 128, max_frames=frames)
    out = rx.finish_coef(np.stack([res[k]["coef"] for k in order]))
    for f, k in enumerate(order):
        assert np.array_equal(out["its"][f], res[k]["its"].astype(np.int32)), f
        assert np.array_equal(out["ok"][f], res[k]["ok"]), f
        ok = res[k]["ok"].astype(bool)
        assert np.array_equal(out["blocks"][f][ok], res[k]["blocks"][ok]), f


def _held(make):
    """Device memory that a handle takes, in bytes."""
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    h = make()
    after = torch.cuda.mem_get_info()[0]
    del h
    return before - after


def test_handles_hold_no_samples_they_do_not_read():
    """A handle's device memory a frame is its transform's, spectrum's and soft values' buffers: the decode's 16-bit samples
    are a bounded workspace (it does not grow past 256 MB), and the handles that never read a frame by it (field
    refinement: the exact walk; eight-parameter refinement: grids) hold none."""
    n, subch = 1536, 1024
    need, vrows, nx = subch * lz.SUB, int(lz.Format(n, subch, 128).uv[1::2].max()) + 1, synth.layout_nodes(128).size
    rx = 8 * vrows * n + 8 * need + 2 * need + 16 * n * nx + 8 * (2 * n + vrows) + 20 * n + 64 * 1024   # Y, C, soft values, the walk's table, the rest
    slack = 64 << 20   # allocations rounded up
    lz.Receiver(n, subch, 128, max_frames=1)   # the module, the tables
    grown = _held(lambda: lz.Receiver(n, subch, 128, max_frames=192)) - _held(lambda: lz.Receiver(n, subch, 128, max_frames=64))
    assert grown <= 128 * rx + slack
    assert _held(lambda: lz.Receiver(n, subch, 128, max_frames=192)) <= 192 * rx + (256 << 20) + slack
    # field refinement: its own pictures, spectra, half-planes and partial sums beside the receiver's
    field = rx + 4 * n * n + 8 * need + 8 * vrows * n + (1 << 20)
    lz.FieldRefiner(n, subch, 128, chunk=1)
    grown = _held(lambda: lz.FieldRefiner(n, subch, 128, chunk=48)) - _held(lambda: lz.FieldRefiner(n, subch, 128, chunk=16))
    assert grown <= 32 * field + slack
    # nine pictures a frame, with their spectra, beside the receiver's
    gn = 9 * (rx + 4 * n * n + 8 * need)
    lz.PilotRefiner(n, subch, 128, chunk=1)
    grown = _held(lambda: lz.PilotRefiner(n, subch, 128, chunk=6)) - _held(lambda: lz.PilotRefiner(n, subch, 128, chunk=2))
    assert grown <= 4 * gn + slack


def test_batches_past_the_samples_workspace():
    """60 frames of n = 1536 by the decode's read: more than the samples' workspace holds, so the transform takes them in
    turns; every output as from two batches that fit, and as the engine's stage-wise run gives them."""
    import ctypes
    import torch
    P = ctypes.c_void_p
    n, subch, span, W, H, F = 1536, 1024, 128, 640, 480, 60
    rng = np.random.default_rng(60)
    side = span + 30
    luma = torch.from_numpy(rng.integers(0, 256, (F, H, W), dtype=np.uint8)).cuda()
    luma[3:5] = 128   # and frames of one grey level
    nn = synth.layout_nodes(span).size
    reg = np.zeros((F, 9 + 2 * nn * nn), np.float32)
    for f in range(F):
        s = 440.0 / side * (1 + 0.02 * rng.uniform(-1, 1))
        reg[f, :9] = [s, 0.02 * rng.uniform(-1, 1), 90.0, 0.02 * rng.uniform(-1, 1), s, 12.0, 1e-5 * rng.uniform(-1, 1), 1e-5 * rng.uniform(-1, 1), 1]
        reg[f, 9:] = rng.normal(0, 0.3, 2 * nn * nn)
    reg = torch.from_numpy(reg).cuda()
    rx = lz.Receiver(n, subch, span, max_frames=F)
    fmt = lz.Format(n, subch, span)
    want, _ = lz.rx_outputs(fmt, F, keep=True)
    wcoef = torch.empty((F, subch * lz.SUB, 2), device="cuda")

    def finish(f0, f1, o, coef):
        out, s = o
        lz._check(lz.lib().lizg_rx_finish_luma_dev(rx._h, P(luma[f0:f1].data_ptr()), W, H, W, W * H, P(reg[f0:f1].data_ptr()), f1 - f0,
                                                   ctypes.byref(s), None, P(coef.data_ptr()), None), "lizg_rx_finish_luma_dev")
        torch.cuda.synchronize()
        return out

    for f0 in (0, 30):
        part = finish(f0, f0 + 30, lz.rx_outputs(fmt, 30, keep=True), wcoef[f0:f0 + 30])
        for k in want:
            want[k][f0:f0 + 30] = part[k]
    coef = torch.empty_like(wcoef)
    got = finish(0, F, lz.rx_outputs(fmt, F, keep=True), coef)
    assert torch.equal(coef.view(torch.int32), wcoef.view(torch.int32))
    for k in want:
        assert np.array_equal(got[k].cpu().numpy(), want[k].cpu().numpy(), equal_nan=k in ("pilot", "est", "sub_est")), k
    assert rx.launches == 5 + 2 + 3 + fmt.tiers   # two turns
    # stage-wise, beside a format whose frames fit
    eng = lz.Engine()
    a, b = eng.add_format(n, subch, span, F), eng.add_format(384, 64, span, 4)
    eng.set_mixed(1)
    big, sb = lz.rx_outputs(fmt, F, keep=True)
    small, ss = lz.rx_outputs(lz.Format(384, 64, span), 4, keep=True)
    eng.run_dev([(a, luma.data_ptr(), W, H, W, W * H, reg.data_ptr(), F, sb),
                 (b, luma.data_ptr(), W, H, W, W * H, reg.data_ptr(), 4, ss)], 0)
    torch.cuda.synchronize()
    for k in want:
        assert np.array_equal(big[k].cpu().numpy(), want[k].cpu().numpy(), equal_nan=k in ("pilot", "est", "sub_est")), k
    rs = lz.Receiver(384, 64, span, max_frames=4)
    one, so = lz.rx_outputs(lz.Format(384, 64, span), 4, keep=True)
    lz._check(lz.lib().lizg_rx_finish_luma_dev(rs._h, P(luma.data_ptr()), W, H, W, W * H, P(reg.data_ptr()), 4, ctypes.byref(so), None, None, None),
              "lizg_rx_finish_luma_dev")
    torch.cuda.synchronize()
    for k in one:
        assert np.array_equal(small[k].cpu().numpy(), one[k].cpu().numpy(), equal_nan=k in ("pilot", "est", "sub_est")), k
